"""When an operation may pass its autograd node by: only where the node would have recorded nothing for anybody."""

import pytest
import torch
import torch.autograd.forward_ad as fwd_ad

from halo_b200.ops import _lib, gemm
from halo_b200.ops.norm import add_rms_norm, rms_norm


def test_condition_under_every_mode():
    assert not _lib.plain_inference()
    with torch.inference_mode():
        assert _lib.plain_inference()
    with torch.no_grad():
        assert _lib.plain_inference()
        with fwd_ad.dual_level():
            assert not _lib.plain_inference()
        seen = []

        def probe(x):
            seen.append(_lib.plain_inference())
            return x * 2

        torch.func.vmap(probe)(torch.ones(3))
        torch.func.jvp(probe, (torch.ones(3),), (torch.ones(3),))
        torch.jit.trace(probe, (torch.ones(3),), check_trace=False)
        assert seen == [False] * 3 and _lib.plain_inference()


@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")
def test_traced_linear_follows_new_inputs(monkeypatch):
    """A product that is written through a pointer, as the kernels do: the tracer sees an allocation and nothing else, so the
    call itself has to be what it records."""

    def through_a_pointer(a, b, a_t=False, b_t=True):
        out = torch.empty(a.shape[0], b.shape[0])
        out.numpy()[...] = a.detach().numpy() @ b.detach().numpy().T
        return out

    monkeypatch.setattr(gemm, "matmul", through_a_pointer)
    w = torch.randn(4, 3)
    with torch.no_grad():
        traced = torch.jit.trace(lambda x: gemm.linear(x, w), (torch.randn(2, 3),), check_trace=False)
        x = torch.randn(2, 3)
        assert torch.equal(traced(x), through_a_pointer(x, w))


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")
@pytest.mark.parametrize("T", [1, 33])
def test_both_routes_agree_bit_for_bit(T):
    from halo_b200.models.qwen3 import DenseMLP

    torch.manual_seed(T)
    H, F = 256, 136
    x, r = torch.randn(T, H, device="cuda").bfloat16(), torch.randn(T, H, device="cuda").bfloat16()
    w, norm = torch.randn(F, H, device="cuda").bfloat16(), torch.rand(H, device="cuda").bfloat16()
    mlp = DenseMLP(H, F, torch.bfloat16, "cuda").requires_grad_(False)
    mlp.gate_up_proj.normal_(0.0, 0.05)
    mlp.down_proj.normal_(0.0, 0.05)

    def call(x, r):
        return (gemm.linear(x, w), rms_norm(x, norm), *add_rms_norm(x, r, norm), mlp(x))

    recorded = [t.detach() for t in call(x.clone().requires_grad_(), r.clone().requires_grad_())]
    with torch.no_grad():
        plain = call(x, r)
        traced = torch.jit.trace(call, (torch.randn_like(x), torch.randn_like(r)), check_trace=False)(x, r)
        with fwd_ad.dual_level():
            dual = call(x, r)
    with torch.inference_mode():
        inference = call(x, r)
    for got in (plain, traced, dual, inference):
        assert all(torch.equal(a, b) for a, b in zip(got, recorded))
