"""Fused linear + cross-entropy and the log-prob scorer against full-logits PyTorch."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,V,chunk", [(300, 256, 4096, 128), (1000, 512, 32000, 4096)])
def test_fused_linear_cross_entropy(T, H, V, chunk):
    from halo_b200.ops.cross_entropy import fused_linear_cross_entropy

    torch.manual_seed(0)
    h = torch.randn(T, H, device="cuda").bfloat16()
    w = (torch.randn(V, H, device="cuda") * 0.05).bfloat16()
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[::7] = -100
    ha, wa = h.clone().requires_grad_(), w.clone().requires_grad_()
    loss = fused_linear_cross_entropy(ha, wa, labels, chunk_rows=chunk)
    loss.backward()
    hb, wb = h.float().requires_grad_(), w.float().requires_grad_()
    ref = torch.nn.functional.cross_entropy((hb @ wb.t()), labels, ignore_index=-100, reduction="sum") / (labels != -100).sum()
    ref.backward()
    assert abs(loss.item() - ref.item()) <= 2e-2 * abs(ref.item())
    assert (ha.grad.float() - hb.grad).abs().max().item() <= 5e-2 * hb.grad.abs().max().item() + 1e-6
    assert (wa.grad.float() - wb.grad).abs().max().item() <= 5e-2 * wb.grad.abs().max().item() + 1e-6


def test_linear_logprobs():
    from halo_b200.ops.cross_entropy import linear_logprobs

    torch.manual_seed(1)
    T, H, V = 500, 256, 8192
    h = torch.randn(T, H, device="cuda").bfloat16()
    w = (torch.randn(V, H, device="cuda") * 0.05).bfloat16()
    labels = torch.randint(0, V, (T,), device="cuda")
    ha, wa = h.clone().requires_grad_(), w.clone().requires_grad_()
    logp, ent = linear_logprobs(ha, wa, labels, chunk_rows=200, want_entropy=True)
    g = torch.randn(T, device="cuda")
    (logp * g).sum().backward()
    hb, wb = h.float().requires_grad_(), w.float().requires_grad_()
    lp = torch.log_softmax(hb @ wb.t(), dim=-1)
    ref = lp.gather(-1, labels[:, None])[:, 0]
    (ref * g).sum().backward()
    ent_ref = -(lp.exp() * lp).sum(-1)
    assert (logp - ref).abs().max().item() <= 5e-2
    assert (ent - ent_ref).abs().max().item() <= 5e-2
    assert (ha.grad.float() - hb.grad).abs().max().item() <= 5e-2 * hb.grad.abs().max().item() + 1e-6
    assert (wa.grad.float() - wb.grad).abs().max().item() <= 5e-2 * wb.grad.abs().max().item() + 1e-6


@pytest.mark.parametrize("T,V,chunk", [(129, 4104, 128), (3, 264, 4096), (7, 40960, 4)])
def test_head_loss_edges_and_upstream_scale(T, V, chunk):
    """Row chunks of one row, vector remainders of the row kernels, all rows of a chunk ignored, and an upstream gradient
    that is not 1, against 64-bit sums over the bf16 logits' own rounding (2 ** -8 of a logit of up to 5 moves a
    log-probability by that much; the stored gradients are rounded to bf16 twice)."""
    from halo_b200.ops.cross_entropy import fused_linear_cross_entropy, linear_logprobs

    torch.manual_seed(T)
    H = 128
    h = torch.randn(T, H, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(V, H, device="cuda") * H ** -0.5).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[0] = V - 1
    labels[-1] = -100
    loss = fused_linear_cross_entropy(h, w, labels, chunk_rows=chunk)
    dh, dw = torch.autograd.grad(3.0 * loss, [h, w], retain_graph=True)
    again = torch.autograd.grad(3.0 * loss, [h, w])
    assert torch.equal(dh, again[0]) and torch.equal(dw, again[1])      # the stored gradients are not consumed
    hd, wd = h.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    z = hd @ wd.t()
    ref = torch.nn.functional.cross_entropy(z, labels, ignore_index=-100)
    (3.0 * ref).backward()
    assert abs(loss.item() - ref.item()) <= 2.0 ** -8 * ref.item()
    assert (dh - hd.grad).norm() <= 2.0 ** -6 * hd.grad.norm() and (dw - wd.grad).norm() <= 2.0 ** -6 * wd.grad.norm()
    logp, ent = linear_logprobs(h.detach(), w.detach(), labels, chunk_rows=chunk, want_entropy=True)
    lp = torch.log_softmax(z.detach(), -1)
    want = torch.where(labels == -100, 0.0, lp.gather(-1, labels.clamp_min(0)[:, None])[:, 0])
    assert (logp - want).abs().max() <= 2.0 ** -8 * 5 and (ent + (lp.exp() * lp).sum(-1)).abs().max() <= 2.0 ** -8 * 5


@pytest.mark.filterwarnings("ignore::UserWarning")
@pytest.mark.parametrize("mode", ["create_graph", "batched", "hooks"])
def test_head_loss_gradients_by_the_uncommon_routes(mode):
    """A derivative with respect to the upstream scalar, a batch of upstream scalars, and saved gradients that a hook hands
    back in another layout: bit for bit what the plain backward gives for the same scalar."""
    from halo_b200.ops.cross_entropy import fused_linear_cross_entropy

    torch.manual_seed(0)
    T, H, V = 70, 128, 520
    h = torch.randn(T, H, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(V, H, device="cuda") * H ** -0.5).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device="cuda")

    def loss():
        return fused_linear_cross_entropy(h, w, labels).reshape(())

    one, three = (torch.autograd.grad(loss(), [h, w], torch.tensor(g, device="cuda")) for g in (1.0, 3.0))
    if mode == "create_graph":
        g = torch.tensor(3.0, device="cuda", requires_grad=True)
        got = torch.autograd.grad(loss(), [h, w], g, create_graph=True)
        assert all(torch.equal(a, b) for a, b in zip(got, three))
        for grad, unit in zip(got, one):
            along = torch.randn_like(unit)
            slope, = torch.autograd.grad(grad, g, along, retain_graph=True)
            want = (unit.double() * along.double()).sum()
            # the products are rounded to bf16 and summed in fp32
            assert abs(slope - want) <= 2.0 ** -8 * (unit.double() * along.double()).abs().sum()
    elif mode == "batched":
        got = torch.autograd.grad(loss(), [h, w], torch.tensor([1.0, 3.0], device="cuda"), is_grads_batched=True)
        for both, a, b in zip(got, one, three):
            assert torch.equal(both[0], a) and torch.equal(both[1], b)
    else:
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.t().contiguous().t() if t.dim() == 2 else t):
            got = torch.autograd.grad(loss(), [h, w], torch.tensor(3.0, device="cuda"))
        assert all(torch.equal(a, b) for a, b in zip(got, three))


def test_a_pending_loss_holds_its_head_gradient_once_in_bf16():
    """What stays allocated between forward and backward: both gradients in bf16 and a few scalars, not the fp32 sums."""
    from halo_b200.ops.cross_entropy import fused_linear_cross_entropy

    T, H, V = 64, 512, 32768
    h = torch.randn(T, H, device="cuda").bfloat16().requires_grad_()
    w = torch.randn(V, H, device="cuda").bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device="cuda")
    fused_linear_cross_entropy(h, w, labels)            # workspaces of the first call
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    loss = fused_linear_cross_entropy(h, w, labels)
    held = torch.cuda.memory_allocated() - before
    assert 2 * V * H <= held <= 2 * (V + T) * H + (1 << 20)
    loss.backward()
    assert w.grad.dtype == torch.bfloat16
