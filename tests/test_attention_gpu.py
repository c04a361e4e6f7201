"""tcgen05 flash attention (packed, causal, GQA) against an fp32 PyTorch attention, fwd and bwd."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _mk(T, Hq, Hkv, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = (torch.randn(T, Hq * 128, device="cuda", generator=g)).bfloat16()
    k = (torch.randn(T, Hkv * 128, device="cuda", generator=g)).bfloat16()
    v = (torch.randn(T, Hkv * 128, device="cuda", generator=g)).bfloat16()
    return q, k, v


def _close(a, b, tol, name):
    err = (a.float() - b.float()).abs().max().item()
    ref = b.float().abs().max().item()
    assert err <= tol * ref + 1e-3, f"{name}: max err {err} vs ref max {ref}"


@pytest.mark.parametrize("lens,Hq,Hkv", [
    ([128], 1, 1),
    ([256], 2, 1),
    ([100], 2, 2),
    ([300, 77, 515], 4, 2),
    ([1024, 33, 1, 640], 8, 2),
])
def test_flash_attention_fwd_bwd(lens, Hq, Hkv):
    from halo_b200.ops import _lib
    from halo_b200.ops.attention import attention_reference, build_plan, flash_attention

    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    T = cu[-1]
    q, k, v = _mk(T, Hq, Hkv)
    plan = build_plan(cu, device="cuda")
    qg, kg, vg = (t.clone().requires_grad_() for t in (q, k, v))
    o = flash_attention(qg, kg, vg, plan, Hq, Hkv)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    o_ref = attention_reference(qr, kr, vr, cu, Hq, Hkv)
    _close(o, o_ref, 2e-2, "out")
    do = torch.randn_like(o)
    o.backward(do)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    o_ref.backward(do.float())
    _close(qg.grad, qr.grad, 3e-2, "dq")
    _close(kg.grad, kr.grad, 3e-2, "dk")
    _close(vg.grad, vr.grad, 3e-2, "dv")


def _row_rel_err(a, b):
    """Largest per-row relative error: ||a_row - b_row|| / (||b_row|| + 2 % of the mean row norm). A row is judged
    against its own size, so a small row cannot hide behind the tensor's largest value; the floor keeps rows that are
    exactly zero in the reference (a document's first query has no gradient) from dividing by nothing."""
    a, b = a.float(), b.float()
    norms = b.norm(dim=-1)
    return ((a - b).norm(dim=-1) / (norms + 0.02 * norms.mean())).max().item()


@pytest.mark.parametrize("lens,scale_logits,bwd_variant", [
    ([16384, 500], 1.0, 2),            # a 16k-token document: 256 key tiles per query tile, every pipeline slot reused many times
    ([4096, 3000, 1096], 8.0, 2),      # logits x8: row maxima jump by far more than 2^8 between tiles (the lazy rescale fires)
    ([2500, 1300], 1.0, 1),            # the first backward form stays correct beside the double-buffered one
])
def test_flash_attention_long_documents_and_large_logits(lens, scale_logits, bwd_variant, monkeypatch):
    import subprocess
    import sys

    if bwd_variant != 2:
        # the variant is read once per process: check the other one in a child
        code = ("import os, sys; os.environ['HALO_ATTN_BWD_VARIANT']='1'; sys.path.insert(0, '.');"
                "import tests.test_attention_gpu as t; t._long_case(%r, %r)" % (lens, scale_logits))
        r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
        return
    _long_case(lens, scale_logits)


def _long_case(lens, scale_logits):
    from halo_b200.ops import _lib
    from halo_b200.ops.attention import attention_reference, build_plan, flash_attention

    Hq, Hkv = 4, 2
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    q, k, v = _mk(cu[-1], Hq, Hkv, seed=3)
    q = (q.float() * scale_logits ** 0.5).bfloat16()
    k = (k.float() * scale_logits ** 0.5).bfloat16()
    plan = build_plan(cu, device="cuda")
    qg, kg, vg = (t.clone().requires_grad_() for t in (q, k, v))
    o = flash_attention(qg, kg, vg, plan, Hq, Hkv)
    do = torch.randn_like(o)
    o.backward(do)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    # the fp32 oracle, one document at a time (a 16k x 16k score matrix per head fits; all heads at once would not)
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    o_ref = attention_reference(qr, kr, vr, cu, Hq, Hkv)
    o_ref.backward(do.float())
    assert _row_rel_err(o, o_ref) < 2e-2
    assert _row_rel_err(vg.grad, vr.grad) < 3e-2
    if scale_logits == 1.0:
        assert _row_rel_err(qg.grad, qr.grad) < 4e-2
        assert _row_rel_err(kg.grad, kr.grad) < 4e-2
    else:
        # nearly one-hot rows: dS = P (dP - delta) cancels almost completely for the winning key, and delta is formed from
        # the bf16 output, so single rows of dQ / dK carry the rounding of O at full size (any bf16 flash backward does);
        # the gradients as a whole must still agree
        for got, want, name in ((qg.grad, qr.grad, "dq"), (kg.grad, kr.grad, "dk")):
            rel = ((got.float() - want).norm() / want.norm()).item()
            assert rel < 5e-2, (name, rel)


@pytest.mark.parametrize("lens,window", [
    ([700, 300, 1048], 256),      # several documents, windows shorter than most of them
    ([2048], 128),                # every key tile is cut by the diagonal or by a window edge
    ([5000, 120], 1024),
    ([333], 4096),                # a window longer than the document: plain causal attention
    ([1500, 777], 100),           # a window that is no multiple of the tile sizes
])
def test_flash_attention_sliding_window(lens, window):
    from halo_b200.ops import _lib
    from halo_b200.ops.attention import attention_reference, build_plan, flash_attention

    Hq, Hkv = 4, 2
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    q, k, v = _mk(cu[-1], Hq, Hkv, seed=7)
    plan = build_plan(cu, device="cuda", window=window)
    qg, kg, vg = (t.clone().requires_grad_() for t in (q, k, v))
    o = flash_attention(qg, kg, vg, plan, Hq, Hkv)
    do = torch.randn_like(o)
    o.backward(do)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    o_ref = attention_reference(qr, kr, vr, cu, Hq, Hkv, window=window)
    o_ref.backward(do.float())
    assert _row_rel_err(o, o_ref) < 2e-2
    assert _row_rel_err(vg.grad, vr.grad) < 3e-2
    assert _row_rel_err(qg.grad, qr.grad) < 4e-2
    assert _row_rel_err(kg.grad, kr.grad) < 4e-2
    # the window changes the result (unless it covers the whole document)
    if window < max(lens):
        full = flash_attention(q, k, v, build_plan(cu, device="cuda"), Hq, Hkv)
        assert (full.float() - o.float()).abs().max().item() > 1e-2


@pytest.mark.parametrize("lens,window", [([700, 300, 1048], 0), ([1500, 777], 200), ([130], 0)])
def test_flash_attention_sinks(lens, window):
    """One logit per head in every row's softmax: output, dq / dk / dv and the gradient of the logits themselves."""
    from halo_b200.ops import _lib
    from halo_b200.ops.attention import attention_reference, build_plan, flash_attention

    Hq, Hkv = 4, 2
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    q, k, v = _mk(cu[-1], Hq, Hkv, seed=11)
    # logits that matter: scores of unit-variance inputs at scale 128^-0.5 have a standard deviation near 1
    sinks = torch.tensor([2.0, -1.0, 0.5, 4.0], device="cuda")
    plan = build_plan(cu, device="cuda", window=window)
    # The sum behind a sink's gradient inherits the outputs' bf16 rounding: an absolute error of about
    # 2 ** -9 * (T * 128) ** 0.5 * P, some 0.01, whatever the gradient itself cancels to. The output gradient is seeded so
    # that no gradient lies near zero, where a relative bound says nothing.
    torch.manual_seed(0)
    qg, kg, vg, sg = (t.clone().requires_grad_() for t in (q, k, v, sinks))
    o = flash_attention(qg, kg, vg, plan, Hq, Hkv, sinks=sg)
    do = torch.randn_like(o)
    o.backward(do)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    qr, kr, vr, sr = (t.float().requires_grad_() for t in (q, k, v, sinks))
    o_ref = attention_reference(qr, kr, vr, cu, Hq, Hkv, window=window, sinks=sr)
    o_ref.backward(do.float())
    assert _row_rel_err(o, o_ref) < 2e-2
    assert _row_rel_err(vg.grad, vr.grad) < 3e-2
    assert _row_rel_err(qg.grad, qr.grad) < 4e-2
    assert _row_rel_err(kg.grad, kr.grad) < 4e-2
    assert ((sg.grad - sr.grad).abs() / (sr.grad.abs() + 0.02 * sr.grad.abs().mean())).max().item() < 3e-2
    # the sinks take mass: the output differs from the sink-free one
    plain = flash_attention(q, k, v, plan, Hq, Hkv)
    assert (plain.float() - o.float()).abs().max().item() > 1e-2


def test_flash_attention_heads_of_64_run_zero_padded():
    from halo_b200.ops import _lib
    from halo_b200.ops.attention import attention_reference, build_plan, flash_attention

    Hq, Hkv, D = 8, 2, 64
    cu = [0, 400, 1000, 1111]
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn(cu[-1], Hq * D, device="cuda", generator=g).bfloat16()
    k = torch.randn(cu[-1], Hkv * D, device="cuda", generator=g).bfloat16()
    v = torch.randn(cu[-1], Hkv * D, device="cuda", generator=g).bfloat16()
    sinks = torch.linspace(-1, 3, Hq, device="cuda")
    plan = build_plan(cu, device="cuda", window=128)
    qg, kg, vg = (t.clone().requires_grad_() for t in (q, k, v))
    o = flash_attention(qg, kg, vg, plan, Hq, Hkv, sinks=sinks)
    assert o.shape == (cu[-1], Hq * D)
    do = torch.randn_like(o)
    o.backward(do)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    o_ref = attention_reference(qr, kr, vr, cu, Hq, Hkv, window=128, sinks=sinks)
    o_ref.backward(do.float())
    assert _row_rel_err(o, o_ref) < 2e-2
    assert _row_rel_err(vg.grad, vr.grad) < 3e-2
    assert _row_rel_err(qg.grad, qr.grad) < 4e-2
    assert _row_rel_err(kg.grad, kr.grad) < 4e-2


def test_rope_attention_fused_matches_reference():
    from halo_b200.ops.attention import build_plan, rope_attention
    from halo_b200.ops.rope import rope_table

    Hq, Hkv, lens = 4, 2, [200, 312]
    cu = [0, 200, 512]
    T = 512
    torch.manual_seed(0)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * 128, device="cuda").bfloat16()
    wq = (1 + 0.1 * torch.randn(128, device="cuda")).bfloat16()
    wk = (1 + 0.1 * torch.randn(128, device="cuda")).bfloat16()
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    table = rope_table(pos, 128, 1e6)
    table_cpu = rope_table(pos.cpu(), 128, 1e6)
    assert (table.cpu() - table_cpu).abs().max().item() < 1e-2
    plan = build_plan(cu, device="cuda")
    a = qkv.clone().requires_grad_()
    wqa, wka = wq.clone().requires_grad_(), wk.clone().requires_grad_()
    o = rope_attention(a, wqa, wka, table, plan, Hq, Hkv)
    do = torch.randn_like(o)
    o.backward(do)
    # oracle: same math on CPU in fp32 (weights/inputs as fp32 leaves)
    b = qkv.cpu().float().requires_grad_()
    wqb, wkb = wq.cpu().float().requires_grad_(), wk.cpu().float().requires_grad_()
    cplan = build_plan(cu)
    o_ref = rope_attention(b, wqb, wkb, table_cpu, cplan, Hq, Hkv)
    o_ref.backward(do.cpu().float())
    _close(o.cpu(), o_ref, 3e-2, "out")
    _close(a.grad.cpu(), b.grad, 4e-2, "dqkv")
    _close(wqa.grad.cpu(), wqb.grad, 5e-2, "dwq")
    _close(wka.grad.cpu(), wkb.grad, 5e-2, "dwk")


@pytest.mark.parametrize("T,Hq,Hkv,use_norm,shift", [(1, 2, 1, True, 0), (5, 26, 1, True, 0), (133, 32, 8, True, 0), (4100, 3, 1, True, 0),
                                                     (33, 8, 4, False, 0), (33, 6, 3, True, 4)])
def test_qk_norm_rope_head_counts_and_alignment(T, Hq, Hkv, use_norm, shift):
    """Odd head counts (a pair of heads that straddles q and k, or the end), more heads than one warp takes, more tokens
    than the fixed backward grid, and rows that start on 8- but not 16-byte boundaries, against 64 bits. Four bf16
    roundings (2 ** -8 each) of values of at most |x| + |partner|; gradients are rounded once."""
    from halo_b200.ops.rope import qk_norm_rope, rope_table

    torch.manual_seed(T + Hq)
    W = (Hq + 2 * Hkv) * 128
    flat = torch.randn(T * W + shift, device="cuda").bfloat16()
    qkv = flat[shift:].view(T, W).detach().requires_grad_()
    wq = (1 + 0.1 * torch.randn(128, device="cuda")).bfloat16().requires_grad_()
    wk = (1 + 0.1 * torch.randn(128, device="cuda")).bfloat16().requires_grad_()
    table = rope_table(torch.arange(T, device="cuda"), 128, 1e6)
    q, k = qk_norm_rope(qkv, wq, wk, table, Hq, Hkv, 1e-6, use_norm)
    gq, gk = torch.randn_like(q), torch.randn_like(k)
    leaves = [qkv, wq, wk] if use_norm else [qkv]
    grads = torch.autograd.grad([q, k], leaves, [gq, gk])
    xd, wqd, wkd = (t.detach().double().requires_grad_() for t in (qkv, wq, wk))
    x = xd.view(T, Hq + 2 * Hkv, 128)[:, :Hq + Hkv]
    if use_norm:
        w = torch.cat([wqd.expand(Hq, 128), wkd.expand(Hkv, 128)])
        x = w * (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6))
    cos, sin = table[:, None, :, 0].double(), table[:, None, :, 1].double()
    a, b = x[..., :64], x[..., 64:]
    y = torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
    bound = 1.02 * 2.0 ** -6 * (x.abs() + torch.cat([b, a], -1).abs()) + 1e-6
    got = torch.cat([q.view(T, Hq, 128), k.view(T, Hkv, 128)], 1)
    assert ((got - y).abs() <= bound).all()
    want = torch.autograd.grad(y, [xd, wqd, wkd] if use_norm else [xd], torch.cat([gq.view(T, Hq, 128), gk.view(T, Hkv, 128)], 1).double())
    for name, u, v in zip(("dqkv", "dwq", "dwk"), grads, want):
        assert (u - v).norm() <= 2.0 ** -7 * v.norm() + 1e-6, name


@pytest.mark.parametrize("direct", [False, True])
@pytest.mark.parametrize("ranks,lens,balance", [(2, [700, 129, 1, 1218], True), (2, [2048], False), (4, [900, 2300, 896], True)])
def test_context_parallel_kernels_on_one_gpu(ranks, lens, balance, direct):
    """The context-parallel instantiations of the attention kernels, every rank's launches one after the other on one GPU
    with all ranks' buffers in its memory (the kernels themselves never wait for a rank): outputs and gradients against the
    unsharded attention, with rows mirrored and with tiles read from their owners."""
    import numpy as np

    from halo_b200.ops import _lib
    from halo_b200.ops.attention import build_plan, flash_attention
    from halo_b200.parallel.context_parallel import TILE, CPExchange, build_cp_plan, cp_attention, make_layout

    class OneGpu(CPExchange):
        def __init__(self, rank, rows, total, cols):
            self.device, self.n_ranks, self.rank, self.direct_reads = torch.device("cuda", 0), ranks, rank, direct
            self.kv, self.dkv, self.mirror = (torch.zeros(n, cols, dtype=torch.bfloat16, device="cuda") for n in (rows, total, total))
            self.mirror_version, self.row_bytes, self.max_local_rows, self.max_row_tokens = 0, cols * 2, rows, total

        def barrier(self):
            pass

    Hq, Hkv, D = 8, 2, 128
    cu = np.concatenate([[0], np.cumsum(lens)])
    T = int(cu[-1])
    torch.manual_seed(T)
    q, k, v = _mk(T, Hq, Hkv)
    do = torch.randn_like(q)
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    ref = flash_attention(*leaves, build_plan(cu, device="cuda"), Hq, Hkv)
    want = [ref.detach(), *torch.autograd.grad(ref, leaves, do)]
    layouts = [make_layout(cu, r, ranks, balance) for r in range(ranks)]
    exchanges = [OneGpu(r, max(layouts[0].rows_of_rank), T + TILE, 2 * Hkv * D) for r in range(ranks)]
    for ex in exchanges:
        ex.kv_ptrs, ex.dkv_ptrs = [e.kv.data_ptr() for e in exchanges], [e.dkv.data_ptr() for e in exchanges]
        ex.kv_ptr_array = (_lib.c_void_p * ranks)(*ex.kv_ptrs)
        ex.mirror_ptr_array = (_lib.c_void_p * 1)(ex.mirror.data_ptr())
    rows = [torch.from_numpy(lay.local_index()).cuda() for lay in layouts]
    local = [[t[i].clone().requires_grad_() for t in (q, k, v)] for i in rows]
    for ex, (_, kl, vl) in zip(exchanges, local):
        ex.publish(kl.detach(), vl.detach())
    outs = [cp_attention(*local[r], layouts[r], build_cp_plan(layouts[r], torch.device("cuda", 0)), None, exchanges[r], Hq, Hkv)
            for r in range(ranks)]
    for _ in range(2):          # the first round fills every rank's staging rows, which the second one's owners then add
        grads = [torch.autograd.grad(outs[r], local[r], do[rows[r]], retain_graph=True) for r in range(ranks)]
    assert _lib.read_status() == 0
    for r in range(ranks):
        for name, got, full, tol in zip(("out", "dq", "dk", "dv"), (outs[r].detach(), *grads[r]), want, (2e-2, 3e-2, 3e-2, 3e-2)):
            _close(got, full[rows[r]].float(), tol, f"rank {r} {name}")
