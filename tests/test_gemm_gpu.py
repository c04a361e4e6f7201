"""tcgen05 GEMM against a plain fp32 PyTorch product, every operand layout and epilogue."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, a_t, b_t):
    af = a.float().t() if a_t else a.float()
    bf = b.float().t() if b_t else b.float()
    return af @ bf


def _rand(shape, scale=1.0):
    return (torch.randn(shape, device="cuda") * scale).to(torch.bfloat16)


@pytest.mark.parametrize("a_t,b_t", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("mnk", [(128, 256, 64), (256, 512, 256), (384, 264, 200), (1000, 776, 520), (4096, 2048, 1024)])
def test_matmul_layouts(a_t, b_t, mnk):
    from halo_b200.ops import _lib
    from halo_b200.ops.gemm import matmul

    M, N, K = mnk
    torch.manual_seed(0)
    a = _rand((K, M) if a_t else (M, K))
    b = _rand((N, K) if b_t else (K, N))
    out = matmul(a, b, a_t=a_t, b_t=b_t)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    ref = _ref(a, b, a_t, b_t)
    err = (out.float() - ref).abs().max().item()
    tol = 2e-2 * ref.abs().max().item() + 1e-3
    assert err <= tol, f"max err {err} > {tol}"


def test_matmul_fp32_and_accumulate():
    from halo_b200.ops.gemm import matmul

    torch.manual_seed(1)
    a, b = _rand((512, 320)), _rand((264, 320))
    ref = _ref(a, b, False, True)
    out = matmul(a, b, out_dtype=torch.float32)
    assert (out - ref).abs().max().item() <= 1e-3 * ref.abs().max().item() + 1e-4
    acc = torch.ones_like(out)
    matmul(a, b, out=acc, accumulate=True, alpha=0.5)
    assert (acc - (1 + 0.5 * ref)).abs().max().item() <= 1e-3 * ref.abs().max().item() + 1e-4
    accb = torch.ones((512, 264), dtype=torch.bfloat16, device="cuda")
    matmul(a, b, out=accb, accumulate=True)
    assert (accb.float() - (1 + ref)).abs().max().item() <= 2e-2 * ref.abs().max().item()


@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (3, 136, 200), (16, 4096, 4096), (17, 1000, 776), (64, 2048, 12288), (65, 264, 8200),
                                   (128, 8192, 512), (129, 4096, 4096), (256, 520, 4104), (257, 264, 4096), (16, 128, 1016),
                                   (16, 136, 1016), (17, 520, 1024), (33, 8200, 2048), (64, 520, 1016), (128, 1000, 2048), (100, 8200, 2056)])
def test_few_rows(M, N, K):
    """Products with few rows at the edges of the dispatch (16, 64, 128 and 256 rows; one to eight cuts of the reduction,
    ragged N and K): bf16, fp32 and SwiGLU stores into strided outputs against 64-bit sums. fp32 sums of K products of
    unit normals: the tensor core adds 16 products at a time and cuts the sum to 24 bits, so each of the K / 16 additions
    loses at most 2 ** -23 of a partial sum that stays below 5 K ** 0.5; bf16 adds 2 ** -8 of the value."""
    from halo_b200.ops import _lib
    from halo_b200.ops.gemm import matmul, swiglu_matmul

    torch.manual_seed(M + N)
    x = torch.randn(M, K + 8, device="cuda").bfloat16()[:, :K]
    w = torch.randn(N, K, device="cuda").bfloat16()
    ref = x.double() @ w.double().t()
    noise = K / 16 * 2.0 ** -23 * 5 * K ** 0.5 + 1e-6
    out = matmul(x, w, out_dtype=torch.float32, alpha=0.5)
    assert ((out - 0.5 * ref).abs() <= noise).all()
    wide = torch.full((M, N + 16), 7.0, dtype=torch.bfloat16, device="cuda")
    matmul(x, w, out=wide[:, :N])
    assert ((wide[:, :N] - ref).abs() <= 2.0 ** -8 * ref.abs() + noise).all() and (wide[:, N:] == 7.0).all()
    scaled = (w.float() * K ** -0.5).bfloat16()
    F = N // 16 * 8
    act, pre = swiglu_matmul(x, scaled[:2 * F], save_pre=True)
    pre_ref = x.double() @ scaled[:2 * F].double().t()
    assert ((pre - pre_ref).abs() <= 2.0 ** -8 * pre_ref.abs() + 1e-4).all()
    g, u = pre[:, :F].double(), pre[:, F:].double()
    act_ref = torch.nn.functional.silu(g) * u
    assert ((act - act_ref).abs() <= 2.0 ** -7 * act_ref.abs() + 1e-6).all()
    assert _lib.read_status() == 0


@pytest.mark.parametrize("M,N,K", [(5000, 4104, 64), (9001, 776, 136), (20000, 264, 200), (2500, 6000, 256), (19000, 520, 328),
                                   (300, 136, 72), (600, 2056, 520), (9472, 264, 264), (4000, 1544, 4104)])
def test_wide_tiles(M, N, K):
    """The 256 x 512 pair tiles at their edges: one to six blocks of the reduction (the second column block starts up to three
    late), ragged rows and columns, a last wave cut into column halves, every operand layout, stores and accumulation in
    both types, SwiGLU. Bounds as for the few-row products."""
    from halo_b200.ops import _lib
    from halo_b200.ops.gemm import matmul, swiglu_matmul

    torch.manual_seed(N)
    noise = K / 16 * 2.0 ** -23 * 5 * K ** 0.5 + 1e-6
    m8 = (M + 7) // 8 * 8
    for a_t in (False, True):
        a = torch.randn((K, m8) if a_t else (M, K), device="cuda").bfloat16()
        a = a[:, :M] if a_t else a
        for b_t in (False, True):
            b = torch.randn((N, K) if b_t else (K, N), device="cuda").bfloat16()
            ref = (a.double().t() if a_t else a.double()) @ (b.double().t() if b_t else b.double())
            out = torch.full((M, N), 2.0, device="cuda")
            matmul(a, b, a_t=a_t, b_t=b_t, out=out, accumulate=True, alpha=0.5)
            assert ((out - 2.0 - 0.5 * ref).abs() <= noise + 2.0 ** -22 * (ref.abs() + 4)).all()
            wide = torch.full((M, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
            matmul(a, b, a_t=a_t, b_t=b_t, out=wide[:, :N])
            assert ((wide[:, :N] - ref).abs() <= 2.0 ** -8 * ref.abs() + noise).all() and (wide[:, N:] == 7.0).all()
            matmul(a, b, a_t=a_t, b_t=b_t, out=wide[:, :N], accumulate=True)
            assert ((wide[:, :N] - 2 * ref).abs() <= 3 * 2.0 ** -8 * ref.abs() * 1.5 + 2 * noise).all()
    x, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(2 * N, K, device="cuda") * K ** -0.5).bfloat16()
    act, pre = swiglu_matmul(x, w, save_pre=True)
    pre_ref = x.double() @ w.double().t()
    assert ((pre - pre_ref).abs() <= 2.0 ** -8 * pre_ref.abs() + 1e-4).all()
    act_ref = torch.nn.functional.silu(pre[:, :N].double()) * pre[:, N:].double()
    assert ((act - act_ref).abs() <= 2.0 ** -7 * act_ref.abs() + 1e-6).all()
    assert torch.equal(swiglu_matmul(x, w)[0], act) and _lib.read_status() == 0


def test_swiglu_epilogue():
    from halo_b200.ops.gemm import swiglu_matmul

    torch.manual_seed(2)
    x, w = _rand((777, 512)), _rand((2 * 384, 512), 0.05)
    act, pre = swiglu_matmul(x, w, save_pre=True)
    pre_ref = (x.float() @ w.float().t())
    assert (pre.float() - pre_ref).abs().max().item() <= 2e-2 * pre_ref.abs().max().item()
    g, u = pre.float()[:, :384], pre.float()[:, 384:]
    act_ref = torch.nn.functional.silu(g) * u
    assert (act.float() - act_ref).abs().max().item() <= 1e-2 * act_ref.abs().max().item() + 1e-3


def test_linear_autograd():
    from halo_b200.ops.gemm import linear

    torch.manual_seed(3)
    x = _rand((3, 100, 256)).requires_grad_()
    w = _rand((384, 256), 0.05).requires_grad_()
    y = linear(x, w)
    gy = _rand(y.shape)
    y.backward(gy)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    yr = xr @ wr.t()
    yr.backward(gy.float())
    for got, ref in ((y, yr), (x.grad, xr.grad), (w.grad, wr.grad)):
        assert (got.float() - ref).abs().max().item() <= 2e-2 * ref.abs().max().item() + 1e-3


@pytest.mark.parametrize("a_t,b_t", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("mnk", [(2048, 1024, 2048), (1000, 520, 1600), (304, 2048, 4096)])
def test_pair_kernel_shapes(a_t, b_t, mnk):
    """Long reductions with narrow outputs take the CTA-pair (cta_group::2) kernel; odd sizes exercise the half
    tiles of the second CTA and the clipped edges."""
    from halo_b200.ops import _lib
    from halo_b200.ops.gemm import matmul

    M, N, K = mnk
    torch.manual_seed(1)
    a = _rand((K, M) if a_t else (M, K), 0.3)
    b = _rand((N, K) if b_t else (K, N), 0.3)
    out = matmul(a, b, a_t=a_t, b_t=b_t)
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    ref = _ref(a, b, a_t, b_t)
    err = (out.float() - ref).abs().max().item()
    assert err <= 2e-2 * ref.abs().max().item() + 1e-3, err


def test_every_product_on_the_pair_kernel_in_a_fresh_process():
    """HALO_GEMM_PAIR=2 routes every dense and grouped product through the pair kernel; the kernel choice is read
    once per process, so the GEMM and MoE numerics run again in a child process with the switch set."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, HALO_GEMM_PAIR="2")
    r = subprocess.run([sys.executable, "-m", "pytest", "tests/test_gemm_gpu.py", "tests/test_moe_gpu.py", "-q", "-m", "gpu", "-x",
                        "-k", "not fresh_process"], cwd=root, env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]


@pytest.mark.parametrize("m,n", [(4096, 4096), (4090, 4092), (4096, 4000)])
def test_accumulate_keeps_subnormals_and_neighbours(m, n):
    """Whole 32-row blocks are added by TMA, ragged ones by the lanes; a zero product changes no bit of either, and nothing
    outside the output's columns is touched."""
    from halo_b200.ops.gemm import matmul

    a = torch.zeros(m, 256, device="cuda", dtype=torch.bfloat16)
    b = torch.zeros(n, 256, device="cuda", dtype=torch.bfloat16)
    buf = torch.full((m, n + 64), 1e-40, device="cuda")
    buf[:, 1::2] = -3e-41
    buf[:, 2::64] = float("inf")
    before = buf.clone()
    matmul(a, b, out=buf[:, :n], accumulate=True)
    assert torch.equal(buf.view(torch.int32), before.view(torch.int32))


def test_few_rows_from_several_threads():
    """Threads on streams of their own, some with the smallest tile's ring and some with the largest: a launch gets the
    shared memory it asks for whatever another thread's call sets in between. The entry point is called bare, so that the
    threads meet inside it and not at the interpreter's lock."""
    import threading

    from halo_b200.ops import _lib

    torch.manual_seed(0)
    N, K = 512, 4096
    w = torch.randn(N, K, device="cuda").bfloat16()
    entry = _lib.lib()._cdll.halo_gemm_bf16
    jobs = []
    for rows in (16, 200, 16, 200):
        x, out = torch.ones(rows, K, device="cuda").bfloat16(), torch.empty(rows, N, device="cuda", dtype=torch.bfloat16)
        stream = torch.cuda.Stream()
        args = (_lib.ptr(x), _lib.ptr(w), _lib.ptr(out), _lib.c_void_p(0), _lib.c_int(rows), _lib.c_int(N), _lib.c_int(K), _lib.c_ll(K),
                _lib.c_ll(K), _lib.c_ll(N), _lib.c_ll(0), _lib.c_int(0), _lib.c_int(0), _lib.c_int(0), _lib.c_float(1.0),
                _lib.ptr(_lib.status_word(w.device)), _lib.c_void_p(stream.cuda_stream))
        jobs.append((x, out, stream, args))
    torch.cuda.synchronize()
    codes = []

    def work(args):
        torch.cuda.set_device(0)
        codes.extend({entry(*args) for _ in range(5000)})

    threads = [threading.Thread(target=work, args=(job[3],)) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [0] * len(jobs), codes
    want = w.double().sum(1)
    for _, out, _, _ in jobs:
        assert ((out - want).abs() <= 2.0 ** -8 * want.abs() + 0.05).all()
    assert _lib.read_status() == 0


@pytest.mark.parametrize("M,N,K", [(3, 40, 72), (64, 4096, 512), (100, 136, 64), (200, 24576, 128), (256, 520, 1000)])
@pytest.mark.parametrize("f32", [False, True])
def test_outputs_off_the_16_byte_boundary(M, N, K, f32):
    """A few rows go to the kernel that stores pairs, whatever the reduction; what only the 16-byte kernels serve is refused."""
    from halo_b200.ops import _lib
    from halo_b200.ops.gemm import matmul

    torch.manual_seed(N)
    x, w = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    buf = torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
    matmul(x, w, out=buf[:, 2:2 + N])
    ref = x.double() @ w.double().t()
    noise = K / 16 * 2.0 ** -23 * 5 * K ** 0.5 + 1e-6
    assert ((buf[:, 2:2 + N] - ref).abs() <= (0.0 if f32 else 2.0 ** -8) * ref.abs() + noise).all()
    assert (buf[:, :2] == 7.0).all() and (buf[:, 2 + N:] == 7.0).all() and _lib.read_status() == 0
    for kwargs in ({"accumulate": True}, {"a_t": True}):
        with pytest.raises((_lib.KernelError, ValueError)):         # a transposed operand of ragged M has no legal row stride
            matmul(x.t().contiguous() if "a_t" in kwargs else x, w, out=buf[:, 2:2 + N], **kwargs)
    tall = torch.zeros(300, N + 8, device="cuda", dtype=buf.dtype)
    with pytest.raises(_lib.KernelError):
        matmul(torch.zeros(300, K, device="cuda", dtype=torch.bfloat16), w, out=tall[:, 2:2 + N])
