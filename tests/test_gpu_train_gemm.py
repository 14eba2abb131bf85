"""The training GEMMs at the edges of their tiles and dispatch: vk_tc_gemm (128 x 128 tiles, K chunks of 128, K splits,
wide and strided operands) against the f64 product of the BF16-rounded operands, vk_gemm's layer-3 kernels against the
f32 sums in k order, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layout(torch, x, order, pad, off):
    """x [rows, cols] in a larger buffer: row-major or column-major with padded stride, `off` elements from its start;
    (tensor, row stride, column stride)."""
    r, c = x.shape
    n, m = (r, c) if order == "row" else (c, r)
    buf = torch.zeros(n * (m + pad) + off, dtype=x.dtype, device=x.device)
    v = buf[off:].view(n, m + pad)[:, :m]
    v.copy_(x if order == "row" else x.t())
    return buf[off:], (m + pad, 1) if order == "row" else (1, m + pad)


@pytest.mark.parametrize("M,N,K", [(1, 16, 1), (127, 16, 16), (128, 128, 128), (129, 144, 129), (300, 256, 250),
                                   (256, 256, 1000), (256, 16, 8192), (64, 272, 513)])
@pytest.mark.parametrize("a_order,b_order,pad,off", [("row", "col", 0, 0), ("col", "row", 0, 0), ("row", "row", 3, 1),
                                                     ("col", "col", 5, 1), ("row", "col", 8, 8)])
@pytest.mark.parametrize("b_bf16", [0, 1])
def test_tc_gemm(M, N, K, a_order, b_order, pad, off, b_bf16):
    import torch
    from vulcan.gpu import _lib as KL
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    A = torch.randn(M, K, device="cuda", generator=g)
    B = torch.randn(K, N, device="cuda", generator=g)
    if b_bf16:
        B = B.to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g)
    a, (sam, sak) = _layout(torch, A, a_order, pad, off)
    b, (sbk, sbn) = _layout(torch, B, b_order, pad, off)
    L = KL.lib()
    ws = torch.empty(max(L.vk_tc_gemm_ws_floats(M, N, K), 1), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for scm, scn in ((N, 1), (N + 3, 1), (1, M)):     # aligned rows, odd rows, transposed
        C = torch.full((M * (N + 3),), 7.0, device="cuda")
        KL.check(L.vk_tc_gemm(M, N, K, KL.ptr(a), sam, sak, KL.ptr(b), b_bf16, sbk, sbn, KL.ptr(bias), 1, 0, KL.ptr(C),
                              scm, scn, KL.ptr(ws), ws.numel(), KL.ptr(status), KL.stream()), "tc_gemm")
        got = torch.as_strided(C, (M, N), (scm, scn)).double()
        a64, b64 = A.to(torch.bfloat16).double(), B.to(torch.bfloat16).double()
        want = (a64 @ b64 + bias.double()).clamp(min=0)
        # f32 accumulation: each of the K + splits + 1 additions rounds a partial sum of at most sum |a b| + |bias|
        bound = (K + 130) * 2.0 ** -24 * (a64.abs() @ b64.abs() + bias.abs().double()) * 2
        assert int(status.item()) == 0
        assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() - bound).max())


@pytest.mark.parametrize("M,N,K,sam,scm", [(1, 1, 1, 1, 1), (63, 1, 127, 127, 1), (64, 1, 128, 130, 2),
                                           (65, 1, 129, 129, 1), (200, 1, 256, 256, 1), (5, 4, 1, 1, 4),
                                           (130, 256, 1, 1, 260), (7, 6, 1, 1, 6), (7, 8, 1, 1, 9)])
@pytest.mark.parametrize("b_bf16,bias,relu,rnd", [(0, False, 0, 0), (1, True, 1, 0), (0, True, 0, 1)])
def test_layer3_gemm_equals_sequential_sums(M, N, K, sam, scm, b_bf16, bias, relu, rnd):
    import torch
    from vulcan.gpu import _lib as KL
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, sam)).astype(np.float32)
    B = torch.from_numpy(rng.standard_normal((K, N)).astype(np.float32))
    B = B.to(torch.bfloat16) if b_bf16 else B
    Bf, bv = B.float().numpy(), rng.standard_normal(N).astype(np.float32)
    acc = np.zeros((M, N), np.float32)
    for k in range(K):
        acc = acc + np.outer(A[:, k], Bf[k]).astype(np.float32)
    if bias:
        acc = acc + bv
    if relu:
        acc = np.maximum(acc, np.float32(0))
    want = torch.from_numpy(acc)
    if rnd:
        want = want.to(torch.bfloat16).float()
    a, b, bd = torch.from_numpy(A).cuda(), B.cuda().contiguous(), torch.from_numpy(bv).cuda()
    C = torch.full((M, scm), 7.0, device="cuda")
    KL.check(KL.lib().vk_gemm(M, N, K, KL.ptr(a), sam, 1, KL.ptr(b), b_bf16, N, 1, KL.ptr(bd) if bias else None, relu,
                              rnd, KL.ptr(C), scm, 1, KL.stream()), "gemm")
    assert torch.equal(C[:, :N].cpu(), want)
    assert bool((C[:, N:] == 7.0).all())


@pytest.mark.parametrize("sizes", [(1,), (256, 1, 4096), (65536, 256, 65536, 256, 256, 1), (5, 7, 300, 1, 2, 3, 4, 6)])
def test_adam_group_equals_adam(sizes):
    import ctypes as C

    import torch
    from vulcan.gpu import _lib as KL
    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    rnd = lambda n: torch.randn(n, device="cuda", generator=g)  # noqa: E731
    one = [[rnd(n), rnd(n), rnd(n) * 0.1, rnd(n).abs() * 0.01, torch.zeros(n, dtype=torch.bfloat16, device="cuda")]
           for n in sizes]
    two = [[x.clone() for x in t] for t in one]
    for step in (1, 2, 9):
        arr = (KL.AdamTensor * len(sizes))()
        for s, (p, gr, m, v, bf), k in zip(arr, two, range(len(sizes))):
            s.n, s.p, s.g, s.m, s.v = p.numel(), KL.ptr(p), KL.ptr(gr), KL.ptr(m), KL.ptr(v)
            s.p_bf16 = KL.ptr(bf) if k % 2 else None
        KL.check(KL.lib().vk_adam_group(C.byref(arr), len(sizes), 2e-3, 0.9, 0.999, 1e-8, step, 0.01, KL.stream()),
                 "adam")
        for k, (p, gr, m, v, bf) in enumerate(one):
            KL.check(KL.lib().vk_adam(p.numel(), KL.ptr(p), KL.ptr(gr), KL.ptr(m), KL.ptr(v), 2e-3, 0.9, 0.999, 1e-8,
                                      step, 0.01, KL.ptr(bf) if k % 2 else None, KL.stream()), "adam")
    for a, b in zip(one, two):
        assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("n,rows,width,off", [(1, 1, 16, 0), (1000, 333, 16, 0), (257, 5000, 16, 1), (64, 90, 6, 0)])
def test_gather_batch_equals_indexing(n, rows, width, off):
    import torch
    from vulcan.gpu import _lib as KL
    X = torch.randn(rows * width + off, device="cuda")[off:].view(rows, width)
    y, w = torch.randn(rows, device="cuda"), torch.randn(rows, device="cuda")
    idx = torch.randint(rows, (n,), device="cuda")
    out = [torch.zeros(n, width, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")]
    KL.check(KL.lib().vk_gather_batch(KL.ptr(idx), n, KL.ptr(X), width, KL.ptr(y), KL.ptr(w),
                                      *[KL.ptr(t) for t in out], KL.stream()), "gather_batch")
    for got, src in zip(out, (X, y, w)):
        assert torch.equal(got, src[idx])
