"""Edges of the product kernels' dispatch: the one-launch kernel for small products (any layout and alignment, K over a
cluster), the operand parts of the streaming kernel, and its weights of any pitch, against an fp64 product.

Bound of an element, with s = sum over k of |a_k b_k|.  3x mode: what the split leaves out is below 2^-21 of each product, and a
chain of at most 512 k accumulates at most 12 products per 32 k, each addition truncated to 2^-23 of a running sum that is at most
s: 192 * 2^-23 s = 2.3e-5 s.  Single pass: both operands rounded to 11 bits, 2^-10 s.  These bounds hold for any signs and are loose
for random ones, so the streaming kernel is also held to a 2-norm and to sums of a single term."""
import numpy as np
import pytest
import torch

from clusternet_b200 import _lib
from oracle import oracle

pytestmark = pytest.mark.gpu

REL_3X, REL_1X = 2.5e-5, 1.05e-3


def place(x, off):
    """Row-major numpy (rows x cols) -> column-major device matrix whose base lies `off` floats past a 16-byte boundary."""
    rows, cols = x.shape
    t = torch.zeros(rows * cols + 4, device="cuda")[off:off + rows * cols].view(cols, rows)
    t.copy_(torch.from_numpy(np.ascontiguousarray(x.T)))
    return t


def check(C, A, B, transA, transB, rel):
    a, b = (A.T if transA else A).astype(np.float64), (B.T if transB else B).astype(np.float64)
    err = np.abs(C.T.cpu().numpy().astype(np.float64) - a @ b)
    bound = rel * (np.abs(a) @ np.abs(b))
    assert np.all(err <= bound), float((err / np.maximum(bound, 1e-300)).max())


# one row, one column, one k-step; tile edges; odd pitches; one CTA per tile, clusters; several accumulation chains
SMALL = [(1, 4096, 1), (17, 33, 15), (128, 31, 128), (129, 97, 127), (127, 1201, 129), (128, 785, 1201), (1201, 128, 1201), (203, 2049, 301),
         (16, 8193, 100), (500, 130, 64)]


@pytest.mark.parametrize("M,K,N", SMALL)
@pytest.mark.parametrize("transA,transB", [(False, False), (True, False), (False, True), (True, True)])
def test_small_products_in_every_layout(ctx, M, K, N, transA, transB):
    rng = np.random.default_rng(M + 3 * K + 5 * N)
    A = rng.standard_normal((K, M) if transA else (M, K)).astype(np.float32)
    B = rng.standard_normal((N, K) if transB else (K, N)).astype(np.float32)
    for off in (0, 1):
        aligned = off == 0 and (N if transB else K) % 4 == 0
        for mode, rel in ((_lib.GEMM_3XTF32, REL_3X), (_lib.GEMM_TF32, REL_1X if aligned else REL_3X)):
            if not aligned and M * N * K < 4096:
                continue
            C = torch.full((N, M), float("nan"), device="cuda")
            ctx.gemm(place(A, off), place(B, off), out=C, transA=transA, transB=transB, mode=mode)
            ctx.gemm_check()
            assert ctx.gemm_last_path().startswith("tcgen05")
            check(C, A, B, transA, transB, rel)


# tiles of 32, 64 and 128 columns, by one CTA and by clusters; more blocks than accumulators
@pytest.mark.parametrize("M,K,N", [(48, 80, 1091), (128, 1200, 10), (1200, 128, 10), (784, 128, 1200), (32, 500, 500), (1200, 120, 1201), (512, 500, 1000), (128, 785, 1100),
                                   (200, 380, 2100), (64, 3000, 600)])
@pytest.mark.parametrize("act", [_lib.ACT_LINEAR, _lib.ACT_RELU, _lib.ACT_LOGISTIC])
def test_small_products_of_every_tile(ctx, M, K, N, act):
    """Bias and activation in both ends of the kernel, the same bits twice; 2-norm of the 3x mode's linear product against the error of
    fp32 sums (random rounding of two TF32 parts, 2^-23, and of 8 sequential additions per chain: 4e-7)."""
    rng = np.random.default_rng(M + K + N)
    A, B, b = rng.uniform(-1, 1, (M, K)).astype(np.float32), rng.uniform(-1, 1, (K, N)).astype(np.float32), rng.uniform(-1, 1, N).astype(np.float32)
    n0 = ctx.lib.cn_kernel_launches()
    C, C2 = (ctx.gemm(place(A, 0), place(B, 0), bias=torch.from_numpy(b).cuda(), activation=act) for _ in range(2))
    assert ctx.lib.cn_kernel_launches() - n0 == 2
    ctx.gemm_check()
    assert torch.equal(C, C2)
    ref, bound = A.astype(np.float64) @ B + b, REL_3X * (np.abs(A).astype(np.float64) @ np.abs(B) + np.abs(b))
    got = C.T.cpu().numpy().astype(np.float64)
    if act == _lib.ACT_LINEAR:
        assert np.linalg.norm(got - ref) <= 4e-7 * np.linalg.norm(ref)
    want = {_lib.ACT_LINEAR: ref, _lib.ACT_RELU: np.maximum(ref, 0), _lib.ACT_LOGISTIC: 1 / (1 + np.exp(-ref))}[act]
    assert np.all(np.abs(got - want) <= bound + 1e-7)


# clusters of 3, 5, 6 and 7 CTAs (tiles of 32, 64 and 128 columns), whose last CTAs finish fewer columns than the others, or none; last
# tiles of a few columns, the last four of them not whole
@pytest.mark.parametrize("M,K,N", [(149, 206, 352), (128, 614, 234), (253, 277, 1373), (100, 784, 1030), (137, 811, 615), (18, 1047, 507), (282, 580, 1467),
                                   (328, 1561, 472), (300, 600, 601), (128, 460, 33)])
@pytest.mark.parametrize("act", [_lib.ACT_LINEAR, _lib.ACT_RELU, _lib.ACT_LOGISTIC])
def test_small_products_over_clusters_of_any_size(ctx, M, K, N, act):
    rng = np.random.default_rng(M + K + N)
    A, B = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    bias = torch.from_numpy(rng.standard_normal(N).astype(np.float32)).cuda()
    buf = torch.full((N + 1, M), 7.0, device="cuda")
    C = buf[:N]
    ctx.gemm(place(A, 0), place(B, 0), out=C, bias=bias, activation=act)
    ctx.gemm_check()
    assert ctx.gemm_last_kernel() == "small"
    assert bool((buf[N] == 7.0).all())   # nothing behind the last column
    z = A.astype(np.float64) @ B.astype(np.float64) + bias.cpu().numpy().astype(np.float64)
    want = z if act == _lib.ACT_LINEAR else np.maximum(z, 0.0) if act == _lib.ACT_RELU else 1.0 / (1.0 + np.exp(-z))
    # the units' slopes are at most 1; the bias and the unit are rounded once each
    bound = REL_3X * (np.abs(A.astype(np.float64)) @ np.abs(B.astype(np.float64))) + 2.0 ** -22 * (np.abs(z) + 1.0)
    assert np.all(np.abs(C.T.cpu().numpy() - want) <= bound)


@pytest.mark.parametrize("mode", [_lib.GEMM_3XTF32, _lib.GEMM_TF32])
@pytest.mark.parametrize("transA,transB", [(False, False), (True, False), (False, True)])
@pytest.mark.parametrize("wide", ["A", "B"])
@pytest.mark.parametrize("M,K,N,off", [(130, 4100, 1028, 0), (64, 40000, 100, 0), (130, 4100, 1028, 1), (64, 40001, 101, 0)])
def test_streaming_product_of_single_terms(ctx, M, K, N, off, wide, transA, transB, mode):
    """One operand has elements over many binades beside each other, the other one nonzero element per row or column, so every output
    is one product.  3x: 2^-20 for what the parts of each operand may leave, 2^-22 for the product of the low parts, four additions
    truncated to 2^-23; high parts alone would leave 2^-11.  Single pass: 2^-10 for what is left of the wide operand, 2^-11 for the
    other one's rounding."""
    rng = np.random.default_rng(K + N + transB)
    binades = 45 if wide == "A" else 60                            # activations: 2^97 in all, weights: any
    A = rng.uniform(1.0, 2.0, (M, K)) * rng.choice([-1.0, 1.0], (M, K))
    W = rng.uniform(1.0, 2.0, (K, N)) * rng.choice([-1.0, 1.0], (K, N))
    if wide == "A":
        at = rng.integers(0, K, N)
        W *= np.arange(K)[:, None] == at
        A *= np.exp2(rng.integers(-binades, binades, (M, K)))
    else:
        at = rng.integers(0, K, M)
        A *= np.arange(K) == at[:, None]
        W *= np.exp2(rng.integers(-binades, binades, (K, N)))
    A, W = A.astype(np.float32), W.astype(np.float32)
    n0 = ctx.lib.cn_kernel_launches()
    C = ctx.gemm(place(np.ascontiguousarray(A.T) if transA else A, 0), place(np.ascontiguousarray(W.T) if transB else W, off), transA=transA,
                 transB=transB, mode=mode).T.cpu().numpy().astype(np.float64)
    assert ctx.lib.cn_kernel_launches() - n0 > 1                   # planes and product at least
    assert ctx.gemm_last_kernel() == "streaming"
    ctx.gemm_check()
    A, W = A.astype(np.float64), W.astype(np.float64)
    ref = A[:, at] * W[at, np.arange(N)] if wide == "A" else A[np.arange(M), at][:, None] * W[at]
    bound = 2.7e-6 if mode == _lib.GEMM_3XTF32 or off or (N if transB else K) % 4 else 2.0 ** -10 + 2.0 ** -11 + 2.0 ** -20
    assert float((np.abs(C - ref) / np.abs(ref)).max()) <= bound


@pytest.mark.parametrize("mode,rel", [(_lib.GEMM_3XTF32, 8e-6), (_lib.GEMM_TF32, 1e-3)])
@pytest.mark.parametrize("transB", [False, True])
@pytest.mark.parametrize("outlier", [1.0, 2.0 ** 20, 2.0 ** 30, 2.0 ** 40])
def test_streaming_product_with_large_elements_opposite_zeros(ctx, outlier, transB, mode, rel):
    """Activations and weights of very different size in one row or column, the large ones opposite zeros: the small ones are the whole
    result.  2-norm of every row and column; 3x: four times the 1.9e-6 of random operands of one size."""
    rng = np.random.default_rng(3)
    M, K, N = 128, 4096, 1024
    A, W = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    ka, kw = np.arange(5, K, 64), np.arange(37, K, 64)
    A[:, ka], W[ka, :] = A[:, ka] * outlier, 0.0
    W[kw, :], A[:, kw] = W[kw, :] * outlier, 0.0
    A, W = A.astype(np.float32), W.astype(np.float32)
    B = np.ascontiguousarray(W.T) if transB else W
    C = ctx.gemm(place(A, 0), place(B, 0), transB=transB, mode=mode).T.cpu().numpy().astype(np.float64)
    ctx.gemm_check()
    ref = A.astype(np.float64) @ W.astype(np.float64)
    for axis in (0, 1):
        assert float((np.linalg.norm(C - ref, axis=axis) / np.linalg.norm(ref, axis=axis)).max()) <= rel


@pytest.mark.parametrize("transB", [False, True])
@pytest.mark.parametrize("M,K,N", [(128, 8192, 512), (300, 5000, 2052)])
def test_streaming_product_of_rows_whose_magnitudes_change(ctx, M, K, N, transB):
    """Weights that grow along k, start with zeros, or fall; activation rows of very different size."""
    rng = np.random.default_rng(N)
    A = rng.uniform(0.25, 1.0, (M, K)) * rng.choice([-1.0, 1.0], (M, K)) * np.exp2(rng.integers(-30, 30, (M, 1)))
    W = rng.uniform(0.5, 1.0, (K, N)) * rng.choice([-1.0, 1.0], (K, N))
    seg = np.arange(K) // 512
    W[:, 1::4] *= np.exp2((np.arange(K) % 512) // 40)[:, None]                   # grows 2^12-fold within every segment
    W[:, 2::4] *= np.exp2(-3.0 * seg)[:, None]                                   # falls from segment to segment
    W[:, 3::4] *= ((np.arange(K) % 512 > 100) & (seg % 2 == 0))[:, None]         # zeros first, then whole segments of zeros
    A, W = A.astype(np.float32), W.astype(np.float32)
    B = np.ascontiguousarray(W.T) if transB else W
    C = ctx.gemm(place(A, 0), place(B, 0), transB=transB)
    ctx.gemm_check()
    check(C, A, B, False, transB, REL_3X)


def test_streaming_product_keeps_non_finite_values_to_their_row_and_column(ctx):
    rng = np.random.default_rng(5)
    M, K, N = 128, 6000, 1028
    A, W = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    clean = ctx.gemm(place(A, 0), place(W, 0)).clone()
    A2, W2 = A.copy(), W.copy()
    A2[7, 900], A2[9, 5000] = np.nan, np.inf
    W2[31, 3], W2[5999, 600] = np.inf, np.nan
    C = ctx.gemm(place(A2, 0), place(W2, 0))
    ctx.gemm_check()
    hit = torch.zeros(N, M, dtype=torch.bool, device="cuda")
    hit[:, [7, 9]] = True
    hit[[3, 600], :] = True
    assert not torch.isfinite(C[hit]).any()
    assert torch.equal(C[~hit], clean[~hit])


@pytest.mark.parametrize("transA,transB", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("off", [0, 1])
def test_small_products_keep_non_finite_and_the_largest_finite_values(ctx, transA, transB, off):
    """NaNs of any bit pattern (0x7fffffff is the one that GPU arithmetic makes) and infinities in either operand stay in their row
    or column and make it non-finite; a value that rounds past the largest TF32 number stays finite in the 3x mode."""
    rng = np.random.default_rng(11)
    M, K, N = 128, 785, 300
    A = rng.standard_normal((K, M) if transA else (M, K)).astype(np.float32)
    B = rng.standard_normal((N, K) if transB else (K, N)).astype(np.float32)
    a, b = (A.T if transA else A), (B.T if transB else B)          # views: op(A)(m, k), op(B)(k, n)
    a[100] = 0.0
    a[100, 3], b[3, :] = np.frombuffer(np.uint32(0x7f7fffff).tobytes(), np.float32)[0], 0.25
    bad = np.frombuffer(np.array([0x7fffffff, 0xffffffff, 0x7fc00000, 0x7f800000], np.uint32).tobytes(), np.float32)
    for i, v in enumerate(bad):
        a.view(np.uint32)[7 + i, 50 * i] = v.view(np.uint32)
        b.view(np.uint32)[60 * i + 1, 11 + i] = v.view(np.uint32)
    for mode in (_lib.GEMM_3XTF32, _lib.GEMM_TF32):
        n0 = ctx.lib.cn_kernel_launches()
        C = ctx.gemm(place(A, off), place(B, off), transA=transA, transB=transB, mode=mode).T.cpu().numpy()
        assert ctx.lib.cn_kernel_launches() - n0 == 1              # the one-launch kernel
        ctx.gemm_check()
        finite = np.isfinite(C)
        assert not finite[7:11].any() and not finite[:, 11:15].any()
        rest = np.ones((M, N), bool)
        rest[7:11], rest[:, 11:15] = False, False
        assert finite[rest].all()
        assert np.allclose(C[100][rest[100]], a[100, 3].astype(np.float64) * 0.25, rtol=REL_1X)


@pytest.mark.parametrize("M,K,N", [(203, 4001, 3001), (5, 2049, 1031), (128, 20003, 131), (300, 130, 20005), (128, 4002, 1026), (64, 5, 500001), (70, 40001, 101)])
@pytest.mark.parametrize("transB", [False, True])
@pytest.mark.parametrize("off", [0, 1, 2, 3])
def test_streaming_weights_of_any_pitch_and_alignment(ctx, M, K, N, transB, off):
    """The four classes of rows of a matrix whose rows TMA cannot read one by one; what lies in front of and behind it is NaN."""
    g = torch.Generator(device="cuda")
    g.manual_seed(M + K + N)
    A = torch.randn((K, M), device="cuda", generator=g)
    inner, outer = (N, K) if transB else (K, N)
    buf = torch.full((inner * outer + 64,), float("nan"), device="cuda")
    W = buf[32 + off:32 + off + inner * outer].view(outer, inner)
    W.copy_(torch.randn((outer, inner), device="cuda", generator=g))
    bias = torch.randn(N, device="cuda", generator=g)
    C = torch.full((N, M), float("nan"), device="cuda")
    ctx.gemm(A, W, out=C, transB=transB, bias=bias, activation=_lib.ACT_RELU)
    ctx.gemm_check()
    assert ctx.gemm_last_path() == "tcgen05_3xtf32"
    Wd, Ad = (W.T if transB else W).double(), A.double()
    ref = torch.relu(Wd @ Ad + bias.double()[:, None])
    bound = REL_3X * (Wd.abs() @ Ad.abs() + bias.double().abs()[:, None])
    assert bool(((C.double() - ref).abs() <= bound).all())
    # the single-pass mode does not make such weights less exact than they were on the fp32 kernel
    C1 = ctx.gemm(A, W, transB=transB, bias=bias, activation=_lib.ACT_RELU, mode=_lib.GEMM_TF32)
    if off or inner % 4:
        assert torch.equal(C1, C)


@pytest.mark.parametrize("M,K,N", [(128, 257, 201), (128, 785, 1201), (203, 2001, 301), (500, 2001, 999), (1280, 2047, 1023), (70, 40001, 101)])
@pytest.mark.parametrize("transB", [False, True])
def test_weights_of_odd_pitch_are_as_exact_as_on_the_fp32_kernel(ctx, M, K, N, transB):
    """2-norm against fp64, small and streaming kernel, beside the fp32 kernel's on the same operands, whose own error scatters by some
    per cent of it and by the last bit of the result (6e-8)."""
    rng = np.random.default_rng(M + K + N)
    A, W = rng.uniform(-1, 1, (M, K)).astype(np.float32), rng.uniform(-1, 1, (K, N)).astype(np.float32)
    dA, dW = place(A, 0), place(np.ascontiguousarray(W.T) if transB else W, 1)
    ref = A.astype(np.float64) @ W.astype(np.float64)
    err = [np.linalg.norm(ctx.gemm(dA, dW, transB=transB, mode=m).T.cpu().numpy() - ref) / np.linalg.norm(ref)
           for m in (_lib.GEMM_3XTF32, _lib.GEMM_FP32_SIMT)]
    ctx.gemm_check()
    assert err[0] <= 1.1 * err[1] + 6e-8, err


@pytest.mark.parametrize("M,K,N", [(768, 3873, 335), (256, 3617, 527), (2059, 1299, 98), (24, 653, 2271)])
@pytest.mark.parametrize("transB", [False, True])
def test_small_products_of_odd_pitch_with_the_longest_chains(ctx, M, K, N, transB):
    """Shapes at which the fastest tiles and clusters would have the longest accumulation chains of the small products' kernel; 2-norm no
    larger than the fp32 kernel's.  (The operands are fixed, so are both errors.)"""
    rng = np.random.default_rng(M + K + N)
    A, W = rng.uniform(-1, 1, (M, K)).astype(np.float32), rng.uniform(-1, 1, (K, N)).astype(np.float32)
    dA, dW = place(A, 0), place(np.ascontiguousarray(W.T) if transB else W, 1)
    ref = A.astype(np.float64) @ W.astype(np.float64)
    n0 = ctx.lib.cn_kernel_launches()
    err = [np.linalg.norm(ctx.gemm(dA, dW, transB=transB, mode=m).T.cpu().numpy() - ref) / np.linalg.norm(ref)
           for m in (_lib.GEMM_3XTF32, _lib.GEMM_FP32_SIMT)]
    assert ctx.lib.cn_kernel_launches() - n0 == 2                  # one launch each: the small products' kernel
    ctx.gemm_check()
    assert err[0] <= err[1], err


@pytest.mark.parametrize("level", [2, 8, 32])
@pytest.mark.parametrize("M,K,N,full", [(128, 320, 40960, True), (130, 4100, 1024, False)])
def test_maxout_fused_into_the_streaming_kernel(ctx, level, M, K, N, full):
    """The shuffle tree over the drain warps' sums: two tiles per CTA, a ragged second tile of rows, bias.  Where the product without
    maxout is not cut along K either (full), its maxima exactly."""
    rng = np.random.default_rng(level + N)
    A, B = rng.uniform(-1, 1, (M, K)).astype(np.float32), rng.uniform(-1, 1, (K, N)).astype(np.float32)
    dA, dB, db = ctx.colmajor(A), ctx.colmajor(B), torch.from_numpy(rng.uniform(-1, 1, N).astype(np.float32)).cuda()
    arg = ctx.empty(M, N // level)
    n0 = ctx.lib.cn_kernel_launches()
    out = ctx.gemm(dA, dB, bias=db, maxout_level=level, argmax_out=arg)
    assert ctx.lib.cn_kernel_launches() - n0 == 2                  # planes and product: no separate reduction
    out = ctx.to_numpy(out)
    plain = ctx.to_numpy(ctx.gemm(dA, dB, bias=db))
    ctx.gemm_check()
    wv, wi = oracle.maxout(plain, level)
    if full:
        assert np.array_equal(out, wv) and np.array_equal(ctx.to_numpy(arg), wi)
    else:
        got = ctx.to_numpy(arg).astype(np.int64)
        assert np.array_equal(got // level, np.broadcast_to(np.arange(N // level), got.shape))
        bound = REL_3X * (np.abs(A) @ np.abs(B)).max()
        assert np.abs(out - wv).max() <= bound
        assert np.abs(np.take_along_axis(plain, got, 1) - out).max() <= bound


@pytest.mark.parametrize("M,K,N", [(5, 20000, 70), (128, 8000, 300), (260, 12000, 130)])
@pytest.mark.parametrize("nt", [1, 2])
def test_few_tiles_in_many_runs(ctx, M, K, N, nt):
    """The reduction with eight columns per CTA: remainders of rows, columns and partial tiles; bit for bit the same twice."""
    from clusternet_b200 import check as status
    rng = np.random.default_rng(M + N)
    A, B = rng.uniform(-1, 1, (M, K)).astype(np.float32), rng.uniform(-1, 1, (K, N)).astype(np.float32)
    bias = torch.from_numpy(rng.uniform(-1, 1, N).astype(np.float32)).cuda()
    dA, dB = ctx.colmajor(A), ctx.colmajor(B)
    status(ctx.lib.cn_gemm_set_tuning(ctx.h, nt, 0, 0))
    try:
        C, C2 = (ctx.gemm(dA, dB, bias=bias, activation=_lib.ACT_RELU) for _ in range(2))
        ctx.gemm_check()
    finally:
        status(ctx.lib.cn_gemm_set_tuning(ctx.h, 0, 0, 0))
    assert torch.equal(C, C2)
    ref = np.maximum(A.astype(np.float64) @ B.astype(np.float64) + bias.cpu().numpy(), 0)
    assert np.linalg.norm(ctx.to_numpy(C) - ref) <= 8e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("M", [1, 3, 4, 5, 31, 127, 129, 133, 255, 257])
@pytest.mark.parametrize("N,nt,splits", [(270, 1, 3), (270, 2, 9), (5000, 1, 2)])
def test_rows_that_partial_tiles_do_not_have(ctx, M, N, nt, splits):
    """Neither written nor read, with 8 or 32 columns per CTA of the reduction: what an earlier product of whole tiles left there, NaN, must not show."""
    from clusternet_b200 import check as status
    rng = np.random.default_rng(M)
    A, B = rng.uniform(-1, 1, (M, 3000)).astype(np.float32), rng.uniform(-1, 1, (3000, N)).astype(np.float32)
    status(ctx.lib.cn_gemm_set_tuning(ctx.h, nt, splits, 0))
    try:
        dB = place(B, 0)
        ctx.gemm(torch.full((3000, (M + 127) // 128 * 128), float("nan"), device="cuda"), dB)
        C = ctx.gemm(place(A, 0), dB)
        ctx.gemm_check()
    finally:
        status(ctx.lib.cn_gemm_set_tuning(ctx.h, 0, 0, 0))
    check(C, A, B, False, False, REL_3X)


@pytest.mark.parametrize("mode,rel", [(_lib.GEMM_3XTF32, REL_3X), (_lib.GEMM_TF32, REL_1X)])
@pytest.mark.parametrize("half", [0, 1])
@pytest.mark.parametrize("M,N,splits", [(128, 256, 7), (200, 1000, 13), (16, 100, 37)])
def test_runs_that_begin_or_end_inside_a_stage_with_left_overs(ctx, M, N, splits, half, mode, rel):
    """Runs of eleven blocks of 32 k, stages of two: the half of a stage that a run does not take has elements that band 0 cannot hold,
    its own half has none, so nothing multiplies the stage's other bands and their copies have to be waited for all the same."""
    from clusternet_b200 import check as status
    K = 32 * 11 * splits
    rng = np.random.default_rng(M + half)
    A, W = rng.uniform(0.5, 1, (M, K)).astype(np.float32), rng.uniform(-1, 1, (K, N)).astype(np.float32)
    for k0 in range(32 * half, K, 64):
        A[::16, k0:k0 + 3] *= 2.0 ** -30                            # something in band 1 ...
        A[5::16, k0 + 7:k0 + 9] *= np.float32(2.0 ** -60)           # ... and in band 2
        A[5::16, k0 + 9] *= np.float32(2.0 ** -30)
    dA, dW = ctx.colmajor(A), ctx.colmajor(W)
    status(ctx.lib.cn_gemm_set_tuning(ctx.h, 0, splits, 0))
    try:
        out = [ctx.gemm(dA, dW, mode=mode).clone() for _ in range(20)]
        ctx.gemm_check()
    finally:
        status(ctx.lib.cn_gemm_set_tuning(ctx.h, 0, 0, 0))
    assert all(torch.equal(o, out[0]) for o in out)
    check(out[0], A, W, False, False, rel)


@pytest.mark.parametrize("rows,cols", [(1, 300001), (3, 1001), (16, 40000), (1023, 7), (1024, 7), (1500, 3)])
def test_bias_activation_of_any_shape(ctx, rows, cols):
    rng = np.random.default_rng(rows)
    A, b = rng.standard_normal((rows, cols)).astype(np.float32), rng.standard_normal(cols).astype(np.float32)
    got = ctx.bias_activation(ctx.colmajor(A), torch.from_numpy(b).cuda(), _lib.ACT_RELU)
    assert np.array_equal(ctx.to_numpy(got), np.maximum(A + b, 0))
    got = ctx.bias_activation(ctx.colmajor(A), None, _lib.ACT_DOUBLE_RELU)
    assert np.array_equal(ctx.to_numpy(got), np.clip(A, 0, 1))


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 262147])
@pytest.mark.parametrize("off", [0, 1])
def test_elementwise_tails_and_alignment(ctx, n, off):
    """16-byte accesses on aligned buffers, single elements on the others and for the remainder."""
    rng = np.random.default_rng(n)
    host = [rng.standard_normal(n).astype(np.float32) for _ in range(3)]
    dev = [torch.zeros(n + 4, device="cuda") for _ in range(4)]
    g, w, r, out = (t[off:off + n] for t in dev)
    sp = ctx.stream_ptr()
    for t, h in zip((g, w), host):
        t.copy_(torch.from_numpy(h))
    rms = np.abs(host[2]) + np.float32(0.1)
    r.copy_(torch.from_numpy(rms))
    assert ctx.lib.cn_mul_activation_gradient(ctx.h, g.data_ptr(), w.data_ptr(), _lib.ACT_RELU, None, out.data_ptr(), n, sp) == 0
    assert np.array_equal(out.cpu().numpy(), host[0] * (host[1] > 0).astype(np.float32))
    assert ctx.lib.cn_dropout(ctx.h, w.data_ptr(), out.data_ptr(), n, 0.5, 3, 0, sp) == 0
    kept = out.cpu().numpy()
    assert np.all((kept == host[1]) | (kept == 0))
    w2, aligned = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    w2.copy_(w)
    assert ctx.lib.cn_dropout(ctx.h, w2.data_ptr(), aligned.data_ptr(), n, 0.5, 3, 0, sp) == 0
    assert torch.equal(aligned, out)                                             # the mask does not depend on the alignment
    assert ctx.lib.cn_rmsprop_update(ctx.h, r.data_ptr(), g.data_ptr(), w.data_ptr(), 0.9, 0.01, n, sp) == 0
    want_r, want_w = oracle.rmsprop_update(rms, host[0], host[1], 0.9, 0.01)
    assert np.abs(r.cpu().numpy() - want_r).max() <= 1e-6 * np.abs(want_r).max()
    assert np.abs(w.cpu().numpy() - want_w).max() <= 2e-6
    for t in dev:                                                                # nothing outside the buffers
        assert float(t[:off].abs().sum()) == 0 and float(t[off + n:].abs().sum()) == 0


@pytest.mark.parametrize("cols", [1, 31, 32, 33])
def test_softmax_at_the_edge_of_the_register_rows(ctx, cols):
    A = (np.random.default_rng(cols).standard_normal((65, cols)) * 3).astype(np.float32)
    out = ctx.empty(65, cols)
    assert ctx.lib.cn_softmax(ctx.h, place(A, 0).data_ptr(), out.data_ptr(), 65, cols, ctx.stream_ptr()) == 0
    assert np.abs(ctx.to_numpy(out) - oracle.softmax_rows(A)).max() < 2e-6       # __expf against libm's exp


@pytest.mark.parametrize("cols", [1, 2, 10, 31, 32])
@pytest.mark.parametrize("rows", [1, 5, 4095])
def test_softmax_of_few_rows_gives_the_bits_of_many(ctx, rows, cols):
    """A warp per row against a thread per row, with infinities and NaN among the values, in place and with the error."""
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    big = torch.randn((cols, 4096 + rows), device="cuda", generator=g) * 5
    big[0, 0], big[-1, 0], big[0, min(2, rows - 1)], big[-1, min(3, rows - 1)] = float("inf"), float("nan"), float("-inf"), -1e38
    labels = torch.randint(0, cols, (4096 + rows,), device="cuda", generator=g).float()
    few, want, want_err, err = big[:, :rows].contiguous(), torch.empty_like(big), torch.empty_like(big), torch.empty((cols, rows), device="cuda")
    lib, h, s = ctx.lib, ctx.h, ctx.stream_ptr()
    assert lib.cn_softmax_error(h, big.data_ptr(), labels.data_ptr(), want.data_ptr(), want_err.data_ptr(), 4096 + rows, cols, s) == 0
    assert lib.cn_softmax_error(h, few.data_ptr(), labels.data_ptr(), few.data_ptr(), err.data_ptr(), rows, cols, s) == 0
    assert torch.equal(few.view(torch.int32), want[:, :rows].contiguous().view(torch.int32))
    assert torch.equal(err.view(torch.int32), want_err[:, :rows].contiguous().view(torch.int32))


# tiles whose K a cluster of CTAs shares (one tile of rows, short K, weights beyond the small products'): one and two tiles of columns per CTA,
# clusters of 2 to 8, rows that give some CTAs nothing to finish, last tiles of few columns; weights of either layout and of odd pitch
SHARED = [(24, 560, 5192), (100, 1500, 2500), (128, 1024, 3000), (17, 640, 9001), (128, 2000, 8000), (1, 992, 6000), (72, 912, 3624), (120, 777, 4099), (97, 528, 7258)]


@pytest.mark.parametrize("M,K,N", SHARED)
@pytest.mark.parametrize("transA,transB", [(False, False), (True, True)])
@pytest.mark.parametrize("act,mode", [(_lib.ACT_LINEAR, _lib.GEMM_3XTF32), (_lib.ACT_LOGISTIC, _lib.GEMM_3XTF32), (_lib.ACT_RELU, _lib.GEMM_TF32)])
def test_tiles_shared_by_clusters(ctx, M, K, N, transA, transB, act, mode):
    """Elements of very different size among them: what the parts leave is in chains of its own."""
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    A, W = torch.randn(M, K, device="cuda", generator=g), torch.randn(K, N, device="cuda", generator=g)
    A[0, ::7] *= 2.0 ** -30
    W[::5, N - 1] *= 2.0 ** -30
    bias = torch.randn(N, device="cuda", generator=g)
    buf = torch.full((N + 1, M), 7.0, device="cuda")
    a, w = (A if transA else A.t()).contiguous(), (W if transB else W.t()).contiguous()
    n0 = ctx.lib.cn_kernel_launches()
    for rep in range(2):
        ctx.gemm(a, w, out=buf[:N], transA=transA, transB=transB, bias=bias, activation=act, mode=mode)
        if rep == 0:
            first = buf.clone()
    assert ctx.lib.cn_kernel_launches() - n0 == 4   # planes and product: no reduction
    ctx.gemm_check()
    assert ctx.gemm_last_kernel() == "streaming"
    assert torch.equal(first, buf) and bool((buf[N] == 7.0).all())
    z = A.double() @ W.double() + bias.double()
    want = {_lib.ACT_LINEAR: z, _lib.ACT_LOGISTIC: torch.sigmoid(z), _lib.ACT_RELU: z.clamp(min=0)}[act]
    aligned = (N if transB else K) % 4 == 0
    rel = REL_1X if mode == _lib.GEMM_TF32 and aligned else REL_3X
    bound = rel * (A.double().abs() @ W.double().abs()) + 2.0 ** -22 * (z.abs() + 1.0)
    assert bool(((buf[:N].t().double() - want).abs() <= bound).all())
