"""Weight gradients of few rows (act^T . err with up to 128 k) in one launch: edges of strips, blocks of columns and blocks of k, strips that
change in the middle of a CTA's work, any pitch and alignment.

Bound per element, of sum |a_k b_k|: TF32 parts leave 2^-22 of an element, the products of two low parts are left out (2^-22), and every product has
at most 32 additions truncated to 2^-23 (hi) or of the small sums (lo): 4.3e-6 + 4e-6, well inside the streaming kernel's 2.5e-5."""
import numpy as np
import pytest
import torch

from clusternet_b200 import _lib

pytestmark = pytest.mark.gpu
REL = 2.5e-5


def place(x, off):
    """torch (cols x rows: column-major rows x cols), its base `off` floats past a 16-byte boundary, between NaNs."""
    buf = torch.full((x.numel() + 64,), float("nan"), device="cuda")
    t = buf[32 + off:32 + off + x.numel()].view(x.shape)
    t.copy_(x)
    return t


# k: seventeen, a block of 32 k less one, whole ones, odd ones, all four; rows: eight, a strip and one more; columns: of one unit, of 16 units and one more;
# 60000 x 40, 100000 x 9: several strips of one block for every CTA, of two for 70; 4884 x 2576: 39 strips shared by all CTAs, some of whose strips end after one block; 9000 rows: 71 strips
SHAPES = [(8, 17, 150000), (129, 31, 33000), (2000, 32, 1700), (2001, 33, 1601), (1540, 64, 3500), (1000, 65, 4001), (1600, 96, 2000), (1537, 97, 2050), (2000, 128, 2000), (2049, 127, 1999),
          (60000, 64, 40), (100000, 96, 9), (60000, 20, 70), (4096, 128, 4096), (4884, 64, 2576), (4884, 127, 2577), (9000, 100, 520), (20000, 128, 17), (300, 128, 9001)]


@pytest.mark.parametrize("M,K,N", SHAPES)
@pytest.mark.parametrize("off", [(0, 0, 0), (1, 0, 1), (0, 3, 2)])
def test_weight_gradients_of_few_rows(ctx, M, K, N, off):
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    act, err = torch.randn(M, K, device="cuda", generator=g).clamp_(min=0), torch.randn(N, K, device="cuda", generator=g)
    err *= torch.exp(3 * torch.randn(N, K, device="cuda", generator=g))   # of very different size within a column
    buf = torch.full((N * M + 64,), 7.0, device="cuda")
    C = buf[32 + off[2]:32 + off[2] + N * M].view(N, M)
    a, w = place(act, off[0]), place(err, off[1])
    n0 = ctx.lib.cn_kernel_launches()
    ctx.gemm(a, w, out=C, transA=True)
    assert ctx.lib.cn_kernel_launches() - n0 == 1
    ctx.gemm_check()
    assert ctx.gemm_last_kernel() == "outer"
    assert bool((buf[:32 + off[2]] == 7.0).all()) and bool((buf[32 + off[2] + N * M:] == 7.0).all())   # nothing beside C
    ref, mag = err.double() @ act.double().t(), err.double().abs() @ act.double().t()
    assert bool(((C.double() - ref).abs() <= REL * mag).all())
    first = C.clone()
    ctx.gemm(a, w, out=C, transA=True)
    assert torch.equal(first, C)   # bit for bit the same again


def test_more_rows_than_a_32_bit_offset_in_bytes_reaches(ctx):
    """Rows from 2^30 on, and those that an offset which wraps would write in their place."""
    M, K, N = (1 << 30) + 300, 20, 1
    if torch.cuda.mem_get_info()[0] < 100e9:
        pytest.skip("needs 92 GB")
    act = torch.empty(M, K, device="cuda").normal_(generator=torch.Generator(device="cuda").manual_seed(5))
    err = torch.randn(N, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6))
    C = torch.full((N, M), 7.0, device="cuda")
    try:
        ctx.gemm(act, err, out=C, transA=True)
        ctx.gemm_check()
        assert ctx.gemm_last_kernel() == "outer"
        for r in (0, 1 << 20, (1 << 30) - 400, M - 400):
            a = act[r:r + 400].double()
            assert bool(((C[:, r:r + 400].double() - err.double() @ a.t()).abs() <= REL * (err.double().abs() @ a.abs().t())).all())
    finally:
        del act, err, C
        torch.cuda.empty_cache()


@pytest.mark.parametrize("off", [0, 1])
def test_non_finite_and_the_largest_finite_values_stay_in_their_row_and_column(ctx, off):
    """NaNs of any bit pattern and infinities of either operand; a value that rounds past the largest TF32 number stays finite."""
    rng = np.random.default_rng(3)
    M, K, N = 2500, 100, 1300
    a, b = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32)
    a[1000] = 0.0
    a[1000, 3], b[:, 3] = np.frombuffer(np.uint32(0x7f7fffff).tobytes(), np.float32)[0], 0.25
    for i, v in enumerate((0x7fffffff, 0xffffffff, 0x7fc00000, 0x7f800000)):
        a.view(np.uint32)[7 + i, 20 * i] = v
        b.view(np.uint32)[60 * i + 1, 11 + i] = v
    C = ctx.gemm(place(torch.from_numpy(a), off), place(torch.from_numpy(b), off), transA=True).cpu().numpy()
    ctx.gemm_check()
    assert ctx.gemm_last_kernel() == "outer"
    finite = np.isfinite(C)
    rows, cols = [1 + 60 * i for i in range(4)], [7 + i for i in range(4)]
    assert not finite[rows].any() and not finite[:, cols].any()
    rest = np.ones((N, M), bool)
    rest[rows], rest[:, cols] = False, False
    assert finite[rest].all()
    ok = [i for i in range(N) if i not in rows]
    assert np.abs(C[ok, 1000] / (np.float64(a[1000, 3]) * 0.25) - 1.0).max() <= REL


# what stays with the kernels it had: a bias, a unit, the single pass, other layouts, a longer K, one round of small products, few rows, a K of one addition
@pytest.mark.parametrize("M,K,N,kw", [(2000, 128, 2000, dict(bias=True)), (2000, 128, 2000, dict(activation=_lib.ACT_RELU)), (2000, 128, 2000, dict(mode=_lib.GEMM_TF32)),
                                      (2000, 128, 2000, dict(transA=False)), (2000, 128, 2000, dict(transB=True)), (2000, 129, 2000, {}), (784, 128, 1200, {}), (7, 128, 150000, {}), (4000, 16, 2000, {})])
def test_what_is_no_such_weight_gradient(ctx, M, K, N, kw):
    g = torch.Generator(device="cuda").manual_seed(1)
    kw = dict(transA=True, transB=False, **{k: v for k, v in kw.items() if k not in ("transA", "transB")}) | {k: v for k, v in kw.items() if k in ("transA", "transB")}
    if kw.pop("bias", False):
        kw["bias"] = torch.randn(N, device="cuda", generator=g)
    A, W = torch.randn((M, K) if kw["transA"] else (K, M), device="cuda", generator=g), torch.randn((K, N) if kw["transB"] else (N, K), device="cuda", generator=g)
    C = ctx.gemm(A, W, **kw)
    ctx.gemm_check()
    assert ctx.gemm_last_kernel() != "outer"
    ref = (W.double().t() if kw["transB"] else W.double()) @ (A.double().t() if kw["transA"] else A.double())
    if "bias" in kw:
        ref += kw["bias"].double()[:, None]
    if "activation" in kw:
        ref = ref.clamp(min=0)
    assert float((C.double() - ref).norm() / ref.norm()) <= (1e-3 if kw.get("mode") else 1e-6)


@pytest.mark.parametrize("M,K,N", [(300001, 17, 3), (200000, 33, 1), (90000, 126, 2)])
def test_few_columns_of_odd_pitch_stay_exact(ctx, M, K, N):
    """Products of two odd numbers of twelve bits: 24 bits, of which the last comes from the parts that eleven bits leave of either."""
    g = torch.Generator(device="cuda").manual_seed(M)
    act = torch.zeros(M, K, device="cuda")
    act[torch.arange(M, device="cuda"), torch.randint(0, K, (M,), device="cuda", generator=g)] = \
        2.0 * torch.randint(1024, 2048, (M,), device="cuda", generator=g).float() + 1.0
    err = 2.0 * torch.randint(1024, 2048, (N, K), device="cuda", generator=g).float() + 1.0
    C = ctx.gemm(act, err, transA=True)
    ctx.gemm_check()
    assert ctx.gemm_last_kernel() == "fma"
    assert torch.equal(C.double(), err.double() @ act.double().t())


# one part of K each with one and two chains, two parts with two chains; aligned and not
@pytest.mark.parametrize("M,K,N", [(4096, 128, 4096), (2001, 77, 3003), (1600, 96, 2000), (4096, 96, 4096), (4000, 20, 3000)])
@pytest.mark.parametrize("x", [-30, -34, -36, -37])
@pytest.mark.parametrize("which", [0, 1])
def test_operands_whose_low_parts_are_near_the_smallest_numbers(ctx, M, K, N, x, which):
    """Steps of 2^-146 leave 2^-148 on average, 2.8e-45: of variates of 1e-37 less than the 4.9e-8 that 22 bits leave.  Sums as ever: up to sixteen additions
    that truncate to 2^-23 of a sum which grows from nothing, a quarter of 16 * 2^-23 in the norm."""
    g = torch.Generator(device="cuda").manual_seed(K)
    scale = [1e36, 1e36]
    scale[which] = 10.0 ** x
    act, err = ((torch.randn(n, K, device="cuda", generator=g).double() * s).float() for n, s in ((M, scale[0]), (N, scale[1])))
    C = ctx.gemm(act, err, transA=True)
    ctx.gemm_check()
    assert ctx.gemm_last_kernel() == "outer"
    ref = err.double() @ act.double().t()
    assert float((C.double() - ref).norm() / ref.norm()) <= 4.8e-7 + 2 * 4.9e-8


@pytest.mark.parametrize("M,K,N", [(4096, 128, 4096), (2001, 77, 3003), (1600, 96, 2000)])
def test_the_largest_values_do_not_overflow(ctx, M, K, N):
    """Low parts are held times 2^10: three quarters of a product at most, of the lowest value of the type, too."""
    g = torch.Generator(device="cuda").manual_seed(K)
    act, err = torch.randn(M, K, device="cuda", generator=g), torch.rand(N, K, device="cuda", generator=g)
    act[:, K // 2] = torch.finfo(torch.float32).min
    act[::2, 1], err[1::2, 1] = torch.finfo(torch.float32).max, 0.0
    err[::2, 1] = 0.5 * err[::2, K // 2]
    C = ctx.gemm(act, err, transA=True)
    ctx.gemm_check()
    assert ctx.gemm_last_kernel() == "outer"
    ref, mag = err.double() @ act.double().t(), err.double().abs() @ act.double().abs().t()
    fits = mag < 3.4e38
    assert float(fits.float().mean()) > 0.5
    assert bool(((C.double() - ref).abs() <= REL * mag)[fits].all())


@pytest.mark.parametrize("M,K,N,level", [(300, 128, 9000, 4), (500, 33, 9000, 2), (2000, 128, 1200, 3), (401, 77, 7000, 7)])
def test_maxima_are_those_of_the_same_product(ctx, M, K, N, level):
    """Where a weight gradient stands in for a small product, it does so with a maxout behind it, too."""
    g = torch.Generator(device="cuda").manual_seed(K)
    act, err = torch.randn(M, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    plain = ctx.gemm(act, err, transA=True)
    assert ctx.gemm_last_kernel() == "outer"
    want, want_arg = ctx.maxout(plain, level)
    arg = torch.empty_like(want_arg)
    out = ctx.gemm(act, err, transA=True, maxout_level=level, argmax_out=arg)
    ctx.gemm_check()
    assert torch.equal(out, want) and torch.equal(arg, want_arg)


# as many additions to one sum as the kernels have that take such a product's neighbours, whose errors these are: two parts of K with two chains each,
# two chains (two, three and four blocks, halves of one in the middle), and one
@pytest.mark.parametrize("M,K,N,bound", [(2000, 128, 2000, 1.3e-7), (1600, 96, 2000, 1.3e-7), (4096, 96, 4096, 2.1e-7), (4001, 77, 4003, 2.1e-7), (6000, 64, 3500, 2.1e-7),
                                         (4001, 127, 4003, 2.1e-7), (4096, 128, 4096, 3.9e-7), (300, 128, 30000, 3.9e-7)])
def test_chains_are_as_short_as_those_of_the_kernels_beside(ctx, M, K, N, bound):
    g = torch.Generator(device="cuda").manual_seed(K)
    act, err = torch.rand(M, K, device="cuda", generator=g) * 2 - 1, torch.rand(N, K, device="cuda", generator=g) * 2 - 1
    C = ctx.gemm(act, err, transA=True)
    ctx.gemm_check()
    assert ctx.gemm_last_kernel() == "outer"
    ref = err.double() @ act.double().t()
    assert float((C.double() - ref).norm() / ref.norm()) <= bound


@pytest.mark.parametrize("M,K,N", [(2000, 128, 2000), (2049, 77, 1999), (4096, 96, 4096), (129, 31, 33000)])
@pytest.mark.parametrize("more", [(4, 4, 4), (5, 0, 3), (0, 1, 0)])
def test_columns_with_room_between_them(ctx, M, K, N, more):
    """Pitches beyond K and M; what lies between the columns is neither used nor written."""
    g = torch.Generator(device="cuda").manual_seed(M)
    act, err = (torch.full((n, K + d), float("nan"), device="cuda") for n, d in ((M, more[0]), (N, more[1])))
    act[:, :K], err[:, :K] = torch.randn(M, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    C = torch.full((N, M + more[2]), 7.0, device="cuda")
    assert ctx.lib.cn_gemm_f32(ctx.h, 1, 0, M, N, K, act.data_ptr(), K + more[0], err.data_ptr(), K + more[1], C.data_ptr(), M + more[2], None,
                               _lib.GEMM_3XTF32, ctx.stream_ptr()) == 0
    ctx.gemm_check()
    assert ctx.gemm_last_kernel() == "outer"
    a, w = act[:, :K].double(), err[:, :K].double()
    assert bool(((C[:, :M].double() - w @ a.t()).abs() <= REL * (w.abs() @ a.abs().t())).all())
    assert bool((C[:, M:] == 7.0).all())
