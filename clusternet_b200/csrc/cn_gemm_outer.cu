// Weight gradients of batches of up to 128 rows for sm_100a: act^T . err, an inner dimension K <= 128 that lies contiguous in both operands, and a large
// output.  One launch, both operands split in the kernel.
//
// As planes (cn_gemm_planes.cu) such a product took three launches, the first of which moves both operands through memory for a K that a CTA
// multiplies in a microsecond, and whose drain warps load scales and look for left-overs for every tile; with weights of odd pitch, or below 2^30
// multiplications, the streaming kernel, which splits every weight anew for each 128 rows and ends its chains every 32 k.  Here
//   * a persistent CTA keeps a strip of 128 rows m, all of K, as TF32 hi / lo parts in tensor memory and walks over blocks of 64 columns n.
//     Sixteen warps do the same work in step: they read a finished block out of its accumulator and store it, split the block of the weights
//     that takes its place in shared memory, and load the one after that from global memory, aligned or not;
//   * two warps issue the MMAs, blocks in turn, each into an accumulator of its own: 64 columns for the products of the high parts and 64 for
//     those with a low part (the activations' high parts are multiplied with both parts of the weights at once);
//   * rows m lie in the lanes, so that a warp stores 128 bytes of a column straight from registers whatever C's pitch and alignment.
// TF32 parts need no scales of rows and columns and leave nothing over: no lists, no second kernel behind this one.  A low part as it is would lose
// bits below 2^-113, where it meets TF32's smallest step, 2^-136 (operands of 1e-36 3.4e-6 off, of 1e-38 3.3e-4).  So all low parts are held
// times 2^OUT_LOW, which the sums of their products lose again: operands keep their 22 bits down to 2^-124, and from there on steps of 2^-146.
//
// us in a series, before / now: 4096 x 128 . 128 x 4096 40 / 25, 2000 x 128 . 128 x 2000 22.0 / 11.9, 6000 x
// 32 . 32 x 6000 63 / 39 (planes); 2001 x 77 . 77 x 3003 58 / 15.8, 1504 x 64 . 64 x 3500 42 / 9.5 (streaming); 3734 x 104 . 104 x 575 15.8 / 10.3 (two rounds of small
// products).  Drawn over batches of 17 to 128 and layers of 300 to 6000: 0.41 of the time of planes, 0.34 of the streaming kernel, 0.68 of small products in two
// rounds, 0.86 at most.
// Bound, per block of 64 columns and K = 128, by the MMAs (1540 clocks at their rate, 2400 with what the two warps need to issue them beside
// the others) and by what the sixteen warps do in turn (1000 clocks of stores, at the 32 bytes per clock that an SM sends to L2; 900 to
// split; 400 to load): 2700 clocks, 25 us for 64 MB that take 12.5 to store alone.
//
// What decided: whole warps wait.  A wait by one lane of a warp whose others stand at the next convergence point costs twice as much as one by all
// (480 clocks against 220 for a round of two mbarriers).  And no spills: with all shared memory taken a spilled register comes back by way of
// L2 behind the stores; 100 bytes of them made 25 us 70.  Tried and taken back: warps with roles of their own for splitting, draining and strips (34 us: every
// hand-over is a wait, and blocks are short), output in a rolled loop of eight columns (48).
#include "cn_epilogue.cuh"
#include "cn_gemm.h"
#include "cn_tc_feed.cuh"

#define OUT_N 64                // columns n of a block
#define OUT_UNIT 16             // columns that work is cut in
#define OUT_WORK 512            // threads of the warps that split, drain and store
#define OUT_THREADS (OUT_WORK + 64)   // warps 16 and 17: MMAs
#define OUT_MAX_BLOCKS 4        // blocks of 32 k: the parts of the strip take half of tensor memory
#define OUT_MAX_K (OUT_MAX_BLOCKS * SM_BK)
#define OUT_ACC_COL 256         // two accumulators behind the strip
#define OUT_ACC_COLS 128
#define OUT_CHUNK_BYTES (2 * OUT_N * 128)   // hi and lo parts of 64 columns x 32 k
#define OUT_LOW 10              // with 11, a sum could exceed fp32's range where the products that it stands for do not
#define OUT_STAGES 3
#define OUT_SMEM (1024 + OUT_STAGES * OUT_MAX_BLOCKS * OUT_CHUNK_BYTES)

struct OuterParams {
    const float *A, *W;     // stored with k contiguous: element (row, k) at [row * pitch + k]
    int64_t lda, ldw;
    int a_vec;              // the activations' rows are aligned to 16 bytes (the weights': W_VEC)
    int M, N, K;
    float *C;
    int64_t ldc;
    int kb;                 // blocks of 32 k
    int passes;             // parts of K that are multiplied into an accumulator each
    int two_chains;         // the products of the high parts of the two halves of such a part are added apart
    float low;              // what an accumulator's second half still has to be multiplied by
    int sh;                 // log2 of 16-byte chunks of k, rounded up to a power of two
    int strips, units;      // of 128 rows m; of 16 columns n per strip
    int per_strip;          // CTAs that share a strip's units; 0: all strips' units, behind one another, are shared by all CTAs
    unsigned int *status;
};

// The blocks of a CTA, in order.
struct OutWalk {
    int strip, u, left;   // where the next block begins, and units of columns to go
    __device__ __forceinline__ explicit OutWalk(const OuterParams &p)
    {
        const int units = p.units;
        if (p.per_strip > 0) {
            strip = blockIdx.x / p.per_strip;
            const int j = blockIdx.x - strip * p.per_strip;
            u = (int)((int64_t)units * j / p.per_strip);
            left = (int)((int64_t)units * (j + 1) / p.per_strip) - u;
        } else {
            const int64_t total = (int64_t)p.strips * units, pos = total * blockIdx.x / gridDim.x;
            left = (int)(total * (blockIdx.x + 1) / gridDim.x - pos);
            strip = (int)(pos / units);
            u = (int)(pos - (int64_t)strip * units);
        }
    }
    // strip, first column and number of columns
    __device__ __forceinline__ bool next(const OuterParams &p, int &strip_, int &n0, int &cols)
    {
        if (left <= 0) return false;
        int take = OUT_N / OUT_UNIT;
        if (take > p.units - u) take = p.units - u;
        if (take > left) take = left;
        strip_ = strip;
        n0 = u * OUT_UNIT;
        cols = take * OUT_UNIT < p.N - n0 ? take * OUT_UNIT : p.N - n0;
        left -= take;
        u += take;
        if (u == p.units) { u = 0; ++strip; }
        return true;
    }
};

// D[tmem] (+)= A[tmem] * B[smem]: 128 rows, TF32; eight columns of tensor memory per k-step.
__device__ __forceinline__ void out_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 bd;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 bd, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], bd, %4, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void out_st4(uint32_t taddr, const uint32_t (&v)[4])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ uint32_t out_at(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }   // 16-byte chunk c of row r

// D[tmem] = A[tmem] * B[smem] + D[tmem] * 2^-OUT_LOW
__device__ __forceinline__ void out_mma_ts_lowered(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 bd;\n\t"
        "setp.eq.b32 p, 0, 0;\n\t"
        "mov.b64 bd, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], bd, %4, p, %5;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(desc_hi), "r"(idesc), "n"(OUT_LOW) : "memory");
}

// The parts of two elements, the low ones times 2^OUT_LOW.
template <bool CAREFUL>
__device__ __forceinline__ void out_split2(float x, float y, uint32_t (&h)[2], uint32_t (&l)[2])
{
    h[0] = sm_tf32<CAREFUL>(x);
    h[1] = sm_tf32<CAREFUL>(y);
    float lx, ly;   // what is left of both by one subtraction and one multiplication, exactly
    asm("{\n\t.reg .b64 a, b, m;\n\t"
        "mov.b64 a, {%2, %3};\n\t"
        "mov.b64 b, {%4, %5};\n\t"
        "mov.b64 m, {%6, %6};\n\t"
        "fma.rn.f32x2 a, b, m, a;\n\t"
        "mov.b64 m, {%7, %7};\n\t"
        "mul.rn.f32x2 a, a, m;\n\t"
        "mov.b64 {%0, %1}, a;\n\t}"
        : "=f"(lx), "=f"(ly)
        : "f"(x), "f"(y), "f"(__uint_as_float(h[0])), "f"(__uint_as_float(h[1])), "f"(-1.0f), "f"((float)(1 << OUT_LOW)));
    l[0] = sm_tf32<CAREFUL>(lx);
    l[1] = sm_tf32<CAREFUL>(ly);
}

// Four elements as parts.
template <bool CAREFUL>
__device__ __forceinline__ void out_split4(const float *y, uint32_t (&h)[4], uint32_t (&l)[4])
{
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
        uint32_t hh[2], ll[2];
        out_split2<CAREFUL>(y[e], y[e + 1], hh, ll);
        h[e] = hh[0]; h[e + 1] = hh[1];
        l[e] = ll[0]; l[e + 1] = ll[1];
    }
}

// The share of a thread of a block of 64 columns n x K: up to 16 elements.  VEC (columns aligned to 16 bytes): 16 bytes along k of up to four
// columns, a warp reads up to 512 bytes of one.  Else one k of up to 16 columns, a warp reads 128 bytes.
template <bool VEC>
struct OutShare {
    const float *src;
    int row, k;
    // threads per column, as a power of two; columns between this thread's, and how many it has
    static __device__ __forceinline__ int shift(const OuterParams &p) { return p.sh + (VEC ? 0 : 2); }
    static __device__ __forceinline__ int rows_on(const OuterParams &p) { return OUT_WORK >> shift(p); }
    static __device__ __forceinline__ int items(const OuterParams &p) { return (OUT_N << shift(p)) / OUT_WORK; }
    __device__ __forceinline__ OutShare(const OuterParams &p, int t)
    {
        const int c = t & ((1 << shift(p)) - 1);
        k = VEC ? 4 * c : c;
        row = t >> shift(p);
        src = p.W + row * p.ldw + k;
    }
    __device__ __forceinline__ void load(const OuterParams &p, int n0, int cols, float (&x)[16]) const
    {
        const float *q = src + n0 * p.ldw;
        const int64_t step = rows_on(p) * p.ldw;
        const int n = items(p);
        if (VEC && cols == OUT_N && p.K == 32 << (p.sh - 3)) {   // whole blocks of 32, 64 or 128 k
#pragma unroll
            for (int i = 0; i < 4; ++i, q += step) {
                if (i >= n) break;
                const float4 v = *reinterpret_cast<const float4 *>(q);
                x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
            }
        } else if (VEC) {
            const int left = p.K - k;
#pragma unroll
            for (int i = 0; i < 4; ++i, q += step) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (i < n && row + i * rows_on(p) < cols) {
                    if (left >= 4) {
                        v = *reinterpret_cast<const float4 *>(q);
                    } else {
                        if (left > 0) v.x = q[0];
                        if (left > 1) v.y = q[1];
                        if (left > 2) v.z = q[2];
                    }
                }
                x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i, q += step) x[i] = i < n && row + i * rows_on(p) < cols && k < p.K ? *q : 0.0f;
        }
    }
    template <bool CAREFUL>
    __device__ __forceinline__ void put(const OuterParams &p, uint32_t stage, const float (&x)[16]) const
    {
        constexpr uint32_t lo = OUT_N * 128;
        if (k >= SM_BK * p.kb) return;   // of the next power of two
        stage += (uint32_t)(k >> 5) * OUT_CHUNK_BYTES + (VEC ? 0 : (k & 3) * 4);
        const int n = items(p);
#pragma unroll
        for (int i = 0; i < (VEC ? 4 : 16); i += VEC ? 1 : 2) {
            if (i >= n) break;
            const uint32_t q = stage + out_at(row + i * rows_on(p), k >> 2 & 7);
            if (VEC) {
                uint32_t h[4], l[4];
                out_split4<CAREFUL>(x + (VEC ? 4 * i : 0), h, l);
                sts4u(q, h[0], h[1], h[2], h[3]);
                sts4u(q + lo, l[0], l[1], l[2], l[3]);
            } else {   // columns come in twos: four, eight or sixteen
                const uint32_t r = stage + out_at(row + (i + 1) * rows_on(p), k >> 2 & 7);
                uint32_t h[2], l[2];
                out_split2<CAREFUL>(x[i], x[i + 1], h, l);
                sts1u(q, h[0]);
                sts1u(q + lo, l[0]);
                sts1u(r, h[1]);
                sts1u(r + lo, l[1]);
            }
        }
    }
    __device__ __forceinline__ void store(const OuterParams &p, uint32_t stage, const float (&x)[16]) const
    {
        float m = 0.0f;   // whether sm_tf32 has to be careful with some of the values
#pragma unroll
        for (int e = 0; e < 16; e += 2) asm("max.NaN.abs.f32 %0, %1, %2, %0;" : "+f"(m) : "f"(x[e]), "f"(x[e + 1]));
        if (m < __uint_as_float(0x7f7ff000u)) put<false>(p, stage, x);
        else put<true>(p, stage, x);
    }
};

// 32 rows x 32 k of the strip from (row0, k0) on, as this lane loads them: 16 bytes along k of eight rows or, unaligned, one k of 32 rows.
__device__ __forceinline__ void out_strip_load(const OuterParams &p, int row0, int rows, int k0, float (&x)[32])
{
    const int lane = threadIdx.x & 31, left = p.K - k0;
    if (p.a_vec && left >= SM_BK) {
        const float *q = p.A + (row0 + (lane >> 3)) * p.lda + (k0 + 4 * (lane & 7));
#pragma unroll
        for (int i = 0; i < 8; ++i, q += 4 * p.lda) {
            const float4 v = 4 * i + (lane >> 3) < rows ? *reinterpret_cast<const float4 *>(q) : make_float4(0.f, 0.f, 0.f, 0.f);
            x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
        }
    } else {
        const float *q = p.A + row0 * p.lda + (k0 + lane);
#pragma unroll
        for (int i = 0; i < 32; ++i, q += p.lda) x[i] = i < rows && lane < left ? *q : 0.0f;
    }
}
// ... into shared memory, 4 KB of this warp
__device__ __forceinline__ void out_strip_turn(const OuterParams &p, int k0, uint32_t turn, const float (&x)[32])
{
    const int lane = threadIdx.x & 31;
    if (p.a_vec && p.K - k0 >= SM_BK) {
#pragma unroll
        for (int i = 0; i < 8; ++i) sts4f(turn + out_at(4 * i + (lane >> 3), lane & 7), x + 4 * i);
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) sts1(turn + out_at(i, lane >> 2) + (lane & 3) * 4, x[i]);
    }
}

template <bool W_VEC>
__global__ void __launch_bounds__(OUT_THREADS, 1)
cn_gemm_outer_kernel(const __grid_constant__ OuterParams p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[OUT_STAGES + 7];
    __shared__ uint32_t s_words[2];   // tensor-memory base, abort flag
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u, stage_bytes = (uint32_t)p.kb * OUT_CHUNK_BYTES;
    // the weights of a stage are there; the products of an accumulator have retired (and the stage that they read is free); an accumulator has
    // been read; a strip is there, strips by turns; the stage by way of which it was made is free again
    const uint32_t full0 = smem_u32(&bars[0]), done0 = full0 + 8 * OUT_STAGES, read0 = done0 + 16, strip0 = read0 + 16, turned_bar = strip0 + 16;
    const uint32_t abort_flag = smem_u32(&s_words[1]);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // the same for the whole warp, which the compiler is told
    cn_pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < OUT_STAGES; ++s) mbar_init(full0 + 8 * s, OUT_WORK / 32);
        for (int b = 0; b < 2; ++b) { mbar_init(done0 + 8 * b, 1); mbar_init(read0 + 8 * b, OUT_WORK / 32); mbar_init(strip0 + 8 * b, OUT_WORK / 32); }
        mbar_init(turned_bar, OUT_WORK / 32);
        s_words[1] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_words[0])), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_words[0];
    OutWalk walk(p);
    int strip, n0, cols;
    bool ok = true;
    if (warp >= 16) {
        // ---------------------------------------------------------------- MMAs: every other block, by either warp
        constexpr uint32_t tf32 = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(SM_BM >> 4) << 24);
        constexpr uint32_t idesc = tf32 | ((uint32_t)(OUT_N >> 3) << 17), idesc2 = tf32 | ((uint32_t)(OUT_ACC_COLS >> 3) << 17);
        const uint64_t d0 = make_kmajor_sw128_desc(ring);
        const uint32_t hi = (uint32_t)(d0 >> 32), b = warp & 1u, acc = tmem + OUT_ACC_COL + b * OUT_ACC_COLS;
        const int first_strip = walk.strip;
        int have = -1;
        uint32_t accs = 0u;
        for (uint32_t i = 0; ok && walk.next(p, strip, n0, cols); ++i) {
            // Either warp waits for every strip, on two barriers in turn: a wait for the phase after the next one would not wait at all, and a
            // strip of a single block may be multiplied, and the next one made, before the warp that has no block there has looked.  That
            // warp has the next strip's first block, so that it is never more than one phase late.
            if (strip != have) {
                have = strip;
                ok = mbar_wait_warp(strip0 + 8 * (strip & 1), (uint32_t)(strip - first_strip) >> 1 & 1u, abort_flag, p.status, 25u);
                if (!ok) break;
            }
            const uint32_t s = i % OUT_STAGES;
            for (int pass = 0; pass < p.passes && ok; ++pass, ++accs) {
                if ((accs & 1u) != b) continue;
                ok = mbar_wait_warp(full0 + 8 * s, i / OUT_STAGES & 1u, abort_flag, p.status, 15u) &&
                     mbar_wait_warp(read0 + 8 * b, (accs >> 1 & 1u) ^ 1u, abort_flag, p.status, 26u);
                if (!ok) break;
                tc_fence_after();
                if (lane == 0) {
                    // Blocks [k0, k1) of 32 k.  Up to kt the products of the high parts go to the accumulator's first half and those with a low part
                    // to the second; the remaining blocks' products with a low part go to the second, too, and then, on top of all of
                    // those, which lose their factor, the products of their high parts.
                    const int k0 = p.kb * pass / p.passes, k1 = p.kb * (pass + 1) / p.passes, kt = p.two_chains ? (k0 + k1) >> 1 : k1;
                    const uint32_t w0 = (uint32_t)d0 + s * (stage_bytes >> 4);
                    uint32_t more = 0u;
#pragma unroll 1
                    for (int kb = k0; kb < kt; ++kb) {
                        const uint32_t w = w0 + kb * (OUT_CHUNK_BYTES >> 4), a = tmem + kb * SM_BK;
#pragma unroll
                        for (int j = 0; j < SM_BK / 8; ++j, more = 1u) {
                            out_mma_ts(acc, a + 8 * j, w + 2 * j, hi, idesc2, more);
                            out_mma_ts(acc + OUT_N, a + OUT_ACC_COL / 2 + 8 * j, w + 2 * j, hi, idesc, 1u);
                        }
                    }
                    if (kt < k1) {
                        // an odd number of blocks: half of one each
                        const bool odd = ((k0 + k1) & 1) != 0;
                        if (odd) {
                            const uint32_t w = w0 + kt * (OUT_CHUNK_BYTES >> 4), a = tmem + kt * SM_BK;
#pragma unroll
                            for (int j = 0; j < SM_BK / 16; ++j, more = 1u) {
                                out_mma_ts(acc, a + 8 * j, w + 2 * j, hi, idesc2, more);
                                out_mma_ts(acc + OUT_N, a + OUT_ACC_COL / 2 + 8 * j, w + 2 * j, hi, idesc, 1u);
                            }
                        }
                        const int j0 = odd ? SM_BK / 16 : 0;   // where the second half begins in block kt
#pragma unroll 1
                        for (int kb = kt; kb < k1; ++kb) {
                            const uint32_t w = w0 + kb * (OUT_CHUNK_BYTES >> 4), a = tmem + kb * SM_BK;
#pragma unroll
                            for (int j = 0; j < SM_BK / 8; ++j) {
                                if (kb == kt && j < j0) continue;
                                out_mma_ts(acc + OUT_N, a + 8 * j, w + (OUT_N * 128 >> 4) + 2 * j, hi, idesc, 1u);
                                out_mma_ts(acc + OUT_N, a + OUT_ACC_COL / 2 + 8 * j, w + 2 * j, hi, idesc, 1u);
                            }
                        }
                        out_mma_ts_lowered(acc + OUT_N, tmem + kt * SM_BK + 8 * j0, w0 + kt * (OUT_CHUNK_BYTES >> 4) + 2 * j0, hi, idesc);
#pragma unroll 1
                        for (int kb = kt; kb < k1; ++kb) {
                            const uint32_t w = w0 + kb * (OUT_CHUNK_BYTES >> 4), a = tmem + kb * SM_BK;
#pragma unroll
                            for (int j = 0; j < SM_BK / 8; ++j)
                                if (kb > kt || j > j0) out_mma_ts(acc + OUT_N, a + 8 * j, w + 2 * j, hi, idesc, 1u);
                        }
                    }
                    tc_commit(done0 + 8 * b);
                }
                __syncwarp();
            }
        }
        __syncwarp();
    } else {
        // ---------------------------------------------------------------- strips, weights, drain, stores
        const int q = warp & 3, g = warp >> 2;   // a quarter of the lanes; 32 k of a strip, 16 columns of a block
        const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
        const OutShare<W_VEC> share(p, (int)threadIdx.x);
        float x[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = 0.0f;
        // by way of a stage that is free.  The last wait is for all warps of the CTA, but bounded: one of them may have given up before.
        const int first_strip = walk.strip;
        auto make_strip = [&](int strip, uint32_t stage) {
            const int row0 = strip * SM_BM + q * 32, rows = p.M - row0 < 32 ? p.M - row0 : 32;   // none, where negative
            if (g < p.kb) {
                const uint32_t turn = stage + (uint32_t)warp * 4096u;
                float raw[32];
                out_strip_load(p, row0, rows, g * SM_BK, raw);
                out_strip_turn(p, g * SM_BK, turn, raw);
                __syncwarp();
                uint32_t to = lanes + g * SM_BK;
                // short code, which a launch has to fetch
#pragma unroll 1
                for (int c = 0; c < 8; ++c, to += 4) {
                    const float4 f = lds4(turn + out_at(lane, c));
                    const float y[4] = {f.x, f.y, f.z, f.w};
                    uint32_t h[4], l[4];
                    out_split4<true>(y, h, l);
                    __syncwarp();
                    out_st4(to, h);
                    out_st4(to + OUT_ACC_COL / 2, l);
                }
                tc_wait_st();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(strip0 + 8 * (strip & 1)); mbar_arrive(turned_bar); }
            ok = mbar_wait_warp(turned_bar, (uint32_t)(strip - first_strip) & 1u, abort_flag, p.status, 27u);   // the stage may be written
        };
        auto put = [&](uint32_t s) {
            share.store(p, ring + s * stage_bytes, x);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + 8 * s);
        };
        OutWalk ahead(p);
        int astrip, an0, acols;
        cn_pdl_wait();
        bool amore = ahead.next(p, astrip, an0, acols), more = walk.next(p, strip, n0, cols);
        if (amore) share.load(p, an0, acols, x);
        make_strip(strip, ring);
        uint32_t accs = 0u, s = 0u;   // s: the stage of the block that is read, and of the one three blocks on
#pragma unroll 1
        for (; s < OUT_STAGES && amore && ok; ++s) {
            put(s);
            amore = ahead.next(p, astrip, an0, acols);
            if (amore) share.load(p, an0, acols, x);
        }
        s = 0u;
        while (more && ok) {
            const int col0 = n0 + g * 16, here = cols - g * 16, m = strip * SM_BM + q * 32 + lane;   // 16 columns of the block; those that exist
            int next_strip = strip;
            more = walk.next(p, next_strip, n0, cols);
            const bool change = more && next_strip != strip;
            float v[16];
            // the sums of the next accumulator, over all products of a part of K
            auto read = [&](bool first) {
                const uint32_t b = accs & 1u, src = lanes + OUT_ACC_COL + b * OUT_ACC_COLS + g * 16;
                ok = mbar_wait_warp(done0 + 8 * b, accs >> 1 & 1u, abort_flag, p.status, 16u);
                if (!ok) return;
                ++accs;
                tc_fence_after();
                if (first) {
                    uint32_t r[2][16];
                    tc_ld_ahead(src, r[0]);
                    tc_ld_ahead(src + OUT_N, r[1]);
                    tc_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        asm volatile("" : "+r"(r[0][e]), "+r"(r[1][e]));   // no use moves before the wait
                        v[e] = fmaf(__uint_as_float(r[1][e]), p.low, __uint_as_float(r[0][e]));
                    }
                } else {   // eight columns at a time: there are no registers for more, and one that spills costs more than all of this
#pragma unroll
                    for (int h = 0; h < 16; h += 8) {
                        uint32_t r[2][8];
                        tc_ld_ahead(src + h, r[0]);
                        tc_ld_ahead(src + OUT_N + h, r[1]);
                        tc_wait_ld();
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            asm volatile("" : "+r"(r[0][e]), "+r"(r[1][e]));
                            v[h + e] += fmaf(__uint_as_float(r[1][e]), p.low, __uint_as_float(r[0][e]));
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(read0 + 8 * b);
            };
            read(true);
            if (p.passes > 1 && ok) read(false);
            if (!ok) break;
            if (m < p.M) {
                // a base that all lanes have in common, and 32 bits of this lane's: its row within the strip (a matrix may have 2^30 rows and more)
                char *to = reinterpret_cast<char *>(p.C + ((int64_t)col0 * p.ldc + (int64_t)strip * SM_BM));
                const uint32_t at = (uint32_t)(q * 32 + lane) * 4u;
                const int64_t column = p.ldc * 4;
                if (here >= 16) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) *reinterpret_cast<float *>(to + e * column + at) = v[e];
                } else {
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        if (e < here) *reinterpret_cast<float *>(to + e * column + at) = v[e];
                }
            }
            // all products that read this strip have retired: the next one takes its place, by way of the stage that they have left
            if (change) make_strip(next_strip, ring + s * stage_bytes);
            if (!ok) break;
            strip = next_strip;
            // Every warp stores first and splits then; stores are bound by the way to L2, which takes 32 bytes per clock from an SM.
            if (amore) {
                put(s);
                amore = ahead.next(p, astrip, an0, acols);
                if (amore) share.load(p, an0, acols, x);
            }
            s = s == OUT_STAGES - 1 ? 0u : s + 1u;
        }
    }
    __syncwarp();
    if (!ok) {   // after a wait that ran out, the products under way get a bounded chance to end
        const long long t0 = clock64();
        while (clock64() - t0 < 20000000LL) {}
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------------ host
//
// Which weight gradients (Tdot, no bias, linear units, 3x mode).  Shapes that the small products' kernel makes in one round stay there: it is up to 15 %
// slower from K = 64 on (784 x 128 . 128 x 1200 8.0 / 6.8 us), but its shares of K are chains of their own, 1.2e-7 off where this one, as fast as
// that, is off by 3.3e-7.  With fewer than eight rows most lanes have no work (up to 1.5 of the streaming kernel's time with one).  Up to 16 k are one addition
// as planes and two here (6.6e-8 / 8.3e-8).
// Other products with so short a K (other layouts, bias, units, the single pass) keep their kernels, though a trial form of this one took 0.51 of their
// time over 133 drawn ones: their layouts, epilogues and single pass are not written here.
bool cn_gemm_outer_shape(int64_t M, int64_t N, int64_t K)
{
    return M >= 8 && K > 16 && K <= OUT_MAX_K && M < (1LL << 31) - 256 && N < (1LL << 31) - 256;
}

template <bool W_VEC>
static int outer_launch(cn_context *ctx, const OuterParams &p, int64_t ctas, cudaStream_t s)
{
    static bool attr_set[64] = {};
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        CN_CUDA(cudaFuncSetAttribute(cn_gemm_outer_kernel<W_VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT_SMEM));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    CN_CUDA(cn_launch_pdl(cn_gemm_outer_kernel<W_VEC>, dim3((unsigned)ctas), OUT_THREADS, (size_t)OUT_SMEM, s, p));
    cn_count_launch();
    return CN_OK;
}

int cn_gemm_outer_launch(cn_context *ctx, int64_t M, int64_t N, int64_t K, const float *A, int64_t lda, const float *B, int64_t ldb, float *C, int64_t ldc,
                         cudaStream_t s, bool fine)
{
    OuterParams p;
    unsigned int *d_status = nullptr;
    int st = cn_status_block(ctx, &d_status);
    if (st != CN_OK) return st;
    auto aligned = [](const float *q, int64_t ld) { return (ld & 3) == 0 && ((uintptr_t)q & 15u) == 0; };
    const bool w_vec = aligned(B, ldb);
    p.A = A; p.W = B;
    p.lda = lda; p.ldw = ldb;
    p.a_vec = aligned(A, lda);
    p.M = (int)M; p.N = (int)N; p.K = (int)K;
    p.C = C; p.ldc = ldc;
    p.kb = (int)((K + SM_BK - 1) / SM_BK);
    // The tensor core truncates when it adds, so the error grows with the additions to one sum.  As few as the kernels had that took such shapes
    // before (2-norm against fp64, theirs / here): planes, 128 k per chain, 3.9e-7 / 3.0e-7 at K = 100 to 128 by one chain of up to
    // sixteen additions, below that 2.1e-7 / 1.5e-7 by two; the streaming kernel's chains of 32 k where the weights have an odd pitch, 2.1e-7 / 1.6e-7
    // by two; the small products' kernel, and planes in its place, 1.3e-7 / 1.2e-7 by two of four additions each, for half of K at a time.
    p.two_chains = fine || !w_vec || K <= 96;
    p.low = p.two_chains ? 1.0f : 1.0f / (1 << OUT_LOW);
    p.passes = fine && p.kb > 2 ? 2 : 1;
    p.sh = p.kb == 1 ? 3 : p.kb == 2 ? 4 : 5;
    p.strips = (int)((M + SM_BM - 1) / SM_BM);
    p.units = (int)((N + OUT_UNIT - 1) / OUT_UNIT);
    p.status = d_status;
    const int64_t sms = ctx->sm_count, total = (int64_t)p.strips * p.units;
    int64_t ctas = total < sms ? total : sms;
    p.per_strip = 0;
    const int64_t per = p.strips <= sms ? sms / p.strips : 0;
    if (per > 0) {
        // Either every strip has CTAs of its own, or all share all units evenly, and most CTAs meet a second strip: the blocks of 64 columns that the
        // busiest makes, where the second strip counts as two more
        const int64_t whole = ((p.units + per - 1) / per + 3) / 4, shared = ((total + ctas - 1) / ctas + 3) / 4 + 2;
        if (whole <= shared) {
            p.per_strip = (int)(per < p.units ? per : p.units);
            ctas = (int64_t)p.per_strip * p.strips;
        }
    }
    st = w_vec ? outer_launch<true>(ctx, p, ctas, s) : outer_launch<false>(ctx, p, ctas, s);
    if (st == CN_OK) {
        ctx->gemm_last_path = "tcgen05_3xtf32";
        ctx->gemm_last_kernel = "outer";
    }
    return st;
}
