// Products of two operands that both lie as planes: fp16 hi / lo parts, k contiguous, with power-of-two scales (see cn_gemm_tc.cu).
//
// The pre-pass that makes planes serves the streaming kernel (activations) and the kernel below, which multiplies planes by planes.
// The streaming kernel converts every weight once per 128 rows of activations; it is meant for weights that are read once.  With more
// rows than that (a large batch, a weight gradient, whose "weights" are the errors) it pays to write the parts of the weights to
// memory once and to leave the main loop to TMA and the tensor cores.
//
// cn_gemm_planes_kernel.  A pair of CTAs (cta_group::2) multiplies a tile of 256 columns n by up to 256 rows m: each CTA loads the
// parts of its 128 columns of the weights and of half the rows of the activations, 64 k per stage, and the tensor cores of both read
// both halves.  Accumulators [128 n][256 m] twice per CTA fill tensor memory, so that two warpgroups add a finished chain (at most
// 512 k, one scale group) to running sums in registers while the next one accumulates.  Persistent pairs; the tiles that do not fill
// a round are cut along K and added by cn_splitk_reduce_kernel, as in the streaming kernel.
//
// What two fp16 parts cannot hold of an element comes as a list: the pre-pass writes the few elements of 16 rows x 512 k that leave
// more than the product may lose (about one in 2^20 of uniform ones) to a cell, and the drain warps multiply them in fp32 FMAs.
// Where a cell overflows (elements of very different size beside each other) this kernel does nothing and the streaming kernel,
// launched behind it and its reduction, does all; else that launch ends at once.  It cuts tiles along K where whole ones would leave most of
// the chip idle (one more launch, see cn_tc_decompose); one reduction behind both kernels, the other order, cost every product with
// cut tiles 3 us.  The pre-pass raises a word at the first overflow, and what it has not written of the weights' planes by then stays
// unwritten.  Lists that overflow, against the streaming kernel alone, us: 520 x 40000 . 40000 x 256 154 / 123 (1296 with whole tiles), 640 x
// 100000 . 100000 x 256 309 / 275 (3148); with whole tiles 520 x 4096 . 4096 x 4096 204 / 132, 1024 rows 212 / 183, 4096^3 650 / 584.
//
// Bound by the tensor cores (their pipe is busy in 80 % of the cycles at 2048 x 4096 . 4096 x 4096): 4096^3, 3x mode, 336 us from an idle GPU, against 476 us on the streaming
// kernel (2048 rows 187 / 263, 1024 rows 120 / 142; single pass 184 / 392): 52 for the pre-pass, which moves 256 MB, 274 for this kernel (1.50 PFLOP/s of
// fp16), 8 for the reduction of the cut tail, 2 for the launch that ends at once.  In a series of seconds the power cap takes the clock to 1.4 GHz, and
// they take 51, 340, 10 and 6: 407.  Short K is bound by the drain warps and the stores: 4096 x 128 . 128 x 4096 44 us with 32-byte
// stores from registers, 39 by TMA (see the epilogue); 1320 x 144 . 144 x 1872 with ReLU 27 -> 23.
#include <cuda.h>
#include <cuda_fp16.h>
#include "cn_epilogue.cuh"
#include "cn_gemm.h"
#include "cn_gemm_tc.h"
#include "cn_tc_split.cuh"

// ------------------------------------------------------------------------------------------ activation pre-pass
// A (M x K) -> planes hi, lo: [M][Kp] fp16 with k contiguous, k in [K, Kp) zero, and the inverse scales a_inv[group][m_pad].
// One CTA per 16 rows and group of 512 k.  What the planes leave of an element (see the top) goes to the next band's planes and
// scales; `bands` tells which blocks of 16 rows x 32 k have any.  Bound by latency for a layer's activations and by memory otherwise: 4 bytes read
// and 4 written per element.  CODED: the consumer-side half of the 8-bit exchange.  The activations arrive as gathered codes
// (column-major like the fp32 matrix; column block r was coded by rank r with scale scales[r]) and are decoded here, inside
// the pre-pass of the GEMM that consumes them, instead of being written out as fp32 first.  This rank's own block is taken
// from its exact fp32 values.  Decode table as kDecompression_8bit builds it (source/clusterKernels.cu:1141-1152).
struct ActCoded {
    const uint8_t *codes;
    const float *scales, *tbl, *own_fp32;
    int own_rank, nranks;
};
#define ACT_ROWS TC_SUB

// Where the planes of an operand are (cn_plane_layout).
struct ActPlanes {
    uint16_t *p;            // band 0: hi, lo (3x mode only), band 1: ...
    int64_t plane, Kp, m_pad, groups;
    float *inv;
    uint8_t *bands;         // null where there is one band only
    int stages;
    int nbands;             // bands to make: TC_BANDS, or 1 for an operand whose left-overs are wanted as cells only
    uint8_t *counts;        // cells of left-overs (cn_planes), null where nobody reads them
    uint2 *cells;
    unsigned int *overflow; // CN_STATUS_OVERFLOW: raised where a cell has no room
    bool optional;          // nobody reads these planes any more once it is raised
    __device__ __forceinline__ uint8_t *band_byte(int64_t m0, int64_t stage) const
    {
        return bands + ((m0 / TC_BM) * stages + stage) * (TC_BM / TC_SUB) + (m0 % TC_BM) / TC_SUB;
    }
};

// What the parts of eight scaled values leave, unscaled; whether that is anything.  A row with an element that is not finite leaves
// nothing, since its sums are not finite anyway.
template <bool LO>
__device__ __forceinline__ bool act_left8(float (&x)[8], float sc, float inv, bool finite)
{
    bool left = false;
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
        uint32_t h, l;
        tc_split2_left<LO>(x[e] * sc, x[e + 1] * sc, h, l, x[e], x[e + 1]);
        x[e] = finite ? x[e] * inv : 0.0f;
        x[e + 1] = finite ? x[e + 1] * inv : 0.0f;
        left |= x[e] != 0.0f || x[e + 1] != 0.0f;
    }
    return left;
}

// Eight consecutive k of one row, scaled, into the planes of a band.  Returns whether the parts may leave something of them: the
// smallest high part tells.
template <bool LO>
__device__ __forceinline__ bool act_store8(const ActPlanes &pl, int band, int64_t at, const float (&x)[8], float sc)
{
    uint32_t h[4], l[4], low = 0x7bff7bffu;
    const uint64_t sc2 = tc_pack2(sc, sc);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        tc_split2<LO>(tc_mul2(tc_pack2(x[2 * e], x[2 * e + 1]), sc2), h[e], l[e]);
        asm("min.xorsign.abs.f16x2 %0, %0, %1;" : "+r"(low) : "r"(h[e]));
    }
    uint16_t *q = pl.p + band * (LO ? 2 : 1) * pl.plane + at;
    *reinterpret_cast<uint4 *>(q) = make_uint4(h[0], h[1], h[2], h[3]);
    if (LO) *reinterpret_cast<uint4 *>(q + pl.plane) = make_uint4(l[0], l[1], l[2], l[3]);
    low &= 0x7fff7fffu;
    return (low >> 16) < tc_safe_f16<LO>() || (low & 0xffffu) < tc_safe_f16<LO>();
}

// Where act_store8 finds a small high part: whether it may be more than a zero's.  The smallest nonzero magnitude tells.  Half of the elements behind a
// rectifier, or behind dropout, are zeros, which leave nothing, but sent nearly every CTA through its block once more (a quarter of the pass over a batch's errors).
template <bool LO>
__device__ __forceinline__ bool act_small8(const float (&x)[8], float sc)
{
    uint32_t amin = 0xffffffffu;   // of 2 |bits| - 1, in which a zero is the largest
#pragma unroll
    for (int e = 0; e < 8; ++e) amin = min(amin, __float_as_uint(x[e]) * 2u - 1u);
    return amin != 0xffffffffu && __uint_as_float((amin + 1u) >> 1) * sc < (LO ? 0.03125f : 6.103515625e-5f);
}

// The cell of a CTA's 16 rows x 512 k: the elements that band 0 leaves something of, in the order of their keys (row << 16 | k), if
// they are few.  begin, add by any threads, end, with barriers between.
struct ActCell {
    uint2 ent[CN_CELL];
    int n;
    __device__ __forceinline__ void add(int row, int k, float x)
    {
        const int at = atomicAdd(&n, 1);
        if (at < CN_CELL) ent[at] = make_uint2((uint32_t)row << 16 | (uint32_t)k, __float_as_uint(x));
    }
    __device__ __forceinline__ void end(const ActPlanes &pl, int64_t cell)
    {
        if (n > CN_CELL) {
            // once: 256 CTAs that store while thousands read cost the pass 25 us
            if (__ldcg(pl.overflow) == 0u) *reinterpret_cast<volatile unsigned int *>(pl.overflow) = 1u;
            return;
        }
        pl.counts[cell] = (uint8_t)n;
        for (int i = 0; i < n; ++i) {   // they came in any order
            int rank = 0;
            for (int j = 0; j < n; ++j) rank += ent[j].x < ent[i].x ? 1 : 0;
            pl.cells[cell * CN_CELL + rank] = ent[i];
        }
    }
};

// Element (k, m) of the block of 512 k x 16 rows in shared memory.  Two k share a line of 128 bytes, whose 16-byte chunks are permuted
// by k / 8 so that neither 16-byte stores of four rows nor reads of eight k each by lanes of four rows x eight k meet in a bank.
__device__ __forceinline__ int act_at(int k, int m)
{
    const int c = ((k & 1) << 2 | (m >> 2)) ^ ((k >> 3) & 7);
    return (k >> 1) * 32 + c * 4 + (m & 3);
}

// Rows that lie m contiguous (or coded), by 256 threads.
template <bool LO, bool CODED>
__device__ __forceinline__ void act_rows(const float *A, int64_t lda, int64_t M, int64_t K, const ActPlanes &pl, const ActCoded &cd, int64_t cta)
{
    __shared__ __align__(128) float tile[TC_GROUP_K * ACT_ROWS];
    __shared__ uint32_t red[16][ACT_ROWS];
    __shared__ float s_sc[ACT_ROWS], s_inv[ACT_ROWS];
    __shared__ bool s_finite[ACT_ROWS];
    __shared__ uint32_t s_left[TC_BANDS][TC_GROUP_KB];   // something is left of these 32 k after the band
    __shared__ ActCell s_cell;
    extern __shared__ float lut[];   // CODED: nranks x 256
    const int tid = threadIdx.x;
    const unsigned int stop = pl.optional && tid == 0 ? __ldcg(pl.overflow) : 0u;
    const bool vec_ok = (lda & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15u) == 0;
    if (CODED) {
        for (int e = tid; e < cd.nranks * 256; e += 256) {
            const int r = e >> 8, c = e & 255, i = c & 127;
            const float p = cd.scales[r];
            float v;
            if (i < CN_CODEBOOK_N) {
                v = __fmul_rn(cd.tbl[i], p);
                if (c >= 128) v = -v;
            } else {
                v = (c == 255) ? -p : p;
            }
            lut[e] = v;
        }
        __syncthreads();
    }
    const int64_t split = CODED ? K / cd.nranks : 0;
    const int64_t Kp = pl.Kp;
    const int m_blocks = (int)(pl.m_pad / ACT_ROWS), g = (int)cta / m_blocks;
    const int64_t m0 = (int64_t)((int)cta - g * m_blocks) * ACT_ROWS, k0 = (int64_t)g * TC_GROUP_K;
    const int lane = tid & 31, warp = tid >> 5;
    if (!CODED && vec_ok) {
        // four rows by eight k per thread, 64 contiguous bytes per k
        const int mq = (tid & 3) * 4, kl = tid >> 2;
        const float *src = A + m0 + mq + (k0 + kl) * lda;
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int64_t k = k0 + kl + 64 * j;
            v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < K && m0 + mq < M) {
                const float *q = src + 64 * j * lda;
                if (m0 + mq + 3 < M) {
                    v[j] = *reinterpret_cast<const float4 *>(q);
                } else {
                    v[j].x = q[0];
                    if (m0 + mq + 1 < M) v[j].y = q[1];
                    if (m0 + mq + 2 < M) v[j].z = q[2];
                }
            }
        }
        uint32_t amax[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            *reinterpret_cast<float4 *>(&tile[act_at(kl + 64 * j, mq)]) = v[j];
            amax[0] = max(amax[0], __float_as_uint(v[j].x) & 0x7fffffffu);
            amax[1] = max(amax[1], __float_as_uint(v[j].y) & 0x7fffffffu);
            amax[2] = max(amax[2], __float_as_uint(v[j].z) & 0x7fffffffu);
            amax[3] = max(amax[3], __float_as_uint(v[j].w) & 0x7fffffffu);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) amax[e] = max(amax[e], __shfl_xor_sync(0xffffffffu, amax[e], o));
            if (lane < 4) { red[warp][mq + e] = amax[e]; red[warp + 8][mq + e] = 0u; }
        }
    } else {
        // Bound by latency.  All 32 elements of a thread (eight, where each is looked up) are on their way before the first is used; in groups of
        // eight memory was waited for four times: 203 x 4001 . 4001 x 3001 45.9 -> 45.2 us, 333 x 4000 . 4000 x 4001 in TF32 mode 56.8 -> 55.7.
        constexpr int BATCH = CODED ? 8 : 32;
        const int ml = tid & 15, kl = tid >> 4;
        const int64_t m = m0 + ml;
        uint32_t amax = 0u;
#pragma unroll 1
        for (int j0 = 0; j0 < TC_GROUP_K / 16; j0 += BATCH) {
            float x[BATCH];
#pragma unroll
            for (int j = 0; j < BATCH; ++j) {
                const int64_t k = k0 + (j0 + j) * 16 + kl;
                x[j] = 0.0f;
                if (m < M && k < K) {
                    if (CODED) {
                        int r = split > 0 ? (int)(k / split) : cd.nranks - 1;
                        if (r > cd.nranks - 1) r = cd.nranks - 1;
                        if (r == cd.own_rank && cd.own_fp32) x[j] = cd.own_fp32[m + (k - split * cd.own_rank) * M];
                        else x[j] = lut[(r << 8) + cd.codes[m + k * M]];
                    } else {
                        x[j] = A[m + k * lda];
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < BATCH; ++j) {
                tile[act_at((j0 + j) * 16 + kl, ml)] = x[j];
                amax = max(amax, __float_as_uint(x[j]) & 0x7fffffffu);
            }
        }
        red[kl][ml] = amax;
    }
    if (tid < TC_BANDS * TC_GROUP_KB) (&s_left[0][0])[tid] = 0u;
    if (tid == 0) s_cell.n = 0;
    const int64_t cell = m0 / ACT_ROWS * pl.groups + g;
    if (__syncthreads_or(stop != 0u)) return;
    for (int band = 0;; ++band) {
        if (band > 0) __syncthreads();
        if (tid < ACT_ROWS) {
            uint32_t amax = 0u;
#pragma unroll
            for (int j = 0; j < 16; ++j) amax = max(amax, red[j][tid]);
            tc_scale<TC_A_EXP>(amax, s_sc[tid], s_inv[tid]);
            s_finite[tid] = amax < 0x7f800000u;
            pl.inv[(band * pl.groups + g) * pl.m_pad + m0 + tid] = s_inv[tid];
        }
        __syncthreads();
        // eight consecutive k per item; a warp covers 4 rows x 64 k (conflict-free reads, whole lines of 128 bytes)
        bool maybe = false;
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int ml = it * 4 + (lane & 3), kk = (warp * 8 + (lane >> 2)) * 8;
            const int64_t m = m0 + ml, k = k0 + kk;
            if (m < M && k < Kp && (band == 0 || s_left[band - 1][kk / TC_WK] != 0u)) {
                float x[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = tile[act_at(kk + e, ml)];
                maybe |= act_store8<LO>(pl, band, m * Kp + k, x, s_sc[ml]) && s_finite[ml] && act_small8<LO>(x, s_sc[ml]);
            }
        }
        // zeros, or elements too small for the scale: what is left takes the elements' place
        bool left = false;
        if (__syncthreads_or(maybe)) {
#pragma unroll 1
            for (int it = 0; it < 4; ++it) {
                const int ml = it * 4 + (lane & 3), kk = (warp * 8 + (lane >> 2)) * 8;
                float x[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = tile[act_at(kk + e, ml)];
                if (act_left8<LO>(x, s_sc[ml], s_inv[ml], s_finite[ml])) {
                    left = true;
                    s_left[band][kk / TC_WK] = 1u;
                    if (band == 0 && pl.counts)
                        for (int e = 0; e < 8; ++e)
                            if (x[e] != 0.0f) s_cell.add(ml, kk + e, x[e]);
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) tile[act_at(kk + e, ml)] = x[e];
            }
            left = __syncthreads_or(left);
        }
        if (band == 0 && pl.counts && tid == 0) s_cell.end(pl, cell);
        if (!left || band == pl.nbands - 1) break;
        // the largest left of each row, as at the start (what the others leave is zero)
        uint32_t amax = 0u;
        for (int j = 0; j < TC_GROUP_K / 16; ++j) amax = max(amax, __float_as_uint(tile[act_at(j * 16 + (tid >> 4), tid & 15)]) & 0x7fffffffu);
        red[tid >> 4][tid & 15] = amax;
    }
    if (pl.bands && tid < TC_GROUP_K / TC_AK && k0 + tid * TC_AK < Kp) {
        uint32_t n = 0u;
        for (int band = 0; band < TC_BANDS - 1; ++band) n += s_left[band][2 * tid] + (s_left[band][2 * tid + 1] << 4);
        *pl.band_byte(m0, k0 / TC_AK + tid) = (uint8_t)n;
    }
}

// Same planes for rows that lie k contiguous (a transposed activation operand, which is also what a row-major M x K batch looks like; an
// untransposed weight matrix): two rows per warp, and of each two times eight k per lane.  16-byte loads whatever the row's alignment:
// the row is read from the 16-byte boundary before it, `d` floats early, and each lane takes the first floats of its neighbour's quads.
#define ACT_ROWS_PER_WARP (ACT_ROWS / 8)
template <bool LO>
__device__ __forceinline__ void act_rows_t(const float *A, int64_t lda, int64_t M, int64_t K, const ActPlanes &pl, int64_t cta)
{
    __shared__ uint32_t s_left[TC_BANDS][TC_GROUP_KB];
    __shared__ ActCell s_cell;
    const int tid = threadIdx.x, lane = tid & 31;
    const int m_blocks = (int)(pl.m_pad / ACT_ROWS), g = (int)cta / m_blocks;
    const int64_t m0 = (int64_t)((int)cta - g * m_blocks) * ACT_ROWS, k0 = (int64_t)g * TC_GROUP_K;
    const int row0 = (tid >> 5) * ACT_ROWS_PER_WARP;
    const unsigned int stop = pl.optional && tid == 0 ? __ldcg(pl.overflow) : 0u;
    if (tid < TC_BANDS * TC_GROUP_KB) (&s_left[0][0])[tid] = 0u;
    if (tid == 0) s_cell.n = 0;
    float x[ACT_ROWS_PER_WARP][2][8], tail[ACT_ROWS_PER_WARP][3];
    int d[ACT_ROWS_PER_WARP];
#pragma unroll
    for (int r = 0; r < ACT_ROWS_PER_WARP; ++r) {
        const int64_t m = m0 + row0 + r;
        const float *src = A + (m < M ? m : 0) * lda + k0;
        d[r] = (int)((reinterpret_cast<uintptr_t>(src) & 15u) / sizeof(float));   // the same for the whole warp
        const float4 *quads = reinterpret_cast<const float4 *>(src - d[r]);
        const int here = m < M ? (int)(K - k0 < TC_GROUP_K ? K - k0 : TC_GROUP_K) + d[r] : 0;   // floats from the boundary to the segment's end
        auto quad = [&](int i) { return 4 * i < here ? quads[i] : make_float4(0.f, 0.f, 0.f, 0.f); };
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float4 a = quad(64 * j + 2 * lane), b = quad(64 * j + 2 * lane + 1);
            x[r][j][0] = a.x; x[r][j][1] = a.y; x[r][j][2] = a.z; x[r][j][3] = a.w;
            x[r][j][4] = b.x; x[r][j][5] = b.y; x[r][j][6] = b.z; x[r][j][7] = b.w;
        }
        const float4 c = d[r] != 0 && lane == 31 ? quad(128) : make_float4(0.f, 0.f, 0.f, 0.f);
        tail[r][0] = c.x; tail[r][1] = c.y; tail[r][2] = c.z;
    }
#pragma unroll
    for (int r = 0; r < ACT_ROWS_PER_WARP; ++r) {
        if (d[r] != 0) {
            float next[2][3];   // the first floats of the next lane's eight; behind lane 31 the other half's, or what lies behind both
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                const float n0 = __shfl_down_sync(0xffffffffu, x[r][0][e], 1), n1 = __shfl_down_sync(0xffffffffu, x[r][1][e], 1),
                            o = __shfl_sync(0xffffffffu, x[r][1][e], 0);
                next[0][e] = lane < 31 ? n0 : o;
                next[1][e] = lane < 31 ? n1 : tail[r][e];
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    auto at = [&](int i) { return i < 8 ? x[r][j][i < 8 ? i : 7] : next[j][i < 8 ? 0 : i - 8]; };
                    x[r][j][e] = d[r] == 1 ? at(e + 1) : d[r] == 2 ? at(e + 2) : at(e + 3);
                }
        }
        if (k0 + TC_GROUP_K > K) {   // what lies behind the row's end in its last quad
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (k0 + 256 * (e >> 3) + 8 * lane + (e & 7) >= K) x[r][e >> 3][e & 7] = 0.0f;
        }
    }
    if (__syncthreads_or(stop != 0u)) return;
    const int64_t cell = m0 / ACT_ROWS * pl.groups + g;
    for (int band = 0;; ++band) {
        float sc[ACT_ROWS_PER_WARP], inv[ACT_ROWS_PER_WARP];
        bool finite[ACT_ROWS_PER_WARP], maybe = false;
#pragma unroll
        for (int r = 0; r < ACT_ROWS_PER_WARP; ++r) {
            const int64_t m = m0 + row0 + r;
            uint32_t amax = 0u;
#pragma unroll
            for (int e = 0; e < 16; ++e) amax = max(amax, __float_as_uint(x[r][e >> 3][e & 7]) & 0x7fffffffu);
            amax = __reduce_max_sync(0xffffffffu, amax);
            tc_scale<TC_A_EXP>(amax, sc[r], inv[r]);
            finite[r] = amax < 0x7f800000u;
            if (lane == 0) pl.inv[(band * pl.groups + g) * pl.m_pad + m] = inv[r];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int kk = 256 * j + 8 * lane;
                if (m < M && k0 + kk < pl.Kp && (band == 0 || s_left[band - 1][kk / TC_WK] != 0u))
                    maybe |= act_store8<LO>(pl, band, m * pl.Kp + k0 + kk, x[r][j], sc[r]) && finite[r];
            }
        }
        // Behind all stores, whose registers it would else be short of (64 a thread).
        if (maybe) {
            maybe = false;
#pragma unroll
            for (int rj = 0; rj < 2 * ACT_ROWS_PER_WARP; ++rj) maybe |= finite[rj >> 1] && act_small8<LO>(x[rj >> 1][rj & 1], sc[rj >> 1]);
        }
        bool left = false;
        if (__syncthreads_or(maybe)) {
#pragma unroll
            for (int rj = 0; rj < 2 * ACT_ROWS_PER_WARP; ++rj) {
                const int r = rj >> 1, j = rj & 1;
                if (!act_left8<LO>(x[r][j], sc[r], inv[r], finite[r])) continue;
                left = true;
                s_left[band][(256 * j + 8 * lane) / TC_WK] = 1u;
                if (band == 0 && pl.counts) {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (x[r][j][e] != 0.0f) s_cell.add(row0 + r, 256 * j + 8 * lane + e, x[r][j][e]);
                }
            }
            left = __syncthreads_or(left);
        }
        if (band == 0 && pl.counts && tid == 0) s_cell.end(pl, cell);
        if (!left || band == pl.nbands - 1) break;
    }
    if (pl.bands && tid < TC_GROUP_K / TC_AK && k0 + tid * TC_AK < pl.Kp) {
        uint32_t n = 0u;
        for (int band = 0; band < TC_BANDS - 1; ++band) n += s_left[band][2 * tid] + (s_left[band][2 * tid + 1] << 4);
        *pl.band_byte(m0, k0 / TC_AK + tid) = (uint8_t)n;
    }
}

// One operand, or two in one launch.  Wait first, then release the product: it may then rely on everything before this pass having
// finished, and start on W.
struct ActJob {
    const float *A;
    int64_t lda, M, K;
    ActPlanes pl;
    int ctas;
};
enum { ACT_ROWS_M = 0, ACT_ROWS_K = 1, ACT_CODED = 2, ACT_NONE = 3 };
template <bool LO, int KIND>
__device__ __forceinline__ void act_job(const ActJob &job, const ActCoded &cd, int cta)
{
    if (KIND == ACT_ROWS_K) act_rows_t<LO>(job.A, job.lda, job.M, job.K, job.pl, cta);
    else if (KIND != ACT_NONE) act_rows<LO, KIND == ACT_CODED>(job.A, job.lda, job.M, job.K, job.pl, cd, cta);
}
template <bool LO, int KIND0, int KIND1>
__global__ void __launch_bounds__(256, 4)
cn_act_planes_kernel(const __grid_constant__ ActJob job0, const __grid_constant__ ActJob job1, const __grid_constant__ ActCoded cd)
{
    cn_pdl_wait();
    cn_pdl_launch_dependents();
    if (KIND1 == ACT_NONE || (int)blockIdx.x < job0.ctas) act_job<LO, KIND0>(job0, cd, blockIdx.x);
    else act_job<LO, KIND1>(job1, cd, blockIdx.x - job0.ctas);
}

// --------------------------------------------------------------------------------------------- planes by planes
#define PL_THREADS 384          // warp 0: TMA producer, warp 1: MMA issuer and tensor-memory owner, warps 4-11: drain and epilogue
#define PL_TILE_BYTES (128 * TC_AK * 2)
#define PL_REGS_WG0 56
#define PL_REGS_DRAIN 224
static_assert(PL_REGS_WG0 + 2 * PL_REGS_DRAIN <= 3 * (65536 / PL_THREADS / 8 * 8), "registers");

// SHORT: tiles of up to PL_SHORT_K k.  A third of the stages makes room for what the drain warps have on its way to C: with two blocks each
// they waited for most of a tile's stores (6900 clocks of 10 400 per tile at 4096 x 128 . 128 x 4096).
// In the single pass, whose tiles take a third of the MMAs, three times as long ones.  Not with logistic units, which bound the drain warps.
#define PL_SHORT_K 256
#define PL_DIRECT_STAGES 12   // of 64 k: up to here logistic units go to C from registers
template <bool MODE3X, bool SHORT>
struct PlCfg {
    static constexpr int PARTS = MODE3X ? 2 : 1;
    static constexpr int STAGES = (MODE3X ? 3 : 6) * (SHORT ? 2 : 3) / 3;
    static constexpr int BATCH = SHORT ? 3 : 1, OUT = 2 * BATCH;    // blocks of output that a drain warp hands over together; that it has room for
    static constexpr int STAGE_BYTES = 2 * PARTS * PL_TILE_BYTES;   // W parts, then activation parts
    static constexpr int TURN_OFF = STAGES * STAGE_BYTES;           // [drain warp][OUT] blocks of 16 rows m x 32 columns n
    static constexpr int TURN_BYTES = OUT * 2048;
    static constexpr int AS_OFF = TURN_OFF + 8 * TURN_BYTES;        // [2 chains][256] inverse scales of the activation rows
    static constexpr int BAR_OFF = AS_OFF + 2 * 256 * 4;
    static constexpr int BARS = 2 * STAGES + 4;
    static constexpr int HOLD_OFF = BAR_OFF + BARS * 8;             // tensor-memory base, abort flag, whether the streaming kernel does it
    static constexpr int SMEM_BYTES = HOLD_OFF + 16 + 768;          // the base is 256-byte aligned, the stages want 1024
    static_assert(SMEM_BYTES <= 232448, "shared memory");
};

struct PlParams {
    int64_t M, N;
    float *C;
    int64_t ldc;
    const float *bias;
    int act;
    int tma_out;            // C has 16-byte aligned columns: tm_c
    int tiles_m;
    int half;               // rows m per CTA and per drain warpgroup: a tile has twice as many; a multiple of 16, at most 128
    int full_tiles, tiles;  // tiles [0, full_tiles) by one pair each, the others cut into runs over tail_pairs pairs
    int tail_pairs;
    int stages;             // of 64 k
    int chain;              // stages per accumulation chain: a power of two, at most 8
    int groups;
    const float *a_inv, *w_inv;      // [group][a_pad], [group][w_pad]
    int64_t a_pad, w_pad;
    const uint8_t *a_counts, *w_counts;   // cells of left-overs, [block of 16 rows][group]
    const uint2 *a_cells, *w_cells;
    const float *A;         // the activations themselves: element (m, k) at A[m * a_m + k * a_k]
    int64_t a_m, a_k;
    const uint16_t *w_planes;
    int64_t Kp, w_plane;
    unsigned int *many;     // CN_STATUS_MANY: receives whether a list overflowed
    float *partials;        // [slot][half of the rows][w][32 quads of m][128 n] float4: slot = pair + tile - full_tiles
    unsigned int *status;
};

// The runs of a pair, in order; in stages of 64 k.
struct PlWalk {
    int t;
    int64_t pos, end;
    __device__ __forceinline__ explicit PlWalk(const PlParams &p)
    {
        const int pair = blockIdx.x >> 1;
        t = pair;
        pos = end = 0;
        if (pair < p.tail_pairs) {
            const int64_t total = (int64_t)(p.tiles - p.full_tiles) * p.stages;
            pos = total * pair / p.tail_pairs;
            end = total * (pair + 1) / p.tail_pairs;
        }
    }
    __device__ __forceinline__ bool next(const PlParams &p, int &tile, int &k0, int &k1, int &slot)
    {
        if (t < p.full_tiles) {
            tile = t;
            k0 = 0;
            k1 = p.stages;
            slot = -1;
            t += gridDim.x >> 1;
            return true;
        }
        if (pos < end) {
            const int r = (int)(pos / p.stages);
            k0 = (int)(pos - (int64_t)r * p.stages);
            const int64_t left = end - pos;
            const int room = p.stages - k0;
            k1 = k0 + (left < room ? (int)left : room);
            tile = p.full_tiles + r;
            slot = (blockIdx.x >> 1) + r;
            pos += k1 - k0;
            return true;
        }
        return false;
    }
};

// D[tmem of both CTAs] (+)= A[smem of both] * B[smem of both]: 256 rows, 128 in each CTA.
__device__ __forceinline__ void pl_mma_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 ad, bd;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 ad, {%1, %3};\n\t"
        "mov.b64 bd, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %4, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives at the barrier of this offset in both CTAs of the pair once the MMAs issued so far have retired.
__device__ __forceinline__ void pl_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// A tile into this CTA's shared memory; the bytes are counted at `bar`, a barrier of the pair's first CTA.
__device__ __forceinline__ void pl_load(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t x, int32_t y, int32_t z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
// A block of 16 rows m by 32 columns n from shared memory to C; what lies outside C is left out.
__device__ __forceinline__ void pl_store(const CUtensorMap *map, uint32_t src, int32_t m, int32_t n)
{
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"((uint64_t)map), "r"(src), "r"(m), "r"(n) : "memory");
}
// The wait for 16 columns of tensor memory, which the registers pass through, so that no use moves before it.
__device__ __forceinline__ void pl_wait_ld16(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]),
                   "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}
__device__ __forceinline__ uint32_t pl_in_first(uint32_t a)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(a));
    return r;
}

// Calls f(row, k, value), by whole warps and in a fixed order, for the left-overs of `blocks` blocks of 16 rows from block b0 on with
// k in [64 k0, 64 k1).
template <class F>
__device__ __forceinline__ void pl_cells(const uint8_t *counts, const uint2 *cells, int groups, int64_t b0, int blocks, int k0, int k1, F f)
{
    const int lane = threadIdx.x & 31, g0 = k0 / (TC_GROUP_K / TC_AK), ng = (k1 - 1) / (TC_GROUP_K / TC_AK) + 1 - g0, total = blocks * ng;
    for (int base = 0; base < total; base += 32) {
        const int i = base + lane;
        const int64_t cell = i < total ? (b0 + i / ng) * groups + g0 + i % ng : 0;
        const uint32_t n = i < total ? __ldcg(counts + cell) : 0u;
        uint32_t some = __ballot_sync(0xffffffffu, n != 0u);
        while (some != 0u) {
            const int l = __ffs(some) - 1;
            some &= some - 1u;
            const int cnt = (int)__shfl_sync(0xffffffffu, n, l);
            const int64_t c = __shfl_sync(0xffffffffu, cell, l);
            const int64_t row0 = c / groups * TC_SUB, kg = c % groups * TC_GROUP_K;
            for (int e = 0; e < cnt; ++e) {
                const uint2 ent = __ldcg(cells + c * CN_CELL + e);
                const int64_t k = kg + (ent.x & 0xffffu);
                if (k >= (int64_t)k0 * TC_AK && k < (int64_t)k1 * TC_AK) f(row0 + (ent.x >> 16), k, __uint_as_float(ent.y));
            }
        }
    }
}

// Whether there are any, in two steps with room for other work between them: the lanes' first counts, then the others.
__device__ __forceinline__ uint32_t pl_first(const uint8_t *counts, int groups, int64_t b0, int blocks, int k0, int k1)
{
    const int g0 = k0 / (TC_GROUP_K / TC_AK), ng = (k1 - 1) / (TC_GROUP_K / TC_AK) + 1 - g0, i = threadIdx.x & 31;
    if (ng == 1) return i < blocks ? __ldcg(counts + (b0 + i) * groups + g0) : 0u;   // without the divisions, on every short tile's way
    return i < blocks * ng ? __ldcg(counts + (b0 + i / ng) * groups + g0 + i % ng) : 0u;
}
__device__ __forceinline__ bool pl_any(uint32_t any, const uint8_t *counts, int groups, int64_t b0, int blocks, int k0, int k1)
{
    const int g0 = k0 / (TC_GROUP_K / TC_AK), ng = (k1 - 1) / (TC_GROUP_K / TC_AK) + 1 - g0, total = blocks * ng;
    for (int i = (threadIdx.x & 31) + 32; i < total; i += 32) any |= __ldcg(counts + (b0 + i / ng) * groups + g0 + i % ng);
    return __any_sync(0xffffffffu, any != 0u);
}

template <bool MODE3X, bool SHORT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PL_THREADS, 1)
cn_gemm_planes_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_c, const __grid_constant__ PlParams p)
{
    using Cfg = PlCfg<MODE3X, SHORT>;
    extern __shared__ __align__(256) uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    auto full_bar = [&](int s) { return smem_base + Cfg::BAR_OFF + 8u * s; };                             // first CTA: both CTAs' tiles have landed
    auto empty_bar = [&](int s) { return smem_base + Cfg::BAR_OFF + 8u * (Cfg::STAGES + s); };            // each CTA: the stage has been multiplied
    auto accfull_bar = [&](int b) { return smem_base + Cfg::BAR_OFF + 8u * (2 * Cfg::STAGES + b); };      // each CTA
    auto accempty_bar = [&](int b) { return smem_base + Cfg::BAR_OFF + 8u * (2 * Cfg::STAGES + 2 + b); }; // first CTA: both CTAs have drained it
    const uint32_t tmem_holder = smem_base + Cfg::HOLD_OFF, abort_flag = tmem_holder + 4, skip_flag = tmem_holder + 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = blockIdx.x & 1u;
    cn_pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(accfull_bar(b), 1); mbar_init(accempty_bar(b), 16); }
        sts1u(abort_flag, 0u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tma_prefetch_map(&tm_w);
        tma_prefetch_map(&tm_a);
        if (p.tma_out) tma_prefetch_map(&tm_c);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_holder), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    cn_pdl_wait();
    // one thread looks at the word: the reads of every warp of all CTAs meet in one line
    if (threadIdx.x == 0) {
        const bool over = __ldcg(p.many + (CN_STATUS_OVERFLOW - CN_STATUS_MANY)) != 0u;
        if (blockIdx.x == 0) *p.many = over ? 1u : 0u;
        sts1u(skip_flag, over ? 1u : 0u);
    }
    __syncthreads();
    tc_fence_after();
    const bool skip = lds1u(skip_flag) != 0u;
    const uint32_t tmem_base = lds1u(tmem_holder);

    if (skip) {
        // the streaming kernel does it
    } else if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PL_REGS_WG0));
        // Whole warps wait, which takes half as long as by one lane; one lane issues.
        if (warp == 0) {
            // ------------------------------------------------------------ TMA producer of this CTA's halves
            PlWalk walk(p);
            int tile, k0, k1, slot;
            uint32_t it = 0;
            bool ok = true;
            while (ok && walk.next(p, tile, k0, k1, slot)) {
                const int32_t n0 = (tile / p.tiles_m) * 256 + (int)rank * 128, m0 = (tile % p.tiles_m) * 2 * p.half + (int)rank * p.half;
                for (int st = k0; st < k1; ++st, ++it) {
                    const int s = it % Cfg::STAGES;
                    ok = mbar_wait_warp(empty_bar(s), ((it / Cfg::STAGES) & 1u) ^ 1u, abort_flag, p.status, 19u);
                    if (!ok) break;
                    if (lane == 0) {
                        if (rank == 0) mbar_expect_tx(full_bar(s), (uint32_t)(2 * Cfg::PARTS * (PL_TILE_BYTES + p.half * TC_AK * 2)));
                        const uint32_t bar = pl_in_first(full_bar(s)), dst = smem_base + s * Cfg::STAGE_BYTES;
#pragma unroll
                        for (int part = 0; part < Cfg::PARTS; ++part) {
                            pl_load(dst + part * PL_TILE_BYTES, &tm_w, bar, st * TC_AK, n0, part);
                            pl_load(dst + (Cfg::PARTS + part) * PL_TILE_BYTES, &tm_a, bar, st * TC_AK, m0, part);
                        }
                    }
                    __syncwarp();
                }
            }
            // the last stages must have been multiplied before the CTA may exit; after a wait that ran out, copies in flight get a
            // bounded chance to land
            for (uint32_t i = it > Cfg::STAGES ? it - Cfg::STAGES : 0; i < it && ok; ++i)
                ok = mbar_wait_warp(empty_bar(i % Cfg::STAGES), (i / Cfg::STAGES) & 1u, abort_flag, p.status, 20u);
            if (!ok) {
                const long long t0 = clock64();
                while (clock64() - t0 < 20000000LL) {}
            }
        } else if (warp == 1 && rank == 0) {
            // ------------------------------------------------------------ MMA issuer of the pair
            PlWalk walk(p);
            int tile, k0, k1, slot;
            const uint32_t idesc = make_idesc_f16(256, 2 * p.half);
            uint32_t it = 0, chains = 0;
            bool ok = true;
            while (ok && walk.next(p, tile, k0, k1, slot)) {
                for (int st = k0; st < k1 && ok; ++st, ++it) {
                    const int s = it % Cfg::STAGES, ab = chains & 1u;
                    const bool first = st == k0 || (st & (p.chain - 1)) == 0;
                    if (first) {   // both CTAs' drain warps must have emptied this accumulator
                        const uint32_t parity = ((chains >> 1) & 1u) ^ 1u;
                        ok = mbar_try_cluster(accempty_bar(ab), parity) != 0u || (mbar_wait(accempty_bar(ab), parity, abort_flag, p.status, 21u) &&
                                                                                 mbar_try_cluster(accempty_bar(ab), parity) != 0u);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                    }
                    ok = mbar_wait_warp(full_bar(s), (it / Cfg::STAGES) & 1u, abort_flag, p.status, 22u);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t acc = tmem_base + ab * 256u;
                    const uint64_t d = make_kmajor_sw128_desc(smem_base + s * Cfg::STAGE_BYTES);
                    const uint32_t hi = (uint32_t)(d >> 32), whi = (uint32_t)d, wlo = whi + (PL_TILE_BYTES >> 4), ahi = whi + (Cfg::PARTS * PL_TILE_BYTES >> 4),
                                   alo = ahi + (PL_TILE_BYTES >> 4);
                    const bool last = st == k1 - 1 || ((st + 1) & (p.chain - 1)) == 0;
                    if (lane == 0) {
                        // 16 fp16 per k-step: 32 bytes (descriptor units of 16 B).  In the first stage of a chain the products with a low part
                        // come first: an addition truncates what it adds to a large sum, and there is none yet.
                        if (MODE3X && first) {
#pragma unroll
                            for (int j = 0; j < TC_AK / 16; ++j) {
                                pl_mma_ss(acc, wlo + 2 * j, ahi + 2 * j, hi, idesc, j == 0 ? 0u : 1u);
                                pl_mma_ss(acc, whi + 2 * j, alo + 2 * j, hi, idesc, 1u);
                            }
                        }
#pragma unroll
                        for (int j = 0; j < TC_AK / 16; ++j) {
                            pl_mma_ss(acc, whi + 2 * j, ahi + 2 * j, hi, idesc, !MODE3X && first && j == 0 ? 0u : 1u);
                            if (MODE3X && !first) {
                                pl_mma_ss(acc, wlo + 2 * j, ahi + 2 * j, hi, idesc, 1u);
                                pl_mma_ss(acc, whi + 2 * j, alo + 2 * j, hi, idesc, 1u);
                            }
                        }
                        pl_commit(empty_bar(s));
                        if (last) pl_commit(accfull_bar(ab));
                    }
                    __syncwarp();
                    if (last) ++chains;
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------------------------------------------------------- drain + epilogue: a warpgroup per half of the rows m
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PL_REGS_DRAIN));
        const int wg = (warp - 4) >> 2, q = warp & 3, row = q * 32 + lane, half = p.half;
        const uint32_t src0 = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(wg * half);
        PlWalk walk(p);
        int tile, k0, k1, slot;
        uint32_t chains = 0, out_it = 0;
        bool ok = true, more = walk.next(p, tile, k0, k1, slot);
        // of a run, fetched while the one before it is stored: the first group's inverse scales, and whether it has left-overs
        int64_t n, m0, ma, nw, wb, ab0;
        int a_blocks, w_blocks;
        float my_inv, wi;
        uint32_t any_w, any_a;
        auto prepare = [&]() {
            n = (int64_t)(tile / p.tiles_m) * 256 + rank * 128 + row;
            m0 = (int64_t)(tile % p.tiles_m) * 2 * half + wg * half;
            ma = m0 + row < p.a_pad ? m0 + row : p.a_pad - 1;
            nw = n < p.w_pad ? n : p.w_pad - 1;
            const int g = k0 / (TC_GROUP_K / TC_AK);
            my_inv = p.a_inv[g * p.a_pad + ma];
            wi = p.w_inv[g * p.w_pad + nw];
            wb = (n - lane) / TC_SUB;   // two blocks of 16 columns per warp
            ab0 = m0 / TC_SUB;
            const int64_t left = p.a_pad / TC_SUB - ab0;
            a_blocks = left < half / TC_SUB ? (int)left : half / TC_SUB;
            w_blocks = n - lane < p.w_pad ? 2 : 0;
            any_w = pl_first(p.w_counts, p.groups, wb, w_blocks, k0, k1);
            any_a = pl_first(p.a_counts, p.groups, ab0, a_blocks, k0, k1);
        };
        if (more) prepare();
        while (ok && more) {
            uint64_t sum[64];   // pairs of rows
#pragma unroll
            for (int i = 0; i < 64; ++i) sum[i] = 0ull;
            int have = k0 / (TC_GROUP_K / TC_AK);
            for (int st = k0; st < k1; ++chains) {
                const int ab = chains & 1u, group = st / (TC_GROUP_K / TC_AK);
                int next = (st & ~(p.chain - 1)) + p.chain;
                if (next > k1) next = k1;
                if (group != have) {
                    my_inv = p.a_inv[group * p.a_pad + ma];
                    wi = p.w_inv[group * p.w_pad + nw];
                    have = group;
                }
                const uint32_t as = smem_base + Cfg::AS_OFF + ((chains & 1u) * 256 + wg * 128) * 4;
                sts1(as + row * 4, my_inv);
                ok = mbar_wait<TC_DRAIN_SLEEP_NS>(accfull_bar(ab), (chains >> 1) & 1u, abort_flag, p.status, 23u);
                {   // all 128 threads of the warpgroup go on together or not at all
                    uint32_t all_ok;
                    asm volatile(
                        "{\n\t.reg .pred pi, po;\n\t"
                        "setp.ne.u32 pi, %1, 0;\n\t"
                        "bar.red.and.pred po, %2, 128, pi;\n\t"
                        "selp.u32 %0, 1, 0, po;\n\t}"
                        : "=r"(all_ok) : "r"((uint32_t)ok), "r"(1 + wg) : "memory");
                    ok = all_ok != 0;
                }
                if (!ok) break;
                tc_fence_after();
                const uint64_t wi2 = tc_pack2(wi, wi);
                const uint32_t src = src0 + ab * 256u;
                uint32_t r[2][16];   // the next 16 columns are on their way while these are added
                tc_ld_ahead(src, r[0]);
#pragma unroll
                for (int cc = 0; cc < 8; ++cc) {
                    if (cc * 16 >= half) break;
                    pl_wait_ld16(r[cc & 1]);
                    if (cc < 7 && cc * 16 + 16 < half) tc_ld_ahead(src + cc * 16 + 16, r[(cc + 1) & 1]);
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const float4 f = lds4(as + (cc * 16 + i) * 4);
                        uint64_t &s0 = sum[(cc * 16 + i) / 2], &s1 = sum[(cc * 16 + i) / 2 + 1];
                        const uint32_t *v = r[cc & 1] + i;
                        s0 = tc_fma2(tc_pack2(__uint_as_float(v[0]), __uint_as_float(v[1])), tc_mul2(tc_pack2(f.x, f.y), wi2), s0);
                        s1 = tc_fma2(tc_pack2(__uint_as_float(v[2]), __uint_as_float(v[3])), tc_mul2(tc_pack2(f.z, f.w), wi2), s1);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(pl_in_first(accempty_bar(ab))) : "memory");
                st = next;
            }
            if (!ok) break;
            // what the parts left: of the weights' elements, times the activations ...
            if (pl_any(any_w, p.w_counts, p.groups, wb, w_blocks, k0, k1))
                pl_cells(p.w_counts, p.w_cells, p.groups, wb, w_blocks, k0, k1, [&](int64_t r, int64_t k, float left) {
                    const bool mine = r == n;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (j * 32 >= half) break;
                        const int64_t m = m0 + j * 32 + lane;
                        const float a = m < p.M ? p.A[m * p.a_m + k * p.a_k] : 0.0f;
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const float a0 = __shfl_sync(0xffffffffu, a, i), a1 = __shfl_sync(0xffffffffu, a, i + 1);
                            uint64_t &s = sum[(j * 32 + i) / 2];
                            if (mine) s = tc_fma2(tc_pack2(a0, a1), tc_pack2(left, left), s);
                        }
                    }
                });
            // ... and of the activations' elements, times the weights' parts
            if (pl_any(any_a, p.a_counts, p.groups, ab0, a_blocks, k0, k1))
                pl_cells(p.a_counts, p.a_cells, p.groups, ab0, a_blocks, k0, k1,
                         [&](int64_t r, int64_t k, float left) {
                             float w = 0.0f;
                             if (n < p.N) {
                                 const uint16_t *at = p.w_planes + n * p.Kp + k;
                                 w = __half2float(__ushort_as_half(__ldcg(at)));
                                 if (MODE3X) w += __half2float(__ushort_as_half(__ldcg(at + p.w_plane)));
                                 w *= p.w_inv[k / TC_GROUP_K * p.w_pad + n];
                             }
                             const float add = left * w;
                             const int ml = (int)(r - m0);
#pragma unroll
                             for (int i = 0; i < 128; i += 2) {
                                 sum[i / 2] = tc_add2(sum[i / 2], tc_pack2(ml == i ? add : 0.0f, ml == i + 1 ? add : 0.0f));
                             }
                         });
            const int64_t nw0 = n - lane, mt = m0;
            const int part = slot;
            const float bias = (part < 0 && p.bias && n < p.N) ? p.bias[n] : 0.0f;
            more = walk.next(p, tile, k0, k1, slot);
            if (more) prepare();
            if (part >= 0) {
                // partial tile: float4 number i of 32 for all 128 columns, then the next, so that a warp writes 512 contiguous bytes
                ulonglong2 *P = reinterpret_cast<ulonglong2 *>(p.partials) + (((int64_t)part * 2 + wg) * 2 + rank) * (TC_BM * TC_BN / 4) + row;
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (i * 4 < half) P[i * TC_BN] = make_ulonglong2(sum[2 * i], sum[2 * i + 1]);
                continue;
            }
            // Every lane holds a column of its own.  Blocks of 16 rows x 32 columns go through buffers of shared memory, 16-byte chunks
            // permuted as the tensor map says, which keeps eight lanes that store together apart, and from there to C by TMA while the warp
            // fills another one or has gone on to the next tile.  Short code: a launch fetches it once, and 128 values with a bias and a choice of
            // units each took 15000 clocks of the first tile.  32-byte stores from registers, each lane into a column of
            // its own, took 8400 clocks per tile, in which nothing was drained.
            const uint32_t turn = smem_base + Cfg::TURN_OFF + (uint32_t)((warp - 4) * Cfg::TURN_BYTES);
            if (p.bias) {
                const uint64_t bias2 = tc_pack2(bias, bias);
#pragma unroll
                for (int i = 0; i < 64; ++i) sum[i] = tc_add2(sum[i], bias2);
            }
            if (p.tma_out) {
                const int blocks = nw0 < p.N && mt < p.M ? ((int)(p.M - mt < half ? p.M - mt : half) + 15) >> 4 : 0;
                const uint32_t turned = (uint32_t)(lane >> 1 & 3) * 16u;
                // room for the next BATCH blocks, when the batch before the last has left it
                auto take = [&]() {
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    __syncwarp();
                    return turn + (out_it++ & 1u) * (Cfg::BATCH * 2048u);
                };
                auto put = [&](uint32_t buf, int i, auto unit) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        float v[4];
                        tc_unpack2(sum[8 * i + 2 * c], v[0], v[1]);
                        tc_unpack2(sum[8 * i + 2 * c + 1], v[2], v[3]);
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(buf + (uint32_t)lane * 64u + ((uint32_t)c * 16u ^ turned)), "f"(unit(v[0])), "f"(unit(v[1])), "f"(unit(v[2])), "f"(unit(v[3])) : "memory");
                    }
                };
                // blocks first to last - 1 to C
                auto give = [&](uint32_t buf, int first, int last) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
#pragma unroll 1
                        for (int i = first; i < last; ++i, buf += 2048u) pl_store(&tm_c, buf, (int32_t)mt + 16 * i, (int32_t)nw0);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                };
                auto straight = [&](auto unit) {
#pragma unroll
                    for (int i = 0; i < 8; i += Cfg::BATCH) {
                        if (i >= blocks) break;
                        const uint32_t buf = take();
#pragma unroll
                        for (int b = 0; b < Cfg::BATCH; ++b)
                            if (i + b < 8) put(buf + 2048u * b, i + b, unit);
                        give(buf, i, blocks < i + Cfg::BATCH ? blocks : i + Cfg::BATCH);
                    }
                };
                if (p.act == CN_ACT_LINEAR) {
                    straight([](float x) { return x; });
                } else if (p.act == CN_ACT_RELU) {
                    straight([](float x) { return fmaxf(x, 0.0f); });   // 0 for a NaN, as x > 0 ? x : 0
                } else if (p.act == CN_ACT_LOGISTIC && p.stages <= PL_DIRECT_STAGES && mt + half <= p.M && (p.ldc & 7) == 0 && (reinterpret_cast<uintptr_t>(p.C) & 31u) == 0) {
                    // short tiles are bound by the function itself: straight code, and no trip through shared memory (704 x 592 . 592 x 9176, single pass, 55 us, 63
                    // by the way below)
                    float *q = p.C + (nw0 + lane) * p.ldc + mt;
#pragma unroll
                    for (int i = 0; i < 128; i += 8) {
                        if (i >= half) break;
                        float v[8];
#pragma unroll
                        for (int e = 0; e < 8; e += 2) tc_unpack2(sum[(i + e) / 2], v[e], v[e + 1]);
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] = cn_apply_activation(v[e], CN_ACT_LOGISTIC);
                        if (nw0 + lane < p.N) stg8(q + i, v);
                    }
                } else {
                    // one copy of the units' longer code (1736 x 2000 . 2000 x 4800 with logistic units: 160 us with straight code, 137)
#pragma unroll 1
                    for (int b = 0; b < blocks; ++b) {
                        const uint32_t buf = take();
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (b == i) put(buf, i, [](float x) { return x; });
                        float v[16];
                        const uint32_t at = buf + (uint32_t)lane * 64u;
#pragma unroll
                        for (int e = 0; e < 16; e += 4) {
                            const float4 q = lds4(at + 4u * e);
                            v[e] = q.x; v[e + 1] = q.y; v[e + 2] = q.z; v[e + 3] = q.w;
                        }
                        if (p.act == CN_ACT_LOGISTIC) {
#pragma unroll
                            for (int e = 0; e < 16; ++e) v[e] = cn_apply_activation(v[e], CN_ACT_LOGISTIC);
                        } else {
#pragma unroll
                            for (int e = 0; e < 16; ++e) v[e] = cn_apply_activation(v[e], CN_ACT_DOUBLE_RELU);
                        }
#pragma unroll
                        for (int e = 0; e < 16; e += 4)
                            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at + 4u * e), "f"(v[e]), "f"(v[e + 1]), "f"(v[e + 2]), "f"(v[e + 3]) : "memory");
                        give(buf, b, b + 1);
                    }
                }
                __syncwarp();   // the next tile's tensor-memory loads need the whole warp
                continue;
            }
            // Columns of C that do not start on 16 bytes: blocks of 32 columns x 32 rows are turned in shared memory (16-byte chunks permuted
            // by the column against bank conflicts), so that a warp stores a column's rows together.
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                if (b * 32 >= half || mt + b * 32 >= p.M) break;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    float v[4];
                    tc_unpack2(sum[b * 16 + 2 * c], v[0], v[1]);
                    tc_unpack2(sum[b * 16 + 2 * c + 1], v[2], v[3]);
                    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(turn + lane * 128 + ((uint32_t)(c ^ (lane & 7)) << 4)), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
                }
                if (p.act != CN_ACT_LINEAR) {
#pragma unroll 1
                    for (int i = 0; i < 8; ++i) {   // 16-byte chunk i of this lane's row
                        const uint32_t at = turn + lane * 128 + ((uint32_t)(i ^ (lane & 7)) << 4);
                        const float4 v = lds4(at);
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(cn_apply_activation(v.x, p.act)), "f"(cn_apply_activation(v.y, p.act)),
                                     "f"(cn_apply_activation(v.z, p.act)), "f"(cn_apply_activation(v.w, p.act)) : "memory");
                    }
                }
                __syncwarp();
                const int rows = half - b * 32 < 32 ? half - b * 32 : 32;   // 16 or 32 of the block belong to this warpgroup
                const int64_t m = mt + b * 32 + lane;
                float *q = p.C + nw0 * p.ldc + m;
                const int cols = lane < rows && m < p.M ? (int)(p.N - nw0 < 32 ? p.N - nw0 : 32) : 0;
#pragma unroll 4
                for (int col = 0; col < cols; ++col, q += p.ldc) *q = lds1(turn + col * 128 + ((uint32_t)((lane >> 2) ^ (col & 7)) << 4) + (lane & 3) * 4);
                __syncwarp();
            }
            __syncwarp();   // the next tile's tensor-memory loads need the whole warp
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    __syncwarp();
    tc_fence_before();
    // neither CTA may leave while the other's MMAs read its shared memory or its commits arrive here
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------------ host
// Geometry of the planes of an M x K operand in one allocation.
void cn_plane_layout(int64_t M, int64_t K, int mode, cn_planes *pl, int bands)
{
    pl->parts = mode == CN_GEMM_3XTF32 ? 2 : 1;
    pl->bands = bands;
    pl->Kp = (K + TC_AK - 1) / TC_AK * TC_AK;
    pl->plane = (M * pl->Kp + 127) / 128 * 128;
    pl->m_pad = (M + TC_BM - 1) / TC_BM * TC_BM;
    pl->groups = (K + TC_GROUP_K - 1) / TC_GROUP_K;
    const size_t cells = (size_t)(pl->m_pad / TC_SUB) * pl->groups;
    pl->inv_off = (size_t)bands * pl->parts * pl->plane * sizeof(uint16_t);
    pl->bands_off = pl->inv_off + (size_t)bands * pl->groups * pl->m_pad * sizeof(float);
    pl->counts_off = (pl->bands_off + (size_t)(pl->m_pad / TC_SUB) * (pl->Kp / TC_AK) + 15) & ~(size_t)15;
    pl->cells_off = (pl->counts_off + cells + 15) & ~(size_t)15;
    pl->bytes = pl->cells_off + cells * CN_CELL * sizeof(uint2);
}

// overflow: also make cells of left-overs, and raise this word where one has no room
static int make_job(ActJob *job, int64_t rows, int64_t K, const float *src, int64_t ld, const cn_planes &pl, void *planes, unsigned int *overflow, bool optional)
{
    const int64_t ctas = pl.groups * (pl.m_pad / ACT_ROWS);
    CN_REQUIRE(ctas < (1LL << 30), CN_ERR_UNSUPPORTED, "cn_gemm_f32: activation matrix too large for the split pre-pass");
    uint8_t *base = (uint8_t *)planes;
    job->A = src; job->lda = ld; job->M = rows; job->K = K; job->ctas = (int)ctas;
    ActPlanes &ap = job->pl;
    ap.p = reinterpret_cast<uint16_t *>(base);
    ap.plane = pl.plane; ap.Kp = pl.Kp; ap.m_pad = pl.m_pad; ap.groups = pl.groups;
    ap.inv = reinterpret_cast<float *>(base + pl.inv_off);
    ap.bands = pl.bands > 1 ? base + pl.bands_off : nullptr;
    ap.stages = (int)(pl.Kp / TC_AK);
    ap.nbands = pl.bands;
    ap.counts = overflow ? base + pl.counts_off : nullptr;
    ap.cells = reinterpret_cast<uint2 *>(base + pl.cells_off);
    ap.overflow = overflow;
    ap.optional = optional;
    return CN_OK;
}

template <bool LO>
static cudaError_t launch_jobs(int kind0, int kind1, const ActJob &j0, const ActJob &j1, const ActCoded &cd, size_t smem, cudaStream_t s)
{
    const dim3 grid((unsigned)(j0.ctas + (kind1 == ACT_NONE ? 0 : j1.ctas)));
#define CN_JOBS(A, W) \
    if (kind0 == A && kind1 == W) return cn_launch_pdl(cn_act_planes_kernel<LO, A, W>, grid, 256, smem, s, j0, j1, cd)
    CN_JOBS(ACT_ROWS_M, ACT_NONE); CN_JOBS(ACT_ROWS_K, ACT_NONE); CN_JOBS(ACT_CODED, ACT_NONE);
    CN_JOBS(ACT_ROWS_M, ACT_ROWS_M); CN_JOBS(ACT_ROWS_M, ACT_ROWS_K); CN_JOBS(ACT_ROWS_K, ACT_ROWS_M); CN_JOBS(ACT_ROWS_K, ACT_ROWS_K);
#undef CN_JOBS
    return cudaErrorInvalidValue;
}

int cn_make_planes(cn_context *ctx, bool k_contiguous, int64_t rows, int64_t K, const float *src, int64_t ld, const cn_coded_src *cs, const cn_planes &pl,
                   void *planes, cudaStream_t s)
{
    ActJob job;
    ActCoded cd = {};
    const int st = make_job(&job, rows, K, src, ld, pl, planes, nullptr, false);
    if (st != CN_OK) return st;
    if (cs) {
        cd.codes = cs->codes; cd.scales = cs->scales; cd.tbl = ctx->d_tbl; cd.own_fp32 = cs->own_fp32;
        cd.own_rank = cs->own_rank; cd.nranks = cs->nranks;
    }
    const int kind = cs ? ACT_CODED : k_contiguous ? ACT_ROWS_K : ACT_ROWS_M;
    const size_t smem = cs ? (size_t)cs->nranks * 256 * sizeof(float) : 0;
    CN_CUDA(pl.parts == 2 ? launch_jobs<true>(kind, ACT_NONE, job, job, cd, smem, s) : launch_jobs<false>(kind, ACT_NONE, job, job, cd, smem, s));
    cn_count_launch();
    return CN_OK;
}

int cn_gemm_tc_split_activations(cn_context *ctx, int transA, int64_t M, int64_t K, const float *A, int64_t lda, int mode, void *planes, cudaStream_t s)
{
    cn_planes pl;
    cn_plane_layout(M, K, mode, &pl);
    return cn_make_planes(ctx, transA != 0, M, K, A, lda, nullptr, pl, planes, s);
}

int cn_make_planes_map(EncodeTiledFn enc, CUtensorMap *map, const uint16_t *base, int64_t Kp, int64_t rows, int64_t plane, int planes, int box_rows)
{
    cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, (cuuint64_t)planes};
    cuuint64_t strides[2] = {(cuuint64_t)Kp * sizeof(uint16_t), (cuuint64_t)plane * sizeof(uint16_t)};
    cuuint32_t box[3] = {(cuuint32_t)TC_AK, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<uint16_t *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CN_REQUIRE(r == CUDA_SUCCESS, CN_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d (planes %lld x %lld)", (int)r, (long long)rows, (long long)Kp);
    return CN_OK;
}

#define PL_MAX_W_BYTES (2LL << 30)   // of workspace for the planes of the weights

// Work decomposition: tiles of 256 columns n by as many rows as divide M evenly, in steps of 32, at most 256
struct PlCut {
    int64_t tiles_m, tiles, full, tail_pairs;
    int half, stages;
};
static PlCut pl_decompose(const cn_context *ctx, int64_t M, int64_t N, int64_t K)
{
    PlCut c;
    c.tiles_m = (M + 255) / 256;
    c.tiles = c.tiles_m * ((N + 255) / 256);
    c.half = (int)(((M + c.tiles_m - 1) / c.tiles_m + 31) / 32 * 16);
    c.stages = (int)((K + TC_AK - 1) / TC_AK);
    const int64_t max_pairs = ctx->sm_count / 2;
    // as in cn_tc_decompose; the reduction of a cut tail takes as long as about 6 stages
    const int64_t rounds = (c.tiles + max_pairs - 1) / max_pairs;
    c.full = c.tiles;
    c.tail_pairs = 0;
    if (rounds * c.stages > c.tiles * c.stages / max_pairs + 6) {
        c.full = c.tiles / max_pairs * max_pairs;
        const int64_t rest = c.tiles - c.full;
        c.tail_pairs = rest * c.stages / 3;
        if (c.tail_pairs > max_pairs) c.tail_pairs = max_pairs;
        if (c.tail_pairs < rest) c.tail_pairs = rest < max_pairs ? rest : max_pairs;
    }
    return c;
}
// Share of the rounds' places that have a tile.
static double pl_busy(int64_t tiles, int64_t places) { return (double)tiles / (double)((tiles + places - 1) / places * places); }

// Writing and reading the planes of the weights costs as much as the streaming kernel's conversions for three to four blocks of 128
// rows (3x mode, this kernel / streaming kernel, us; 4096 x 4096 weights: 77 / 60 with 256 rows, 86 / 87 with 512, 111 / 126 with 800, 187 / 263
// with 2048; 2000 x 20000: 138 / 105, 175 / 173, 223 / 268).  In the single pass the streaming kernel saves less on its conversions, and
// weights that TMA cannot read cost it more (512 rows, 4096 x 4096: 62 / 72; 4097 x 4099: 93 / 101).  With fewer than 256 columns
// half of a pair idles.
//
// A pair's last tile costs as much as its others, so that a last round with few tiles is lost where K is too short to be cut.  Two rounds of
// the small products' kernel (`fine`) are as fast up to K = 128 where the pairs are less than three quarters busy (3x mode, this kernel / the
// other one, us: 1056 x 40 . 40 x 4096, 80 tiles for 2 x 74, 28 / 23; 2800 x 72 . 72 x 1000 28 / 23; 800 x 72 . 72 x 4096, 64 for 74, 22 / 24; 1056 x 264
// . 264 x 4096 37 / 36).  The streaming kernel is where its own rounds of 148 CTAs are fuller (520 x 264 . 264 x 19112, 225 tiles for 4 x
// 74 against 375 for 3 x 148, 62 / 45; 800 x 324 . 324 x 10552 49 / 43; 1056 x 264 . 264 x 19112 89 / 81), in the 3x mode: the single pass has
// shorter tiles (600 x 152 . 152 x 19112 0.94 of the streaming kernel's time).
bool cn_gemm_planes_shape(const cn_context *ctx, int64_t M, int64_t N, int64_t K, int mode, bool w_aligned, bool fine)
{
    if (M <= (mode == CN_GEMM_3XTF32 && w_aligned ? 512 : 384) || N < 256 || K < 1) return false;
    if (K >= (1LL << 31) - 64 || M >= (1LL << 31) - 512 || N >= (1LL << 31) - 512) return false;
    if (!w_aligned && cn_gemm_any_chain(K) < TC_AK / TC_WK) return false;   // chains shorter than a stage
    cn_planes pl;
    cn_plane_layout(N, K, mode, &pl, 1);
    if (pl.bytes > (size_t)PL_MAX_W_BYTES) return false;
    const PlCut c = pl_decompose(ctx, M, N, K);
    if (c.tail_pairs > 0 || K > 512) return true;
    const double busy = pl_busy(c.tiles, ctx->sm_count / 2);
    if (fine) return K > 128 || busy >= 0.75;
    if (mode != CN_GEMM_3XTF32 || busy >= 0.85) return true;
    const cn_tc_cut s = cn_tc_decompose(ctx, M, N, K, CN_TC_ALONE, false);
    return (s.rest() > 0 ? 1.0 : pl_busy(s.tiles, ctx->sm_count)) <= busy + 0.06;
}

// Stages per accumulation chain.  The error grows with the chain (2-norm against fp64, uniform operands, 3x mode: 4.3e-7 with 128 k,
// 9.2e-7 with 256, 1.8e-6 with 512; the streaming kernel's chains of 512: 1.87e-6, less where it ends a chain at left-overs or cuts a
// tile along K into shorter ones), and draining one costs little: 4096^3 331 us with 512 k, 344 with 256.  So 256 k; 128 where K is
// short; 64 where the small products' kernel, whose chains are as short there, would else have the shape (`fine`).  The single pass, whose
// operands are rounded to 2.6e-4, has no time to drain more often than every 512 k (186 us, 229 with 256).
static int planes_chain(int64_t K, int mode, bool w_aligned, bool fine)
{
    if (!w_aligned) return cn_gemm_any_chain(K) / (TC_AK / TC_WK);
    return mode != CN_GEMM_3XTF32 ? 8 : K <= 128 && fine ? 1 : K <= 512 ? 2 : 4;
}


// C (M x N, column-major) in blocks of 16 rows by 32 columns, 64 bytes of a column per line of shared memory.
static int pl_make_out_map(EncodeTiledFn enc, CUtensorMap *map, float *C, int64_t M, int64_t N, int64_t ldc)
{
    cuuint64_t dims[2] = {(cuuint64_t)M, (cuuint64_t)N};
    cuuint64_t strides[1] = {(cuuint64_t)ldc * sizeof(float)};
    cuuint32_t box[2] = {16, 32};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, C, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CN_REQUIRE(r == CUDA_SUCCESS, CN_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d (output %lld x %lld)", (int)r, (long long)M, (long long)N);
    return CN_OK;
}

template <bool MODE3X, bool SHORT>
static int planes_launch_cfg(cn_context *ctx, const CUtensorMap &mw, const CUtensorMap &ma, const CUtensorMap &mc, const PlParams &prm, int64_t pairs, cudaStream_t s)
{
    constexpr int smem = PlCfg<MODE3X, SHORT>::SMEM_BYTES;
    static bool attr_set[64] = {};   // per device: the attribute belongs to the device's copy of the function
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        CN_CUDA(cudaFuncSetAttribute(cn_gemm_planes_kernel<MODE3X, SHORT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    CN_CUDA(cn_launch_pdl(cn_gemm_planes_kernel<MODE3X, SHORT>, dim3((unsigned)(2 * pairs)), PL_THREADS, smem, s, mw, ma, mc, prm));
    cn_count_launch();
    return CN_OK;
}

int cn_gemm_planes_launch(cn_context *ctx, int64_t M, int64_t N, int64_t K, const float *A, int64_t lda, const float *B, int64_t ldb, float *C, int64_t ldc,
                          const cn_epilogue *epi, int mode, cudaStream_t s, int transA, int transB, bool w_aligned, bool fine, bool *done)
{
    *done = false;
    EncodeTiledFn enc = nullptr;
    int st = cn_get_encode_fn(ctx, &enc);
    if (st != CN_OK) return st;
    unsigned int *d_status = nullptr;
    if ((st = cn_status_block(ctx, &d_status)) != CN_OK) return st;
    cn_planes pa, pw;
    cn_plane_layout(M, K, mode, &pa);
    cn_plane_layout(N, K, mode, &pw, 1);

    const PlCut cut = pl_decompose(ctx, M, N, K);
    const int64_t tiles_m = cut.tiles_m, tiles = cut.tiles, full = cut.full, tail_pairs = cut.tail_pairs, max_pairs = ctx->sm_count / 2;
    const int half = cut.half, stages = cut.stages;
    const int64_t rest = tiles - full, pairs = tail_pairs > (full < max_pairs ? full : max_pairs) ? tail_pairs : (full < max_pairs ? full : max_pairs);
    size_t part_bytes = rest > 0 ? (size_t)(tail_pairs + rest) * 4 * TC_BM * TC_BN * sizeof(float) : 0;
    // the streaming kernel behind this one finds its room before anything is launched
    const size_t other_bytes = cn_tc_decompose(ctx, M, N, K, CN_TC_BEHIND, false).partial_bytes();
    if (part_bytes < other_bytes) part_bytes = other_bytes;
    if (tiles >= (1LL << 29)) return CN_OK;
    // A workspace that would have to grow cannot while the stream records a graph.  The small products' kernel needs none, and a graph that
    // it was recorded in may be replayed after a larger product has had the workspaces moved.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const bool recorded = cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone;
    const size_t *have = ctx->gemm->bytes;
    if (recorded && (fine || have[CN_GEMM_SLOT_ASPLIT] < pa.bytes || have[CN_GEMM_SLOT_WSPLIT] < pw.bytes || have[CN_GEMM_SLOT_SPLITK] < part_bytes)) return CN_OK;
    // The planes of the weights last: the streaming kernel, which takes the product where they find no room, needs the other two, and either
    // of those may make room by giving the last product's planes of the weights back.
    void *ba = nullptr, *bw = nullptr, *parts = nullptr;
    if (cn_gemm_scratch(ctx, CN_GEMM_SLOT_ASPLIT, pa.bytes, &ba) != CN_OK || (part_bytes && cn_gemm_scratch(ctx, CN_GEMM_SLOT_SPLITK, part_bytes, &parts) != CN_OK) ||
        cn_gemm_scratch(ctx, CN_GEMM_SLOT_WSPLIT, pw.bytes, &bw) != CN_OK)
        return CN_OK;
    if (recorded) ctx->gemm->wsplit_recorded = true;
    *done = true;
    ActJob ja, jw;
    unsigned int *overflow = d_status + CN_STATUS_OVERFLOW;
    if ((st = make_job(&ja, M, K, A, lda, pa, ba, overflow, false)) != CN_OK || (st = make_job(&jw, N, K, B, ldb, pw, bw, overflow, true)) != CN_OK) return st;
    const int ka = transA ? ACT_ROWS_K : ACT_ROWS_M, kw = transB ? ACT_ROWS_M : ACT_ROWS_K;
    CN_CUDA(mode == CN_GEMM_3XTF32 ? launch_jobs<true>(ka, kw, ja, jw, ActCoded(), 0, s) : launch_jobs<false>(ka, kw, ja, jw, ActCoded(), 0, s));
    cn_count_launch();
    cudaEvent_t stop = nullptr;
    if ((st = cn_gemm_profile_start(ctx, s, &stop)) != CN_OK) return st;
    const uint8_t *a8 = (const uint8_t *)ba, *w8 = (const uint8_t *)bw;

    PlParams prm;
    prm.M = M; prm.N = N;
    prm.C = C; prm.ldc = ldc;
    prm.bias = epi ? epi->bias : nullptr;
    prm.act = epi ? epi->activation : CN_ACT_LINEAR;
    prm.tiles_m = (int)tiles_m; prm.half = half;
    prm.full_tiles = (int)full; prm.tiles = (int)tiles; prm.tail_pairs = (int)tail_pairs;
    prm.stages = stages;
    prm.chain = planes_chain(K, mode, w_aligned, fine);
    prm.groups = (int)pa.groups;
    prm.a_inv = reinterpret_cast<const float *>(a8 + pa.inv_off); prm.w_inv = reinterpret_cast<const float *>(w8 + pw.inv_off);
    prm.a_pad = pa.m_pad; prm.w_pad = pw.m_pad;
    prm.a_counts = a8 + pa.counts_off; prm.w_counts = w8 + pw.counts_off;
    prm.a_cells = reinterpret_cast<const uint2 *>(a8 + pa.cells_off); prm.w_cells = reinterpret_cast<const uint2 *>(w8 + pw.cells_off);
    prm.A = A; prm.a_m = transA ? lda : 1; prm.a_k = transA ? 1 : lda;
    prm.w_planes = reinterpret_cast<const uint16_t *>(w8);
    prm.Kp = pw.Kp; prm.w_plane = pw.plane;
    prm.many = d_status + CN_STATUS_MANY;
    prm.partials = (float *)parts;
    prm.status = d_status;

    CUtensorMap mw, ma, mc = {};
    if ((st = cn_make_planes_map(enc, &mw, reinterpret_cast<const uint16_t *>(bw), pw.Kp, N, pw.plane, pw.parts, 128)) != CN_OK) return st;
    if ((st = cn_make_planes_map(enc, &ma, reinterpret_cast<const uint16_t *>(ba), pa.Kp, M, pa.plane, pa.parts, half)) != CN_OK) return st;
    prm.tma_out = (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15u) == 0;
    if (prm.tma_out && (st = pl_make_out_map(enc, &mc, C, M, N, ldc)) != CN_OK) return st;
    const bool shorter = K <= (mode == CN_GEMM_3XTF32 ? 1 : 3) * PL_SHORT_K && prm.tma_out && prm.act != CN_ACT_LOGISTIC;
    if (mode == CN_GEMM_3XTF32) st = shorter ? planes_launch_cfg<true, true>(ctx, mw, ma, mc, prm, pairs, s) : planes_launch_cfg<true, false>(ctx, mw, ma, mc, prm, pairs, s);
    else                        st = shorter ? planes_launch_cfg<false, true>(ctx, mw, ma, mc, prm, pairs, s) : planes_launch_cfg<false, false>(ctx, mw, ma, mc, prm, pairs, s);
    if (st != CN_OK) return st;
    if (rest > 0) {
        ReduceParams rp = {};
        rp.partials = prm.partials; rp.nt = 2; rp.mt = 2; rp.rows = half; rp.tail_ctas = (int)tail_pairs; rp.kb_total = stages;
        rp.tail_tiles = (int)rest; rp.full_tiles = (int)full; rp.tiles_m = (int)tiles_m; rp.M = M; rp.N = N;
        rp.C = C; rp.ldc = ldc; rp.bias = prm.bias; rp.act = prm.act; rp.status = d_status;
        if ((st = cn_splitk_reduce_launch(ctx, rp, s)) != CN_OK) return st;
    }
    const cn_tc_cond cond = {prm.many, ba};
    st = cn_gemm_tc_launch(ctx, M, N, K, A, lda, B, ldb, C, ldc, epi, mode, s, nullptr, transA, transB, &cond);
    if (stop) CN_CUDA(cudaEventRecord(stop, s));
    return st;
}
