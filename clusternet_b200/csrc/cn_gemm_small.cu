// Small products for sm_100a: one launch, both operands split in the kernel, K split over a thread-block cluster.
//
// The streaming kernel (cn_gemm_tc.cu) takes three launches - planes of the activations, product, reduction - which is the
// right price for weights that have to come from HBM.  A layer of a small network (128 x 784 . 784 x 1024, the weight gradients
// and back-propagated errors of a 784-1200-1200-10 network) is over in a few microseconds; there the launches, the passes
// over memory between them and the idle SMs of a product with eight tiles are the cost.  Here
//   * a CTA takes a tile of 128 columns n by up to 128 rows m and a share of K.  Four warps load and split 128 x 32 blocks of
//     the weights, four those of the activations, straight from global memory in whatever layout they have (either operand
//     transposed or not, any alignment), with the next block's loads in flight while the current one is split;
//   * the operands are TF32 hi / lo parts in shared memory (K-major, 128-byte swizzle), three tcgen05.mma kind::tf32 products per
//     k-step as CN_GEMM_3XTF32 promises, one for CN_GEMM_TF32; one thread issues them;
//   * the CTAs of a cluster share a tile: each multiplies its part of K, sends every other CTA its slice of the partial tile
//     through distributed shared memory, adds the slices it received in K order (reproducible), and finishes its slice: bias,
//     activation, 512-byte runs of stores to C and, for the fused all-gather, to the peers.
// The tensor core's accumulator truncates, so a share of K (at most SM_MAX_BLOCKS_ANY blocks) is cut into as many chains as tensor memory
// holds accumulators for, four, and the chains are added in round-to-nearest fp32.
//
// Bound by latency.  128 x 784 . 784 x 1024 + bias + ReLU: 13.2 us a call, against 22.5 us in three launches.
#include "cn_epilogue.cuh"
#include "cn_gemm.h"
#include "cn_tc.cuh"

#define SM_BN 128
#define SM_BM 128
#define SM_BK 32
#define SM_THREADS 288          // warps 0-3: weights, 4-7: activations, 8: MMA issuer
#define SM_STAGES 2
#define SM_TILE_BYTES (128 * 128)
#define SM_STAGE_BYTES (4 * SM_TILE_BYTES)   // W hi, W lo, A hi, A lo
#define SM_MAX_BLOCKS 12
#define SM_MAX_BLOCKS_ANY 16   // weights that TMA cannot read, of which the streaming kernel wants four rows at least
#define SM_MAX_CHAINS 4
#define SM_MAX_CLUSTER 8
#define SM_RING_BYTES (SM_STAGES * SM_STAGE_BYTES)
#define SM_TURN_BYTES (SM_BN * SM_BM * 4)
#define SM_SMEM_BYTES(cluster) (1024 + SM_RING_BYTES + ((cluster) > 1 ? SM_TURN_BYTES : 0))

// How an operand lies in memory: k contiguous with 16-byte rows, k contiguous otherwise, or the tile's rows contiguous.
enum { SM_K_VEC = 0, SM_K_SCALAR = 1, SM_ROWS = 2 };

struct SmallParams {
    const float *W, *A;
    int64_t ldw, lda;
    int64_t M, N, K;
    float *C;
    int64_t ldc;
    const float *bias;
    int act;
    int tiles_m;
    int cluster;
    int kb_total;
    int fine_chains;      // chains end between k-steps of 8, not blocks (see cn_gemm_small_launch)
    unsigned int *status;
    int npeers;
    float *peerC[CN_MAX_PEERS];
    const unsigned int *ready;
    unsigned int *const *peer_flags;
    int nranks, my_rank;
    unsigned int epoch;
};

// fp32 -> TF32, round to nearest with ties away from zero: add half a TF32 ulp to the magnitude bits and truncate.  That carry takes
// the finite values from 0x7f7ff000 up to infinity and a NaN with a full mantissa (0x7fffffff, the one GPU arithmetic makes)
// over into the sign bit, to -0.  CAREFUL truncates those instead, NaNs after an addition that makes them the canonical one.
template <bool CAREFUL>
__device__ __forceinline__ uint32_t sm_tf32(float x)
{
    if (!CAREFUL) return (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    const float top = __uint_as_float(0x7f7ff000u);
    return (fabsf(x) < top ? __float_as_uint(x) + 0x1000u : __float_as_uint(__fadd_rn(x, 0.0f))) & 0xffffe000u;
}

__device__ __forceinline__ void sts4u(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// D[tmem] (+)= A[smem] * B[smem], both K-major TF32 tiles.
__device__ __forceinline__ void sm_mma_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 ad, bd;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 ad, {%1, %3};\n\t"
        "mov.b64 bd, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], ad, bd, %4, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate) : "memory");
}

// One 128 x 32 block of an operand, spread over 128 threads: 32 values per thread.
// `rows`: rows of the tile that exist; everything else reads as zero.
template <int KIND>
__device__ __forceinline__ void sm_load(const float *base, int64_t ld, int rows, int64_t k0, int64_t K, int t, float (&x)[32])
{
    if (KIND == SM_K_VEC) {   // eight lanes per row (128 bytes), sixteen rows per pass
        const int c = t & 7;
        const int64_t k = k0 + 4 * c;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = i * 16 + (t >> 3);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < rows) {
                const float *p = base + (int64_t)r * ld + k;
                if (k + 3 < K) {
                    v = *reinterpret_cast<const float4 *>(p);
                } else {
                    if (k < K) v.x = p[0];
                    if (k + 1 < K) v.y = p[1];
                    if (k + 2 < K) v.z = p[2];
                }
            }
            x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
        }
    } else if (KIND == SM_K_SCALAR) {   // one row (128 bytes) per warp and pass
        const int64_t k = k0 + (t & 31);
        const float *p = base + (int64_t)(t >> 5) * ld + k;
        const bool in_k = k < K;
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = (in_k && i * 4 + (t >> 5) < rows) ? p[(int64_t)(i * 4) * ld] : 0.0f;
    } else {   // one row per thread, consecutive threads on consecutive rows
        const float *p = base + t + k0 * ld;
        const bool in_r = t < rows;
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = (in_r && k0 + i < K) ? p[(int64_t)i * ld] : 0.0f;
    }
}

// Whether sm_tf32 has to be CAREFUL with some of the values.
__device__ __forceinline__ bool sm_unsafe(const float (&x)[32])
{
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; i += 2) asm("max.NaN.abs.f32 %0, %1, %2, %0;" : "+f"(m) : "f"(x[i]), "f"(x[i + 1]));
    return !(m < __uint_as_float(0x7f7ff000u));
}

// The same block -> TF32 parts in shared memory: 16-byte chunk c of row r lies at r * 128 + ((c ^ (r & 7)) << 4).
template <int KIND, bool MODE3X, bool CAREFUL>
__device__ __forceinline__ void sm_store(uint32_t hi, uint32_t lo, int need_rows, int t, const float (&x)[32])
{
    if (KIND == SM_K_SCALAR) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const int r = i * 4 + (t >> 5), kk = t & 31;
            if (r >= need_rows) continue;
            const uint32_t at = (uint32_t)(r * 128 + (((kk >> 2) ^ (r & 7)) << 4) + (kk & 3) * 4);
            const uint32_t h = sm_tf32<CAREFUL>(x[i]);
            sts1u(hi + at, h);
            if (MODE3X) sts1u(lo + at, sm_tf32<CAREFUL>(x[i] - __uint_as_float(h)));
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = KIND == SM_K_VEC ? i * 16 + (t >> 3) : t, c = KIND == SM_K_VEC ? (t & 7) : i;
            if (r >= need_rows) continue;
            const uint32_t at = (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4));
            uint32_t h[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) h[e] = sm_tf32<CAREFUL>(x[4 * i + e]);
            sts4u(hi + at, h[0], h[1], h[2], h[3]);
            if (MODE3X)
                sts4u(lo + at, sm_tf32<CAREFUL>(x[4 * i] - __uint_as_float(h[0])), sm_tf32<CAREFUL>(x[4 * i + 1] - __uint_as_float(h[1])),
                      sm_tf32<CAREFUL>(x[4 * i + 2] - __uint_as_float(h[2])), sm_tf32<CAREFUL>(x[4 * i + 3] - __uint_as_float(h[3])));
        }
    }
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// The loading side of one operand: blocks kb0 .. kb1 - 1 of its tile into the ring.
template <int KIND, bool MODE3X>
__device__ __forceinline__ bool sm_feed(const float *base, int64_t ld, int rows, int need_rows, int64_t K, int kb0, int kb1, int t, uint32_t ring,
                                        uint32_t operand_off, uint32_t full0, uint32_t empty0, uint32_t abort_flag, unsigned int *status)
{
    float x[2][32];
    const int n = kb1 - kb0;
    bool ok = true;
    sm_load<KIND>(base, ld, rows, (int64_t)kb0 * SM_BK, K, t, x[0]);
    for (int i0 = 0; i0 < n && ok; i0 += 2) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = i0 + u;
            if (i >= n || !ok) continue;
            if (i + 1 < n) sm_load<KIND>(base, ld, rows, (int64_t)(kb0 + i + 1) * SM_BK, K, t, x[u ^ 1]);
            const bool unsafe = sm_unsafe(x[u]);
            ok = mbar_wait(empty0 + 8 * u, ((uint32_t)(i >> 1) & 1u) ^ 1u, abort_flag, status, 14u);
            if (!ok) continue;
            const uint32_t hi = ring + u * SM_STAGE_BYTES + operand_off;
            if (unsafe) sm_store<KIND, MODE3X, true>(hi, hi + SM_TILE_BYTES, need_rows, t, x[u]);
            else        sm_store<KIND, MODE3X, false>(hi, hi + SM_TILE_BYTES, need_rows, t, x[u]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if ((t & 31) == 0) mbar_arrive(full0 + 8 * u);
        }
    }
    return ok;
}

template <int WKIND, int AKIND, bool MODE3X>
__global__ void __launch_bounds__(SM_THREADS, 1)
cn_gemm_small_kernel(const __grid_constant__ SmallParams p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * SM_STAGES + 1];
    __shared__ uint32_t s_words[2];   // tensor-memory base, abort flag
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[SM_STAGES]), acc_bar = smem_u32(&bars[2 * SM_STAGES]);
    const uint32_t abort_flag = smem_u32(&s_words[1]);
    const uint32_t turn = p.cluster > 1 ? ring + SM_RING_BYTES : ring;   // partial-tile slices; with one CTA per tile the idle ring serves
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x % p.cluster, tile = blockIdx.x / p.cluster;
    const int64_t m0 = (int64_t)(tile % p.tiles_m) * SM_BM, n0 = (int64_t)(tile / p.tiles_m) * SM_BN;
    const int m_rows = (int)(p.M - m0 < SM_BM ? p.M - m0 : SM_BM), n_rows = (int)(p.N - n0 < SM_BN ? p.N - n0 : SM_BN);
    const int m_need = (m_rows + 15) & ~15;   // UMMA N
    const int kb0 = (int)((int64_t)p.kb_total * rank / p.cluster), kb1 = (int)((int64_t)p.kb_total * (rank + 1) / p.cluster);
    // accumulation chains, in k-steps of 8
    const int steps = (kb1 - kb0) * (SM_BK / 8);
    const int chain_steps = p.fine_chains ? (steps + SM_MAX_CHAINS - 1) / SM_MAX_CHAINS : (kb1 - kb0 + SM_MAX_CHAINS - 1) / SM_MAX_CHAINS * (SM_BK / 8);
    const int chains = (steps + chain_steps - 1) / chain_steps;
    cn_pdl_launch_dependents();
    if (p.cluster > 1) cluster_arrive();   // every CTA of the cluster has started: waited for before the first remote store
    if (threadIdx.x == 0) {
        for (int s = 0; s < SM_STAGES; ++s) { mbar_init(full0 + 8 * s, 8); mbar_init(empty0 + 8 * s, 1); }
        mbar_init(acc_bar, 1);
        s_words[1] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t cols = chains == 1 ? 128u : chains == 2 ? 256u : 512u;
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_words[0])), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_words[0];
    cn_pdl_wait();
    if (p.npeers > 0 && blockIdx.x == 0 && threadIdx.x < p.nranks && (int)threadIdx.x != p.my_rank) {
        // fused all-gather: this rank's copy of C may be overwritten by its peers (slot 0 of their flag block)
        __threadfence_system();
        volatile unsigned int *f = p.peer_flags[threadIdx.x] + p.my_rank;
        *f = p.epoch;
    }
    bool ok = true;
    if (warp < 4) {
        const float *base = WKIND == SM_ROWS ? p.W + n0 : p.W + n0 * p.ldw;
        ok = sm_feed<WKIND, MODE3X>(base, p.ldw, n_rows, SM_BN, p.K, kb0, kb1, threadIdx.x, ring, 0, full0, empty0, abort_flag, p.status);
    } else if (warp < 8) {
        const float *base = AKIND == SM_ROWS ? p.A + m0 : p.A + m0 * p.lda;
        ok = sm_feed<AKIND, MODE3X>(base, p.lda, m_rows, m_need, p.K, kb0, kb1, threadIdx.x - 128, ring, 2 * SM_TILE_BYTES, full0, empty0, abort_flag,
                                    p.status);
    } else if (lane == 0) {
        // kind::tf32 instruction descriptor: D fp32, A and B TF32 (format 2), K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28
        const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(m_need >> 3) << 17) | ((uint32_t)(SM_BN >> 4) << 24);
        const int n = kb1 - kb0;
        uint32_t acc = tmem;
        int in_chain = 0;
        for (int i = 0; i < n; ++i) {
            const int s = i & 1;
            ok = mbar_wait(full0 + 8 * s, (uint32_t)(i >> 1) & 1u, abort_flag, p.status, 15u);
            if (!ok) break;
            tc_fence_after();
            const uint64_t d = make_kmajor_sw128_desc(ring + s * SM_STAGE_BYTES);
            const uint32_t hi = (uint32_t)(d >> 32), whi = (uint32_t)d, wlo = whi + (SM_TILE_BYTES >> 4), ahi = wlo + (SM_TILE_BYTES >> 4),
                           alo = ahi + (SM_TILE_BYTES >> 4);
#pragma unroll
            for (int j = 0; j < SM_BK / 8; ++j) {   // 8 TF32 per k-step: 32 bytes (descriptor units of 16 B)
                if (in_chain == chain_steps) { in_chain = 0; acc += SM_BM; }
                sm_mma_ss(acc, whi + 2 * j, ahi + 2 * j, hi, idesc, in_chain++ != 0 ? 1u : 0u);
                if (MODE3X) {
                    sm_mma_ss(acc, wlo + 2 * j, ahi + 2 * j, hi, idesc, 1u);
                    sm_mma_ss(acc, whi + 2 * j, alo + 2 * j, hi, idesc, 1u);
                }
            }
            tc_commit(empty0 + 8 * s);
        }
        if (ok) tc_commit(acc_bar);
    }
    __syncwarp();
    const int R = SM_BN / p.cluster;   // columns n this CTA finishes
    if (warp < 8) {
        ok = ok && mbar_wait(acc_bar, 0u, abort_flag, p.status, 16u);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
    }
    if (p.cluster > 1) cluster_wait();
    else __syncthreads();              // the ring is about to be overwritten: every warp has seen the last MMA retire
    if (warp < 8 && ok) {
        // warps w and w + 4 share a lane quarter and take 64 rows m each
        const int n_l = (warp & 3) * 32 + lane, col0 = (warp >> 2) * 64;
        const int dst = n_l / R, i = n_l - dst * R;
        uint32_t slice = turn + (uint32_t)((rank * R + i) * SM_BM) * 4;
        if (p.cluster > 1) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(slice) : "r"(slice), "r"(dst));
        const uint32_t src = tmem + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
            const int col = col0 + cc * 16;
            if (col >= m_need) break;
            uint32_t r[16];
            tc_ld16(src + col, r);
            for (int ch = 1; ch < chains; ++ch) {
                uint32_t q[16];
                tc_ld16(src + ch * SM_BM + col, q);
#pragma unroll
                for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) + __uint_as_float(q[e]));
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {   // 16-byte chunk col/4 + c of the row, chunks permuted by the row against bank conflicts
                const uint32_t at = slice + ((uint32_t)((col / 4 + c) ^ (i & 7)) << 4);
                if (p.cluster > 1)
                    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(r[4 * c]), "r"(r[4 * c + 1]), "r"(r[4 * c + 2]), "r"(r[4 * c + 3]) : "memory");
                else
                    sts4u(at, r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
            }
        }
    }
    tc_fence_before();
    if (p.cluster > 1) { cluster_arrive(); cluster_wait(); }
    else __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
        return;
    }
    if (p.npeers > 0) {   // peers must have announced that their copy of C may be overwritten (bounded wait)
        if (threadIdx.x == 0) {
            const long long t0 = clock64();
            for (int r = 0; r < p.nranks; ++r) {
                if (r == p.my_rank) continue;
                const volatile unsigned int *f = p.ready + r;
                while ((int)(*f - p.epoch) < 0) {
                    if (clock64() - t0 > TC_WAIT_LIMIT) { atomicMax(p.status, 9u); break; }
                    __nanosleep(100);
                }
            }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    // this CTA's slice: column n0 + rank * R + i, four rows m per lane
    const int64_t m = m0 + lane * 4;
    const bool vec = (m + 4 <= p.M) && ((p.ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15u) == 0);
    for (int i = warp; i < R; i += 8) {
        const int64_t n = n0 + rank * R + i;
        if (n >= p.N || m >= p.M) continue;
        const uint32_t at = turn + (uint32_t)(i * SM_BM) * 4 + ((uint32_t)(lane ^ (i & 7)) << 4);
        float4 a = lds4(at);
        for (int s = 1; s < p.cluster; ++s) {
            const float4 b = lds4(at + (uint32_t)(s * R * SM_BM) * 4);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
        }
        const float b = p.bias ? p.bias[n] : 0.0f;
        float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = cn_apply_activation(p.bias ? v[e] + b : v[e], p.act);
        const int64_t off = n * p.ldc + m;
        for (int d = 0; d <= p.npeers; ++d) {
            float *q = (d == 0 ? p.C : p.peerC[d - 1]) + off;
            if (vec) {
                *reinterpret_cast<float4 *>(q) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (m + e < p.M) q[e] = v[e];
            }
        }
    }
}

// CTAs per tile: a power of two, as many as there are SMs for, each with at least two K blocks.
static int small_cluster(int64_t tiles, int kb, int sms)
{
    int c = 1;
    while (c < SM_MAX_CLUSTER && tiles * c * 2 <= sms && kb >= c * 4) c *= 2;
    return c;
}

bool cn_gemm_small_shape(const cn_context *ctx, int64_t M, int64_t N, int64_t K, bool w_aligned, int max_rounds)
{
    if (M < 1 || N < 1 || K < 1) return false;
    if (N > (1 << 21) / K) return false;   // at most 8 MB of weights
    const int64_t tiles = ((M + SM_BM - 1) / SM_BM) * ((N + SM_BN - 1) / SM_BN);
    const int kb = (int)((K + SM_BK - 1) / SM_BK);
    const int c = small_cluster(tiles, kb, ctx->sm_count);
    const int64_t per_cta = (kb + c - 1) / c, rounds = (tiles * c + ctx->sm_count - 1) / ctx->sm_count;
    // more than two rounds of CTAs cost more than the streaming kernel's three launches: the 4096 x 4096 weight gradient of a batch of
    // 128 (1024 tiles, seven rounds) took 108 us here; the whole backward pass went from 210 to 162 us
    // a block costs a CTA 1.5 us, the streaming kernel's launches and reduction 15 to 20: 16 x 8000 . 8000 x 64 (32 blocks) took 43 us here
    if (per_cta > (w_aligned ? SM_MAX_BLOCKS : SM_MAX_BLOCKS_ANY) || rounds > max_rounds) return false;
    // weights that TMA cannot read must not become less exact than on the fp32 kernel (cn_gemm_any_chain); a TF32 block has twice the
    // additions of an fp16 one
    const int chain = cn_gemm_any_chain(K) / 2;
    return w_aligned || (per_cta + SM_MAX_CHAINS - 1) / SM_MAX_CHAINS <= (chain > 1 ? chain : 1);
}

template <int WKIND, int AKIND, bool MODE3X>
static int small_launch(cn_context *ctx, const SmallParams &p, int64_t ctas, cudaStream_t s)
{
    static bool attr_set[64] = {};
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        CN_CUDA(cudaFuncSetAttribute(cn_gemm_small_kernel<WKIND, AKIND, MODE3X>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_SMEM_BYTES(2)));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(SM_THREADS);
    cfg.dynamicSmemBytes = SM_SMEM_BYTES(p.cluster);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.cluster > 1 ? 2 : 1;
    CN_CUDA(cudaLaunchKernelEx(&cfg, cn_gemm_small_kernel<WKIND, AKIND, MODE3X>, p));
    cn_count_launch();
    return CN_OK;
}

template <bool MODE3X>
static int small_pick(cn_context *ctx, const SmallParams &p, int wk, int ak, int64_t ctas, cudaStream_t s)
{
#define CN_SMALL(W) \
    return ak == SM_K_VEC ? small_launch<W, SM_K_VEC, MODE3X>(ctx, p, ctas, s) : ak == SM_K_SCALAR ? small_launch<W, SM_K_SCALAR, MODE3X>(ctx, p, ctas, s) \
                                                                                                    : small_launch<W, SM_ROWS, MODE3X>(ctx, p, ctas, s)
    if (wk == SM_K_VEC) CN_SMALL(SM_K_VEC);
    if (wk == SM_K_SCALAR) CN_SMALL(SM_K_SCALAR);
    CN_SMALL(SM_ROWS);
#undef CN_SMALL
}

int cn_gemm_small_launch(cn_context *ctx, int transA, int transB, int64_t M, int64_t N, int64_t K, const float *A, int64_t lda, const float *B, int64_t ldb,
                         float *C, int64_t ldc, const cn_epilogue *epi, int mode, cudaStream_t s, const cn_peer_out *peers, bool w_aligned)
{
    SmallParams p;
    unsigned int *d_status = nullptr;
    int st = cn_status_block(ctx, &d_status);
    if (st != CN_OK) return st;
    p.W = B; p.A = A; p.ldw = ldb; p.lda = lda;
    p.M = M; p.N = N; p.K = K;
    p.C = C; p.ldc = ldc;
    p.bias = epi ? epi->bias : nullptr;
    p.act = epi ? epi->activation : CN_ACT_LINEAR;
    p.tiles_m = (int)((M + SM_BM - 1) / SM_BM);
    const int64_t tiles = (int64_t)p.tiles_m * ((N + SM_BN - 1) / SM_BN);
    p.kb_total = (int)((K + SM_BK - 1) / SM_BK);
    p.cluster = small_cluster(tiles, p.kb_total, ctx->sm_count);
    p.fine_chains = !w_aligned;
    p.status = d_status;
    p.npeers = 0;
    p.ready = nullptr; p.peer_flags = nullptr;
    p.nranks = 0; p.my_rank = 0; p.epoch = 0;
    for (int i = 0; i < CN_MAX_PEERS; ++i) p.peerC[i] = nullptr;
    if (peers && peers->npeers > 0) {
        p.npeers = peers->npeers;
        for (int i = 0; i < peers->npeers; ++i) p.peerC[i] = peers->C[i];
        p.ready = peers->ready; p.peer_flags = peers->peer_flags;
        p.nranks = peers->nranks; p.my_rank = peers->my_rank; p.epoch = peers->epoch;
    }
    auto kind = [](bool k_contiguous, int64_t ld, const float *q) {
        return !k_contiguous ? SM_ROWS : ((ld & 3) == 0 && ((uintptr_t)q & 15u) == 0) ? SM_K_VEC : SM_K_SCALAR;
    };
    const int wk = kind(!transB, ldb, B), ak = kind(transA != 0, lda, A);
    st = mode == CN_GEMM_3XTF32 ? small_pick<true>(ctx, p, wk, ak, tiles * p.cluster, s) : small_pick<false>(ctx, p, wk, ak, tiles * p.cluster, s);
    if (st == CN_OK) ctx->gemm_last_path = mode == CN_GEMM_3XTF32 ? "tcgen05_3xtf32" : "tcgen05_tf32";
    return st;
}
