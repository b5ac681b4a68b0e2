// Small products for sm_100a: one launch, both operands split in the kernel, K split over a thread-block cluster.
//
// The streaming kernel (cn_gemm_tc.cu) takes three launches - planes of the activations, product, reduction - which is the
// right price for weights that have to come from HBM.  A layer of a small network (128 x 784 . 784 x 1024, the weight gradients
// and back-propagated errors of a 784-1200-1200-10 network) is over in a few microseconds; there the launches, the passes
// over memory between them and the idle SMs of a product with eight tiles are the cost.  Here
//   * a CTA takes a tile of 128 rows m by NT = 32, 64 or 128 columns n and a share of K.  Eight warps each load and split blocks of 32 k of
//     the activations and the weights, straight from global memory in whatever layout they have (either operand transposed or not, any
//     alignment), three blocks of loads in flight;
//   * the operands are TF32 hi / lo parts in shared memory (K-major, 128-byte swizzle), three tcgen05.mma kind::tf32 products per
//     k-step as CN_GEMM_3XTF32 promises, one for CN_GEMM_TF32; one thread issues them;
//   * the accumulator tile has the rows m in tensor memory's lanes, so that a warp holds 32 consecutive rows of a column: it sends
//     and stores whole lines of 128 bytes without turning anything;
//   * the CTAs of a cluster (up to eight, any number) share a tile: each multiplies its part of K, sends every other CTA its columns of the
//     partial tile through distributed shared memory, adds the parts it received in K order (reproducible), and finishes its columns:
//     bias, activation, stores to C and, for the fused all-gather, to the peers.
// The tensor core's accumulator truncates, so a share of K is cut into as many chains as tensor memory holds accumulators for, and the
// chains are added in round-to-nearest fp32.  The products with a low part have accumulators of their own, which costs no instruction (one
// MMA multiplies the activations' high parts with both parts of the weights, whose rows lie behind one another): an addition
// truncates what it adds to a large sum.
//
// Bound by latency and, per block of K, by shared memory: the feeding warps write, and the MMAs read, 64 to 144 KB of it, 0.6 us at 128
// bytes per clock for tiles of 128 columns.  In a series, with tiles of 128 columns n in the lanes, partial tiles of 64 KB through the cluster
// and output by way of shared memory before: 128 x 784 . 784 x 1024 14.3 -> 10.9 us, 128 x 1200 . 1200 x 10 13.5 -> 7.4, weight gradient
// 1200 x 128 . 128 x 1200 16.3 -> 9.0.
//
// The exchange.  Distributed shared memory takes about 20 bytes per clock from a CTA.  Sent as single floats between two barriers of the
// cluster, and added and stored a float at a time, a tile of 128 columns took 11 300 of the kernel's 19 000 clocks (by clock64 in a copy of it:
// 3500 until a CTA had sent, 4100 until all had, 3700 to finish).  Now a lane sends four columns of its row at once, st.async counts the
// bytes at the receiver's mbarrier (no release has to wait for every store's acknowledgement), a CTA's own share stays where it is, and the
// sums of four columns are one pass over the senders with a single copy of the activation's code, which a launch has to fetch once: 128 x
// 784 . 784 x 1024 11.1 -> 9.3 us, 128 x 1200 . 1200 x 1200 12.6 -> 10.5, 1200 x 10 8.2 -> 7.1.  Setting the CTA up before the predecessor has
// ended, and clusters of 3, 5, 6 and 7 where more of them fit, are in these figures.
#include <limits.h>
#include "cn_epilogue.cuh"
#include "cn_gemm.h"
#include "cn_tc_feed.cuh"

#define SM_FEED 256             // threads that load and split an operand: warps 0-7 the activations, 8-15 the weights; all of them the epilogue
#define SM_EPI (2 * SM_FEED)
#define SM_THREADS (SM_EPI + 32)   // warp 16: MMA issuer
#define SM_STAGES 2
#define SM_AHEAD 3              // blocks of loads in flight
#define SM_A_TILE (SM_BM * 128)
#define SM_MAX_BLOCKS 12
#define SM_MAX_BLOCKS_ANY 16   // weights that TMA cannot read, of which the streaming kernel wants four rows at least
#define SM_MAX_CLUSTER 8

template <int NT, bool MODE3X>
struct SmCfg {
    static constexpr int W_TILE = NT * 128;
    static constexpr int STAGE_BYTES = 2 * (SM_A_TILE + W_TILE);   // A hi, A lo, W hi, W lo
    static constexpr int RING_BYTES = SM_STAGES * STAGE_BYTES;
    // what the cluster's CTAs send: [sender][four columns][128 m] float4
    static constexpr int part_bytes(int cluster) { return cluster > 1 ? cluster * ((NT / 4 + cluster - 1) / cluster) * SM_BM * 16 : 0; }
    // An accumulator has NT columns for the products of the high parts and, in the 3x mode, NT for those with a low part
    static constexpr int ACC_COLS = MODE3X ? 2 * NT : NT;
    static constexpr int MAX_CHAINS = 512 / ACC_COLS < 8 ? 512 / ACC_COLS : 8;
    static constexpr int smem(int cluster) { return 1024 + RING_BYTES + part_bytes(cluster); }
    static constexpr int SMEM_MAX = 1024 + RING_BYTES + (NT / 4 + SM_MAX_CLUSTER - 1) * SM_BM * 16;
    static_assert(SMEM_MAX <= 232448 - 1024, "shared memory");
};

// An operand: element (row, k) at p[row * sr + k * sk].
struct SmOperand {
    const float *p;
    int64_t sr, sk;
    int vec;                // 16-byte aligned along the contiguous one of the two
};
static inline SmOperand sm_operand(const float *p, bool k_contiguous, int64_t ld)
{
    SmOperand o;
    o.p = p;
    o.sr = k_contiguous ? ld : 1;
    o.sk = k_contiguous ? 1 : ld;
    o.vec = (ld & 3) == 0 && ((uintptr_t)p & 15u) == 0;
    return o;
}

struct SmallParams {
    SmOperand A, W;
    int64_t M, N, K;
    float *C;
    int64_t ldc;
    const float *bias;
    int act;
    int tiles_m;
    int cluster;
    int per, per_inv;       // of a tile's columns, in fours, those that a CTA of the cluster finishes; 65536 / per, rounded up
    int kb_total;
    unsigned int *status;
    int npeers;
    float *peerC[CN_MAX_PEERS];
    const unsigned int *ready;
    unsigned int *const *peer_flags;
    int nranks, my_rank;
    unsigned int epoch;
};

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

// The share of one thread of a block of ROWS x 32 k: up to four 16-byte chunks (a chunk is four consecutive k of a row).
// QUADS false: chunks of rows 32 apart; with k contiguous, eight lanes read a row's 128 bytes, 16 at a time where the rows are aligned;
// else (rows contiguous but not aligned) a chunk's four elements are read one by one.
// QUADS true (rows contiguous and aligned): four rows by four k, read 16 bytes at a time along the rows and turned in registers.
// Lanes: two quads of rows, eight chunks, two quads again, so that eight lanes that store together meet in no bank.
template <int ROWS, bool QUADS>
struct SmShare {
    static constexpr int CHUNKS = QUADS ? 4 : ROWS * 8 / SM_FEED;
    const float *src;       // the first element of chunk 0 (QUADS: of row 4 q)
    int64_t sr, sk;
    int row0, c0, rows;
    bool vec;
    // t: 0 .. SM_FEED - 1
    __device__ __forceinline__ SmShare(const SmOperand &o, int64_t first_row, int rows_here, int t)
    {
        vec = o.vec;
        rows = rows_here;
        sr = o.sr;
        sk = o.sk;
        if (QUADS) {
            row0 = 4 * ((t & 1) | (t >> 3 & 2) | (t >> 5 << 2));
            c0 = t >> 1 & 7;
        } else if (o.sk == 1) {
            row0 = t >> 3;
            c0 = t & 7;
        } else {   // a warp reads 32 rows
            row0 = t & 31;
            c0 = t >> 5;
        }
        src = o.p + (first_row + row0) * o.sr + 4 * c0 * o.sk;
    }
    __device__ __forceinline__ bool mine() const { return !QUADS || row0 < ROWS; }
    __device__ __forceinline__ void load(int64_t k0, int64_t K, float4 (&x)[CHUNKS]) const
    {
        const float *q = src + k0 * sk;
        const int left = (int)(K - k0 < SM_BK ? K - k0 : SM_BK) - 4 * c0;   // k of this chunk that exist
#pragma unroll
        for (int i = 0; i < CHUNKS; ++i) x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (QUADS) {
            if (left >= 4 && row0 + 3 < rows) {
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = *reinterpret_cast<const float4 *>(q + e * sk);
            } else if (mine()) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (e >= left) continue;
                    if (row0 < rows) x[e].x = q[e * sk];
                    if (row0 + 1 < rows) x[e].y = q[e * sk + 1];
                    if (row0 + 2 < rows) x[e].z = q[e * sk + 2];
                    if (row0 + 3 < rows) x[e].w = q[e * sk + 3];
                }
            }
        } else if (vec && left >= 4 && sk == 1) {
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i)
                if (row0 + 32 * i < rows) x[i] = *reinterpret_cast<const float4 *>(q + 32 * i * sr);
        } else {
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i) {
                if (row0 + 32 * i >= rows) continue;
                if (left > 0) x[i].x = q[32 * i * sr];
                if (left > 1) x[i].y = q[32 * i * sr + sk];
                if (left > 2) x[i].z = q[32 * i * sr + 2 * sk];
                if (left > 3) x[i].w = q[32 * i * sr + 3 * sk];
            }
        }
    }
    // TF32 parts into shared memory: 16-byte chunk c of row r lies at r * 128 + ((c ^ (r & 7)) << 4).
    template <bool MODE3X, bool CAREFUL>
    __device__ __forceinline__ void put(uint32_t hi, uint32_t lo, const float4 (&x)[CHUNKS]) const
    {
#pragma unroll
        for (int i = 0; i < CHUNKS; ++i) {
            const int r = row0 + (QUADS ? i : 32 * i);
            const uint32_t at = (uint32_t)(r * 128 + ((c0 ^ (r & 7)) << 4));
            auto of = [](const float4 &v, int e) { return e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w; };
            float y[4];
            uint32_t h[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                y[e] = QUADS ? of(x[QUADS ? e : 0], i) : of(x[i], e);
                h[e] = sm_tf32<CAREFUL>(y[e]);
            }
            sts4u(hi + at, h[0], h[1], h[2], h[3]);
            if (MODE3X)
                sts4u(lo + at, sm_tf32<CAREFUL>(y[0] - __uint_as_float(h[0])), sm_tf32<CAREFUL>(y[1] - __uint_as_float(h[1])),
                      sm_tf32<CAREFUL>(y[2] - __uint_as_float(h[2])), sm_tf32<CAREFUL>(y[3] - __uint_as_float(h[3])));
        }
    }
    template <bool MODE3X>
    __device__ __forceinline__ void store(uint32_t hi, uint32_t lo, const float4 (&x)[CHUNKS]) const
    {
        if (!mine()) return;
        float m = 0.0f;   // whether sm_tf32 has to be careful with some of the values
#pragma unroll
        for (int i = 0; i < CHUNKS; ++i) {
            asm("max.NaN.abs.f32 %0, %1, %2, %0;" : "+f"(m) : "f"(x[i].x), "f"(x[i].y));
            asm("max.NaN.abs.f32 %0, %1, %2, %0;" : "+f"(m) : "f"(x[i].z), "f"(x[i].w));
        }
        if (m < __uint_as_float(0x7f7ff000u)) put<MODE3X, false>(hi, lo, x);
        else put<MODE3X, true>(hi, lo, x);
    }
};

// Blocks kb0 .. kb0 + n - 1 of one operand's tile into the ring.  begin() issues the first loads, run() does the rest.
template <class Share, bool MODE3X>
struct SmFeed {
    const Share share;
    float4 x[SM_AHEAD][Share::CHUNKS];
    __device__ __forceinline__ SmFeed(const SmOperand &o, int64_t first_row, int rows, int t) : share(o, first_row, rows, t) {}
    __device__ __forceinline__ void begin(int kb0, int n, int64_t K)
    {
#pragma unroll
        for (int u = 0; u < SM_AHEAD; ++u)
            if (u < n) share.load((int64_t)(kb0 + u) * SM_BK, K, x[u]);
    }
    __device__ __forceinline__ bool run(int kb0, int n, int64_t K, uint32_t ring, int stage_bytes, uint32_t hi_off, uint32_t lo_off, uint32_t full0, uint32_t empty0,
                                        uint32_t abort_flag, unsigned int *status)
    {
        bool ok = true;
        for (int i0 = 0; i0 < n && ok; i0 += SM_AHEAD) {
#pragma unroll
            for (int u = 0; u < SM_AHEAD; ++u) {
                const int i = i0 + u, s = i & 1;
                if (i >= n || !ok) continue;
                ok = mbar_wait_warp(empty0 + 8 * s, ((uint32_t)(i >> 1) & 1u) ^ 1u, abort_flag, status, 14u);
                if (!ok) continue;
                const uint32_t stage = ring + s * stage_bytes;
                share.template store<MODE3X>(stage + hi_off, stage + lo_off, x[u]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if ((threadIdx.x & 31) == 0) mbar_arrive(full0 + 8 * s);
                if (i + SM_AHEAD < n) share.load((int64_t)(kb0 + i + SM_AHEAD) * SM_BK, K, x[u]);
            }
        }
        return ok;
    }
};

// Columns of the accumulators of all chains, in K order, the products with a low part last.
template <int NT, bool MODE3X, int COLS>
__device__ __forceinline__ void sm_sum(uint32_t taddr, int chains, float (&v)[COLS])
{
    using Cfg = SmCfg<NT, MODE3X>;
    constexpr int PARTS = MODE3X ? 2 : 1, GROUP = COLS == 8 ? 4 : 1;   // accumulators that are loaded before the wait
    float low[COLS];
#pragma unroll
    for (int c = 0; c < COLS; ++c) v[c] = low[c] = 0.0f;
#pragma unroll 1
    for (int ch0 = 0; ch0 < chains; ch0 += GROUP) {
        uint32_t r[GROUP][PARTS][COLS];
#pragma unroll
        for (int ch = 0; ch < GROUP; ++ch) {
            if (ch0 + ch >= chains) break;
#pragma unroll
            for (int part = 0; part < PARTS; ++part) tc_ld_ahead(taddr + (ch0 + ch) * Cfg::ACC_COLS + part * NT, r[ch][part]);
        }
        tc_wait_ld();
#pragma unroll
        for (int ch = 0; ch < GROUP; ++ch) {
            if (ch0 + ch >= chains) break;
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
#pragma unroll
                for (int part = 0; part < PARTS; ++part) asm volatile("" : "+r"(r[ch][part][c]));   // no use moves before the wait
                v[c] += __uint_as_float(r[ch][0][c]);
                if (MODE3X) low[c] += __uint_as_float(r[ch][PARTS - 1][c]);
            }
        }
    }
    if (MODE3X) {
#pragma unroll
        for (int c = 0; c < COLS; ++c) v[c] += low[c];
    }
}

// Peers must have announced that their copy of C may be overwritten (bounded wait).
__device__ __forceinline__ void sm_wait_peers(const SmallParams &p)
{
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

template <int NT, bool MODE3X, bool A_QUADS, bool W_QUADS>
__global__ void __launch_bounds__(SM_THREADS, 1)
cn_gemm_small_kernel(const __grid_constant__ SmallParams p)
{
    using Cfg = SmCfg<NT, MODE3X>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * SM_STAGES + 2];
    __shared__ uint32_t s_words[2];   // tensor-memory base, abort flag
    __shared__ float s_bias[NT];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u, part = ring + Cfg::RING_BYTES;
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[SM_STAGES]), acc_bar = smem_u32(&bars[2 * SM_STAGES]);
    const uint32_t part_bar = acc_bar + 8;   // this CTA's columns of all partial tiles have arrived
    const uint32_t abort_flag = smem_u32(&s_words[1]);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x % p.cluster, tile = blockIdx.x / p.cluster;
    const int64_t m0 = (int64_t)(tile % p.tiles_m) * SM_BM, n0 = (int64_t)(tile / p.tiles_m) * NT;
    const int m_rows = (int)(p.M - m0 < SM_BM ? p.M - m0 : SM_BM), n_rows = (int)(p.N - n0 < NT ? p.N - n0 : NT);
    const int kb0 = p.kb_total * rank / p.cluster, n_blocks = p.kb_total * (rank + 1) / p.cluster - kb0;
    const int per_chain = (n_blocks + Cfg::MAX_CHAINS - 1) / Cfg::MAX_CHAINS, chains = (n_blocks + per_chain - 1) / per_chain;
    // the columns of the tile in fours: this CTA finishes `per` of them, from `mine` on; those from `fours` on do not exist
    const int per = p.per, mine = rank * per, fours = (n_rows + 3) >> 2, n_mine = fours - mine < per ? fours - mine : per;
    cn_pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < SM_STAGES; ++s) { mbar_init(full0 + 8 * s, SM_EPI / 32); mbar_init(empty0 + 8 * s, 1); }
        mbar_init(acc_bar, 1);
        mbar_init(part_bar, 1);
        if (n_mine > 0) mbar_expect_tx(part_bar, (uint32_t)((p.cluster - 1) * n_mine * SM_BM * 16));
        s_words[1] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (p.cluster > 1) cluster_arrive();   // every CTA of the cluster has started and its barriers are there: waited for before the first remote store
    uint32_t cols = 32;
    while (cols < (uint32_t)(chains * Cfg::ACC_COLS)) cols <<= 1;
    if (warp == 16) {
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
    if (warp < 8) {
        SmFeed<SmShare<SM_BM, A_QUADS>, MODE3X> feed(p.A, m0, m_rows, threadIdx.x);
        feed.begin(kb0, n_blocks, p.K);
        if ((int)threadIdx.x < n_rows && p.bias) s_bias[threadIdx.x] = p.bias[n0 + threadIdx.x];
        ok = feed.run(kb0, n_blocks, p.K, ring, Cfg::STAGE_BYTES, 0, SM_A_TILE, full0, empty0, abort_flag, p.status);
    } else if (warp < 16) {
        SmFeed<SmShare<NT, W_QUADS>, MODE3X> feed(p.W, n0, n_rows, threadIdx.x - SM_FEED);
        feed.begin(kb0, n_blocks, p.K);
        ok = feed.run(kb0, n_blocks, p.K, ring, Cfg::STAGE_BYTES, 2 * SM_A_TILE, 2 * SM_A_TILE + Cfg::W_TILE, full0, empty0, abort_flag, p.status);
    }
    if (warp == 16) {   // the whole warp waits, which takes half as long as by one lane; one issues
        // kind::tf32 instruction descriptor: D fp32, A and B TF32 (format 2), K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28
        const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(SM_BM >> 4) << 24);
        const uint32_t idesc2 = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(Cfg::ACC_COLS >> 3) << 17) | ((uint32_t)(SM_BM >> 4) << 24);
        int in_chain = 0;
        uint32_t acc = tmem;
        for (int i = 0; i < n_blocks; ++i) {
            const int s = i & 1;
            ok = mbar_wait_warp(full0 + 8 * s, (uint32_t)(i >> 1) & 1u, abort_flag, p.status, 15u);
            if (!ok) break;
            tc_fence_after();
            const uint64_t d = make_kmajor_sw128_desc(ring + s * Cfg::STAGE_BYTES);
            const uint32_t hi = (uint32_t)(d >> 32), ahi = (uint32_t)d, alo = ahi + (SM_A_TILE >> 4), w = alo + (SM_A_TILE >> 4);
            if (in_chain == per_chain) { in_chain = 0; acc += Cfg::ACC_COLS; }
            const bool first = in_chain++ == 0;
            if (lane == 0) {
#pragma unroll
                for (int j = 0; j < SM_BK / 8; ++j) {   // 8 TF32 per k-step: 32 bytes (descriptor units of 16 B)
                    // the weights' low rows lie behind the high ones: one instruction multiplies both with the activations' high parts
                    sm_mma_ss(acc, ahi + 2 * j, w + 2 * j, hi, idesc2, first && j == 0 ? 0u : 1u);
                    if (MODE3X) sm_mma_ss(acc + NT, alo + 2 * j, w + 2 * j, hi, idesc, 1u);
                }
                tc_commit(empty0 + 8 * s);
            }
            __syncwarp();
        }
        if (ok && lane == 0) tc_commit(acc_bar);
    }
    __syncwarp();
    if (p.cluster > 1) {
        cluster_wait();
    } else if (p.npeers > 0) {
        if (threadIdx.x == 0) sm_wait_peers(p);
        __syncthreads();
    }
    if (warp < 16) {
        if (p.bias) asm volatile("bar.sync 1, %0;" ::"n"(SM_EPI) : "memory");   // s_bias
        ok = ok && mbar_wait_warp(acc_bar, 0u, abort_flag, p.status, 16u);   // a warp's lanes agree on ok
        tc_fence_after();
        if (ok) {
            // four warps share a lane quarter and take a quarter of the columns each
            const int ml = (warp & 3) * 32 + lane, col0 = (warp >> 2) * (NT / 4);
            const int64_t m = m0 + ml;
            const uint32_t src = tmem + ((uint32_t)((warp & 3) * 32) << 16);
            constexpr int COLS = NT == 32 ? 8 : 16;   // per pass
#pragma unroll 1
            for (int col = col0; col < col0 + NT / 4 && col < n_rows; col += COLS) {
                float v[COLS];
                sm_sum<NT, MODE3X, COLS>(src + col, chains, v);
                if (p.cluster > 1) {
#pragma unroll
                    for (int e = 0; e < COLS; e += 4) {   // four columns of a row: 512 contiguous bytes per warp
                        const int four = (col + e) >> 2, dst = four * p.per_inv >> 16;
                        if (four >= fours) break;
                        const uint32_t at = part + (uint32_t)((rank * per + four - dst * per) * SM_BM + ml) * 16;
                        if (dst == rank) {
                            sts4f(at, v + e);
                            continue;
                        }
                        st_async2(in_cta(at, dst), in_cta(part_bar, dst), tc_pair(v[e], v[e + 1]), tc_pair(v[e + 2], v[e + 3]));
                    }
                } else if (m < p.M) {
                    float *q = p.C + (n0 + col) * p.ldc + m;
                    const int cols_here = n_rows - col < COLS ? n_rows - col : COLS;
                    if (p.bias) {
#pragma unroll
                        for (int e = 0; e < COLS; ++e) v[e] += s_bias[col + e];
                    }
                    if (p.act == CN_ACT_RELU) {
#pragma unroll
                        for (int e = 0; e < COLS; ++e) v[e] = v[e] > 0.0f ? v[e] : 0.0f;
                    } else if (p.act != CN_ACT_LINEAR) {
                        // one copy of the units' longer code: eight of them, with the switch around each, took 2500 clocks per pass, rectifiers too
#pragma unroll 1
                        for (int e = 0; e < COLS; ++e) {
                            const float y = cn_apply_activation(v[0], p.act);
#pragma unroll
                            for (int i = 0; i < COLS - 1; ++i) v[i] = v[i + 1];
                            v[COLS - 1] = y;
                        }
                    }
#pragma unroll
                    for (int e = 0; e < COLS; ++e, q += p.ldc)
                        if (e < cols_here) *q = v[e];
                    if (p.npeers > 0) {
#pragma unroll
                        for (int e = 0; e < COLS; ++e) {
                            if (e >= cols_here) continue;
                            for (int d = 0; d < p.npeers; ++d) p.peerC[d][(n0 + col + e) * p.ldc + m] = v[e];
                        }
                    }
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 16) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
    }
    if (p.cluster == 1) return;
    cluster_arrive_relaxed();   // this CTA has sent what it sends
    if (warp < 16) {
        if (p.npeers > 0) {
            if (threadIdx.x == 0) sm_wait_peers(p);
            asm volatile("bar.sync 1, %0;" ::"n"(SM_EPI) : "memory");
        }
        if (ok && n_mine > 0) ok = mbar_wait(part_bar, 0u, abort_flag, p.status, 24u) && mbar_try_cluster(part_bar, 0u) != 0u;
        // this CTA's columns, four at a time, a row m per lane
#pragma unroll 1
        for (int x = threadIdx.x; x < n_mine * SM_BM && ok; x += SM_EPI) {
            const int ml = x % SM_BM, col = 4 * (mine + x / SM_BM);
            const int64_t m = m0 + ml;
            if (m >= p.M) continue;
            uint32_t at = part + (uint32_t)x * 16;
            float4 v = lds4(at);
#pragma unroll 1
            for (int s = 1; s < p.cluster; ++s) {
                const float4 w = lds4(at += (uint32_t)(per * SM_BM * 16));
                v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
            }
            // one copy of the activations' code: it is fetched once per launch
            int64_t off = (n0 + col) * p.ldc + m;
#pragma unroll 1
            for (int e = col; e < col + 4 && e < n_rows; ++e, off += p.ldc) {
                const float y = cn_apply_activation(p.bias ? v.x + s_bias[e] : v.x, p.act);
                v.x = v.y; v.y = v.z; v.z = v.w;
                p.C[off] = y;
                for (int d = 0; d < p.npeers; ++d) p.peerC[d][off] = y;
            }
        }
    }
    // no CTA leaves before the others have sent; after a wait that ran out, what is under way gets a bounded chance to land
    __syncwarp();
    if (!ok) {
        const long long t0 = clock64();
        while (clock64() - t0 < 20000000LL) {}
    }
    __syncwarp();
    cluster_wait();
}

// Clusters of c CTAs that the device holds at once: the SMs of a cluster have to lie in one GPC.
static int max_clusters(const cn_context *ctx, int c)
{
    static int known[64][SM_MAX_CLUSTER + 1] = {};
    const int dev = ctx->device;
    if (c == 1) return ctx->sm_count;
    if (dev >= 0 && dev < 64 && known[dev][c] > 0) return known[dev][c];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ctx->sm_count / c * c));
    cfg.blockDim = dim3(SM_THREADS);
    cfg.dynamicSmemBytes = SmCfg<64, true>::smem(c);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(cn_gemm_small_kernel<64, true, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmCfg<64, true>::SMEM_MAX) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, cn_gemm_small_kernel<64, true, false, false>, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = 1;
    }
    if (dev >= 0 && dev < 64) known[dev][c] = n;
    return n;
}

// Columns per tile and CTAs per tile: the least of a rough model in ns, in which the blocks of K that a CTA takes (700 each) weigh most, then
// what comes once per CTA, the exchange in the cluster, and the output.  Measured with 128 rows (columns / CTAs, us): 784 x 1024 weights 64 / 5
// 9.3, 64 / 6 9.3, 128 / 8 9.3, 64 / 4 9.9, 32 / 4 10.7, 64 / 2 14.4; 400 x 400 32 / 5 6.1, 32 / 6 6.3, 32 / 4 6.7, 128 / 8 9; 1200 x 10 32 / 8 7.0, 128 / 8
// 7.8.  Clusters that wait for room (the GPCs hold 15 of eight or seven CTAs, 22 of six, 26 of five, 33 of four) cost a whole round more
// (1200 x 1200, 128 / 8 10.5, 64 / 8 18.0).
//
// In the 3x mode blocks_per_chain bounds the accumulation chains: tiles of 128 columns leave room for two accumulators, of 64 for four, of 32
// for eight, and a cluster of fewer CTAs makes them longer.  768 x 3873 . 3873 x 335 by four CTAs of 128 columns, 16 blocks per chain,
// was off by 1.17e-6, the fp32 kernel by 1.12e-6; see small_chain.
// Both passes over the plans, 36 at most, cost the host nothing that shows: 6.62 us per call, 6.64 with the twelve plans of powers of two (median of 250
// drawn products, queued without a wait).
// Clusters of three, five, six or seven CTAs only with chains no longer than those of the best plan without them, on average over the blocks
// (372 x 436 . 436 x 1512 by three CTAs in place of four was off by 2.5e-7 instead of 1.8e-7).
struct SmallPlan {
    int nt, cluster;
    int64_t ctas;
    double chain;   // blocks in the chain of a block, on average
};
static SmallPlan small_plan(const cn_context *ctx, int64_t M, int64_t N, int kb, int mode, int blocks_per_chain)
{
    // 32-bit numbers: the shapes that come here have at most two rounds of CTAs, and this runs on every call
    const int tiles_m = (int)((M + SM_BM - 1) / SM_BM), n32 = (int)((N + 31) / 32);
    auto least = [&](bool any_cluster, double max_chain) {
        SmallPlan best = {};
        int best_cost = INT_MAX;
        for (int c = 1; c <= SM_MAX_CLUSTER; c += any_cluster ? 1 : c) {
            if (c > 1 && kb < 2 * c) break;
            const int more = kb % c, least_blocks = kb / c, blocks = least_blocks + (more > 0), places = max_clusters(ctx, c);
            for (int nt = 32; nt <= 128; nt *= 2) {
                const int chains = nt == 128 ? SmCfg<128, true>::MAX_CHAINS : nt == 64 ? SmCfg<64, true>::MAX_CHAINS : SmCfg<32, true>::MAX_CHAINS;
                auto squares = [&](int b) { const int l = (b + chains - 1) / chains; return b / l * l * l + (b % l) * (b % l); };   // of a CTA's chains
                const double chain = (double)(more * squares(blocks) + (c - more) * squares(least_blocks)) / kb;
                if (mode == CN_GEMM_3XTF32 && ((blocks + chains - 1) / chains > blocks_per_chain || chain > max_chain)) continue;
                const int tiles = tiles_m * ((n32 + nt / 32 - 1) / (nt / 32)), rounds = (tiles + places - 1) / places;
                const int cost = rounds * (4000 + blocks * 700 + (c == 1 ? nt * 15 : 1500 + nt * 12));
                if (cost < best_cost) {
                    best_cost = cost;
                    best.nt = nt; best.cluster = c; best.chain = chain; best.ctas = (int64_t)tiles * c;
                }
            }
        }
        return best;
    };
    return least(true, least(false, blocks_per_chain).chain);
}

// CTAs per tile of 128 x 128 that there are SMs for, each with at least two K blocks; the measure of which products are small, and of how
// long their chains may be.  The CTAs that run are small_plan's.
static int small_cluster(int64_t tiles, int kb, int sms)
{
    int c = 1;
    while (c < SM_MAX_CLUSTER && tiles * c * 2 <= sms && kb >= c * 4) c *= 2;
    return c;
}

// Blocks of 32 k per accumulation chain that a small product may have.  The error grows with the additions to a running sum, four per block
// (the products with a low part, whose sums are small, have an accumulator of their own).  The measure of small products was found with
// four chains per CTA of that cluster and twelve additions per block, all in one accumulator, for weights that TMA cannot read with chains
// that ended between the k-steps of a block: no more additions than that, 12 ceil(b / 4) and 3 b for b blocks per CTA.  Every tile
// width has a plan within the limit: that cluster.  2059 x 1299 . 1299 x 98, six blocks per CTA: 18.9 us and 4.2e-7 by chains of six, 26.1
// and 2.6e-7 by what the limit leaves; 3.6e-7 with the eighteen additions of before.
static int small_chain(const cn_context *ctx, int64_t M, int64_t N, int kb, bool w_aligned)
{
    const int c = small_cluster(((M + SM_BM - 1) / SM_BM) * ((N + 127) / 128), kb, ctx->sm_count), blocks = (kb + c - 1) / c;
    return w_aligned ? 3 * ((blocks + 3) / 4) : blocks > 1 ? blocks * 3 / 4 : 1;
}

bool cn_gemm_small_shape(const cn_context *ctx, int64_t M, int64_t N, int64_t K, bool w_aligned, int max_rounds)
{
    if (M < 1 || N < 1 || K < 1) return false;
    if (N > (1 << 21) / K) return false;   // at most 8 MB of weights
    const int64_t tiles = ((M + SM_BM - 1) / SM_BM) * ((N + 127) / 128);
    const int kb = (int)((K + SM_BK - 1) / SM_BK);
    const int c = small_cluster(tiles, kb, ctx->sm_count);
    const int64_t per_cta = (kb + c - 1) / c, rounds = (tiles * c + ctx->sm_count - 1) / ctx->sm_count;
    // Where the line lies was measured with tiles of 128 columns, 1.5 us per block and that cluster; the plan that is launched (small_plan)
    // is faster, so that shapes just beyond the line may be faster here, too.  More than two rounds of CTAs cost more than the streaming
    // kernel's three launches: the 4096 x 4096 weight gradient of a batch of 128 (1024 tiles, seven rounds) took 108 us; the whole
    // backward pass went from 210 to 162 us.  The streaming kernel's launches and reduction cost 15 to 20 us: 16 x 8000 . 8000 x 64 (32 blocks)
    // took 43 us here.
    if (per_cta > (w_aligned ? SM_MAX_BLOCKS : SM_MAX_BLOCKS_ANY) || rounds > max_rounds) return false;
    // weights that TMA cannot read must not become less exact than on the fp32 kernel (cn_gemm_any_chain): a quarter of a CTA's blocks, of
    // twelve additions each, are the additions of a chain (see small_chain); a block of the streaming kernel has six
    const int chain = cn_gemm_any_chain(K) / 2;
    return w_aligned || (per_cta + 3) / 4 <= (chain > 1 ? chain : 1);
}

template <int NT, bool MODE3X, bool A_QUADS, bool W_QUADS>
static int small_launch(cn_context *ctx, const SmallParams &p, int64_t ctas, cudaStream_t s)
{
    static bool attr_set[64] = {};
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        CN_CUDA(cudaFuncSetAttribute(cn_gemm_small_kernel<NT, MODE3X, A_QUADS, W_QUADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmCfg<NT, MODE3X>::SMEM_MAX));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(SM_THREADS);
    cfg.dynamicSmemBytes = SmCfg<NT, MODE3X>::smem(p.cluster);
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
    CN_CUDA(cudaLaunchKernelEx(&cfg, cn_gemm_small_kernel<NT, MODE3X, A_QUADS, W_QUADS>, p));
    cn_count_launch();
    return CN_OK;
}

template <int NT, bool MODE3X>
static int small_pick(cn_context *ctx, const SmallParams &p, int64_t ctas, cudaStream_t s)
{
    const bool aq = p.A.sk != 1 && p.A.vec, wq = p.W.sk != 1 && p.W.vec;
    return aq ? (wq ? small_launch<NT, MODE3X, true, true>(ctx, p, ctas, s) : small_launch<NT, MODE3X, true, false>(ctx, p, ctas, s))
              : (wq ? small_launch<NT, MODE3X, false, true>(ctx, p, ctas, s) : small_launch<NT, MODE3X, false, false>(ctx, p, ctas, s));
}

int cn_gemm_small_launch(cn_context *ctx, int transA, int transB, int64_t M, int64_t N, int64_t K, const float *A, int64_t lda, const float *B, int64_t ldb,
                         float *C, int64_t ldc, const cn_epilogue *epi, int mode, cudaStream_t s, const cn_peer_out *peers)
{
    SmallParams p;
    unsigned int *d_status = nullptr;
    int st = cn_status_block(ctx, &d_status);
    if (st != CN_OK) return st;
    p.A = sm_operand(A, transA != 0, lda);
    p.W = sm_operand(B, transB == 0, ldb);
    p.M = M; p.N = N; p.K = K;
    p.C = C; p.ldc = ldc;
    p.bias = epi ? epi->bias : nullptr;
    p.act = epi ? epi->activation : CN_ACT_LINEAR;
    p.tiles_m = (int)((M + SM_BM - 1) / SM_BM);
    p.kb_total = (int)((K + SM_BK - 1) / SM_BK);
    const SmallPlan plan = small_plan(ctx, M, N, p.kb_total, mode, small_chain(ctx, M, N, p.kb_total, p.W.vec != 0));
    p.cluster = plan.cluster;
    p.per = (plan.nt / 4 + plan.cluster - 1) / plan.cluster;
    p.per_inv = (65536 + p.per - 1) / p.per;
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
    const bool m3 = mode == CN_GEMM_3XTF32;
    if (plan.nt == 32)      st = m3 ? small_pick<32, true>(ctx, p, plan.ctas, s) : small_pick<32, false>(ctx, p, plan.ctas, s);
    else if (plan.nt == 64) st = m3 ? small_pick<64, true>(ctx, p, plan.ctas, s) : small_pick<64, false>(ctx, p, plan.ctas, s);
    else                    st = m3 ? small_pick<128, true>(ctx, p, plan.ctas, s) : small_pick<128, false>(ctx, p, plan.ctas, s);
    if (st == CN_OK) {
        ctx->gemm_last_path = m3 ? "tcgen05_3xtf32" : "tcgen05_tf32";
        ctx->gemm_last_kernel = "small";
    }
    return st;
}
