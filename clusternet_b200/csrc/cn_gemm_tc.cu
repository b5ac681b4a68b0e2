// Tensor-core GEMM for sm_100a: TMA -> shared memory -> (converter warps) -> TMEM -> tcgen05.mma -> TMEM
// accumulators -> tcgen05.ld -> fused bias / activation / maxout -> global stores.
//
// Problem: C (M x N) = A (M x K) . W (K x N), everything fp32 column-major (the reference's device layout),
// which is the product ClusterNet::dot hands to cublasSgemm (source/clusterNet.cpp:459-461).
//
// Operands.  Every fp32 value is split into a high and a low part of 11 significand bits each (the TF32 split), and three
// products per k-step give fp32-level accuracy: D += Whi.Ahi + Wlo.Ahi + Whi.Alo.  CN_GEMM_TF32 issues only the first.
// TF32 and fp16 carry the same 11 significand bits, but the tensor cores multiply fp16 at twice the rate and its operands
// take half the room, so the parts are kept as fp16.  What fp16 lacks is exponent range; that is supplied by a power-of-two
// scale per row of the operand and segment of at most TC_GROUP_K = 512 k, exact to apply and to remove:
//   * activations: row m, segment of 512 k: the largest magnitude is brought into [2^14, 2^15);
//   * weights: column n, accumulation chain (below): the first K block that is not all zero brings its largest magnitude
//     into [2^13, 2^14); a later block that would leave fp16's range ends the chain early and starts a new one with a new scale.
// hi = fp16(s x) is exact to 2^-12 |s x|, lo = fp16(s x - hi) to 2^-24 |s x| or 2^-25, whichever is larger.  So an element within
// a factor 2^-15 of the largest of its segment keeps all 22 bits of the split, one 2^-19 below it 20.
//
// What fp16 cannot hold.  Of a smaller element more is lost, all of it from 2^-39 down; that counts where the large one meets a
// zero.  What hi + lo leave of an element, if it is more than 2^-20 of it (2^-10 in the single pass), is multiplied as well, in
// accumulation chains of its own with scales of their own:
//   * activations: what is left goes to a second pair of planes, scaled anew, and what that leaves to a third: 58 more binades.  They
//     are written, loaded and multiplied only for the blocks of 16 rows x 32 k that have something in them;
//   * weights: a converter warp that finds such elements in its 32 rows of a block writes what is left of them, 2^38 times the scale,
//     to an operand stage of its own, and again until nothing is left (elements 2^115 below the largest lose bits after all).
// Random operands have a few such elements by chance (uniform ones about 1 in 2^20); their chains cost less than the runs of a
// measurement differ, looking for them 5 to 10 %: 4096^3 432 -> 476 us, 128 x 100000 . 100000 x 40000 3450 -> 3700 us, single pass 128 x
// 40000 . 40000 x 40000 1030 -> 1078 us.  Measured on the same boxes: three bf16 parts of 8 bits and six products, which need no scales,
// 647, 5290 and (as TF32) 1310 us.
//
// Mapping.  A column-major W has its K index contiguous for a fixed column n, i.e. it is a K-major operand with
// N "rows".  The kernel therefore computes the transposed tile D[n, m] = sum_k W[k, n] * A[m, k]:
//   * the tcgen05 "A" operand (128 rows = 128 columns n of W) is read from TENSOR MEMORY.  W is streamed from
//     HBM exactly once as raw fp32 by TMA; four converter warps read each 128 x 32 tile from shared memory, scale and split
//     every value in registers and write both parts to TMEM with tcgen05.st.  No shared-memory traffic is spent on the split
//     and the raw weights never need a second copy in HBM;
//   * the tcgen05 "B" operand (UMMA N = 128 rows m of the activations) is read from shared memory.  The
//     activations are small next to W (M = 128 in the reference's layers), so a pre-pass re-lays them K-major
//     and pre-split into hi / lo planes once per call; every CTA then pulls 128 x 64 tiles of both planes by TMA;
//   * the accumulator tile lives in TMEM with lane = n and column = m, so in the epilogue one thread owns one
//     output column n and 128 consecutive rows m: the bias is a per-thread scalar, and maxout over L consecutive columns is a
//     shuffle across L lanes.
//
// Work decomposition.  One persistent CTA per SM; a tile is 128 rows m by NT * 128 columns n.  As many whole tiles as there
// are full rounds over the SMs are multiplied over all of K by one CTA each (in lockstep along K, so that the activation tiles
// are shared through L2); the tiles that are left are cut into equal runs of K blocks over all SMs.  A run leaves its partial
// tile in scratch and a second, grid-wide kernel adds the partial tiles in K order (a fixed order, so results are
// reproducible) and runs the epilogue.
//
// Every wait on an mbarrier is bounded by a clock limit; a wait that runs out sets a status word that the host
// reads back as CN_ERR_TIMEOUT, lets the other roles drain, frees the tensor memory and returns.
#include <cuda.h>
#include <stdlib.h>
#include "cn_epilogue.cuh"
#include "cn_gemm.h"
#include "cn_gemm_tc.h"
#include "cn_tc_split.cuh"

#define TC_W_TILE_BYTES (TC_BN * TC_WK * 4)
#define CN_TC_MAX_CLUSTER 8

// How the weights lie in memory: k contiguous or n contiguous ("transposed"), the rows of that layout 16-byte aligned or not.
//
// TMA wants 16-byte aligned rows.  For any other pitch or base the rows of the stored matrix are read as four tensors: rows
// r, r + 4, r + 8, ... lie 4 * pitch floats = 16 * pitch bytes apart, a multiple of 16 for every pitch, and all start at the same
// offset d_r of 0 to 3 floats behind a 16-byte boundary.  Tensor r starts at that boundary and is d_r floats wider; its box is four
// floats wider than the tile, and the converters begin to read d_r floats in.  What is read to the left of a row is not used; behind
// its end and below the last row TMA fills with zeros, as for aligned weights.  Every weight is still read from memory once, with
// no copy of the matrix.  203 x 4001 . 4001 x 3001: 412 us on the fp32 FMA kernel that took such weights before, 57 us here.
enum { W_K = 0, W_N = 1, W_K_ANY = 2, W_N_ANY = 3 };
#define TC_CLASSES 4
#define TC_WK_PITCH (TC_WK + 4)                                  // floats per row of a W_K_ANY box (32 rows), conflict-free for odd pitches
#define TC_WK_CLASS_BYTES (TC_BN / TC_CLASSES * TC_WK_PITCH * 4)
#define TC_WN_PITCH (TC_BN + 4)                                  // floats per row of a W_N_ANY box (8 rows)
#define TC_WN_CLASS_BYTES (TC_WK / TC_CLASSES * TC_WN_PITCH * 4)
static_assert(TC_WK_CLASS_BYTES % 128 == 0 && TC_WN_CLASS_BYTES % 128 == 0, "TMA destinations");
__host__ __device__ constexpr bool w_any(int wk) { return wk >= W_K_ANY; }
__host__ __device__ constexpr int w_box_bytes(int wk)
{
    return wk == W_K_ANY ? TC_CLASSES * TC_WK_CLASS_BYTES : wk == W_N_ANY ? TC_CLASSES * TC_WN_CLASS_BYTES : TC_W_TILE_BYTES;
}

template <int NT, bool MODE3X, int WK>
struct TcCfg {
    static constexpr int THREADS = 128 + 256 * NT;    // WG0 (producers, MMA), per W tile one converter and one drain warpgroup
    // Two shared-memory rings with their own depth: raw W blocks (released by the converters as soon as they have
    // been read) and activation hi / lo tiles (released when the MMAs that read them retire).
    static constexpr int W_STAGES = NT == 1 ? 6 : 3;
    static constexpr int A_STAGES = 3;
    static constexpr int W_TILE_BYTES = w_any(WK) ? TC_CLASSES * TC_WK_CLASS_BYTES : TC_W_TILE_BYTES;
    static constexpr int W_STAGE_BYTES = NT * W_TILE_BYTES;
    static constexpr int A_STAGE_BYTES = 2 * TC_A_TILE_BYTES;
    static constexpr int W_RING = 0;
    static constexpr int A_RING = W_STAGES * W_STAGE_BYTES;
    static constexpr int RING_BYTES = A_RING + A_STAGES * A_STAGE_BYTES;
    static_assert(A_RING % 1024 == 0, "swizzled tiles");
    static_assert(A_STAGES >= TC_BANDS, "the bands of a stage are held together");
    static constexpr int TMEM_STAGES = NT == 2 && MODE3X ? 3 : 4;
    static constexpr int ACC_BUFS = NT == 1 ? 2 : 1;  // accumulators per W tile
    static constexpr int ACC_COL = 0;                 // NT * ACC_BUFS accumulators of 128 columns
    static constexpr int OP_COL = NT * ACC_BUFS * TC_BM;   // then TMEM_STAGES x NT x 2 k-steps x (8 hi + 8 lo) columns (no lo in the single pass)
    static constexpr int STEP_COLS = MODE3X ? 16 : 8, OP_COLS = 2 * STEP_COLS;
    static constexpr int OP_STAGE_COLS = NT * OP_COLS;
    static constexpr int LEFT_COL = OP_COL + TMEM_STAGES * OP_STAGE_COLS;   // what is left of a block of weights, per W tile
    static_assert(LEFT_COL + OP_STAGE_COLS <= 512, "tensor memory");
    // Scales of the W rows, one slot per W block: the drain warps read the slot of a chain's last block.  The converters
    // run at most TMEM_STAGES blocks ahead of the MMAs, and the MMAs at most ACC_BUFS - 1 chains ahead of the drain.
    static constexpr int WS_SLOTS = NT == 1 ? 32 : 8;
    static_assert(WS_SLOTS > TMEM_STAGES + (ACC_BUFS - 1) * TC_GROUP_KB, "a scale must outlive its chain");
    static constexpr int WS_OFF = RING_BYTES;                              // [WS_SLOTS][NT][128] floats
    static constexpr int AS_OFF = WS_OFF + WS_SLOTS * NT * TC_BN * 4;      // [2][NT][128] floats
    static constexpr int BRK_OFF = AS_OFF + 2 * NT * TC_BM * 4;            // [TMEM_STAGES][NT] words of four bytes, one per converter warp
    static constexpr int LEFT_OFF = BRK_OFF + TMEM_STAGES * NT * 4;        // [NT] words: whether more is left, a byte per converter warp
    static constexpr int BAND_OFF = LEFT_OFF + NT * 4;        // [A_STAGES] words: blocks of 16 rows with left-overs, a byte per 32 k and band
    static_assert(TC_BANDS == 3, "four bytes");
    static constexpr int INFO_OFF = BAND_OFF + A_STAGES * 4;               // [NT][ACC_BUFS] pairs of words
    static constexpr int BAR_OFF = (INFO_OFF + NT * ACC_BUFS * 8 + 7) & ~7;
    static constexpr int BARS = 2 * (W_STAGES + A_STAGES + NT * TMEM_STAGES + NT * ACC_BUFS + NT * 4) + 1;
    static constexpr int HOLD_OFF = BAR_OFF + BARS * 8;                    // tensor-memory base, abort flag
    static constexpr int SMEM_BYTES = HOLD_OFF + 16 + 1024 /*align*/;
    static_assert(SMEM_BYTES <= 232448, "shared memory");
    // register budgets after the warpgroups re-balance: multiples of 8, their sum over the warpgroups at most what the launch has
    // (NT = 2: 5 x 96, NT = 1: 3 x 168).  4096^3: 495 us with 48 and 168, 476 with 56 and 160; single pass 128 x 40000 x 40000: 1090 and 1101.
    static constexpr int REGS_WG0 = NT == 1 ? 88 : 48;
    static constexpr int REGS_CONV = NT == 1 ? 104 : MODE3X ? 56 : 48;
    static constexpr int REGS_DRAIN = NT == 1 ? 232 : MODE3X ? 160 : 168;
    static_assert(REGS_WG0 + NT * (REGS_CONV + REGS_DRAIN) <= (1 + 2 * NT) * (65536 / THREADS / 8 * 8), "registers");
};

struct TcParams {
    int64_t M, N;
    float *C;
    int64_t ldc;
    const float *bias;
    int act;
    int maxout_level;
    float *argmax;
    int tiles_n;            // groups of NT*128 columns
    int tiles_m;
    int full_tiles;         // tiles [0, full_tiles): all of K by one CTA; the others are cut into runs over tail_ctas CTAs
    int tail_ctas;
    int kb_total;           // K blocks of 32
    int cluster;            // CTAs that share a tile's K and add its parts themselves; 1: runs leave partial tiles
    int chain_mask;         // K blocks per accumulation chain - 1 (a power of two, at most TC_GROUP_KB)
    const float *a_inv;     // [band][group of 512 k][m_pad] inverse scales of the activation rows
    int64_t m_pad;
    int groups;
    const uint8_t *a_bands; // [tile of 128 rows][64 k][block of 16 rows]: bands behind the first that have something in them, four bits per 32 k
    int a_stages;           // ceil(K / 64)
    float *partials;        // [slot][w][32 quads of m][128 n] float4: slot = CTA + tile - full_tiles
    unsigned int *status;
    uint32_t w_shift;       // byte r: d_r of the weights' rows r, r + 4, ... (see W_K_ANY)
    unsigned int *cond;     // CN_STATUS_MANY: run only where this word is not zero (see cn_tc_cond); null: always
    int w_ready;            // nothing before the pre-pass still writes W: it may be loaded before the pre-pass has finished
    // fused all-gather: the peers are told that this rank's C may be overwritten; the tiles go to them in the reduction
    int npeers;
    unsigned int *const *peer_flags;
    int nranks;
    int my_rank;
    unsigned int epoch;
};

// One run of K blocks of one tile.
struct TcSeg {
    int tile, k0, k1;
    int slot;       // where the partial tile goes; -1: the run is the whole tile and is finished in place
};

// A cluster's CTAs share the rows m of their tile in units of 16: CTA number `rank` finishes `mine` of them, from unit rank * per on.
struct TcShare {
    int rank, units, per, mine;
    __device__ __forceinline__ explicit TcShare(const TcParams &p)
    {
        const int tile = (int)blockIdx.x / p.cluster;
        const int64_t rows = p.M - (int64_t)(tile % p.tiles_m) * TC_BM;
        rank = (int)blockIdx.x - tile * p.cluster;
        units = rows < TC_BM ? (int)(rows + 15) >> 4 : TC_BM / 16;
        per = (units + p.cluster - 1) / p.cluster;
        mine = units - rank * per < per ? units - rank * per : per;
    }
};

// The runs of CTA `cta`, in order.  All roles of a CTA walk the same list.
struct TcWalk {
    int t;
    int64_t pos, end;
    __device__ __forceinline__ explicit TcWalk(const TcParams &p)
    {
        t = blockIdx.x;
        pos = end = 0;
        if ((int)blockIdx.x < p.tail_ctas) {
            const int64_t total = (int64_t)(p.tiles_n * p.tiles_m - p.full_tiles) * p.kb_total;
            pos = total * blockIdx.x / p.tail_ctas;
            end = total * (blockIdx.x + 1) / p.tail_ctas;
        }
    }
    __device__ __forceinline__ bool next(const TcParams &p, TcSeg &s)
    {
        if (t < p.full_tiles) {
            s.tile = t;
            s.k0 = 0;
            s.k1 = p.kb_total;
            s.slot = -1;
            t += gridDim.x;
            return true;
        }
        if (pos < end) {
            const int r = (int)(pos / p.kb_total);
            s.k0 = (int)(pos - (int64_t)r * p.kb_total);
            const int64_t left = end - pos;
            const int room = p.kb_total - s.k0;
            s.k1 = s.k0 + (left < room ? (int)left : room);
            s.tile = p.full_tiles + r;
            s.slot = blockIdx.x + r;
            pos += s.k1 - s.k0;
            return true;
        }
        return false;
    }
};

// D[tmem] (+)= A[tmem] * B[smem desc]; A: 128 lanes x 16 fp16 (two per column: 8 columns), B: 128 x 16 K-major fp16 tile.
// The descriptor travels as two 32-bit halves so that stepping along K is a 32-bit add on the low half.
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_desc_lo, uint32_t b_desc_hi, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 bd;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 bd, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], bd, %4, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_desc_lo), "r"(b_desc_hi), "r"(idesc), "r"(accumulate) : "memory");
}

// -------------------------------------------------------------------------------------------------- main kernel
// Four consecutive k of one row of a 128 x 32 W tile (chunk c of 8).  `base` is the address tc_row_base gives.
// W_N: the tiles arrive in shared memory as [32 k][128 n] without swizzle and are read column-wise (conflict-free: consecutive
// lanes read consecutive n).  The _ANY layouts lie in four boxes, one per class of rows.
template <int WK>
__device__ __forceinline__ uint32_t tc_row_base(uint32_t tile, int row, uint32_t w_shift)
{
    if (WK == W_N || WK == W_N_ANY) return tile + row * 4;
    if (WK == W_K_ANY) return tile + (row & 3) * TC_WK_CLASS_BYTES + (row >> 2) * (TC_WK_PITCH * 4) + ((w_shift >> ((row & 3) * 8)) & 0xffu) * 4;
    // 16-byte chunk c of row r sits at chunk position c ^ (r & 7) under the 128-byte swizzle (tiles are 1024-byte aligned)
    return tile + row * 128 + ((row & 7) << 4);
}
template <int WK>
__device__ __forceinline__ float4 tc_read4(uint32_t base, int c, uint32_t w_shift)
{
    if (WK == W_N)
        return make_float4(lds1(base + (4 * c) * (TC_BN * 4)), lds1(base + (4 * c + 1) * (TC_BN * 4)), lds1(base + (4 * c + 2) * (TC_BN * 4)),
                           lds1(base + (4 * c + 3) * (TC_BN * 4)));
    if (WK == W_K_ANY) return make_float4(lds1(base + 16 * c), lds1(base + 16 * c + 4), lds1(base + 16 * c + 8), lds1(base + 16 * c + 12));
    if (WK == W_N_ANY) {
        const uint32_t q = base + c * (TC_WN_PITCH * 4);
        return make_float4(lds1(q + (w_shift & 0xffu) * 4), lds1(q + TC_WN_CLASS_BYTES + ((w_shift >> 8) & 0xffu) * 4),
                           lds1(q + 2 * TC_WN_CLASS_BYTES + ((w_shift >> 16) & 0xffu) * 4), lds1(q + 3 * TC_WN_CLASS_BYTES + (w_shift >> 24) * 4));
    }
    return lds4(base ^ (c << 4));
}

template <int WK>
__device__ __forceinline__ void tc_write4(uint32_t base, int c, uint32_t w_shift, float4 v)
{
    if (WK == W_K) {
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(base ^ (c << 4)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
        return;
    }
    const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (WK == W_N) sts1(base + (4 * c + e) * (TC_BN * 4), x[e]);
        if (WK == W_K_ANY) sts1(base + 16 * c + 4 * e, x[e]);
        if (WK == W_N_ANY) sts1(base + c * (TC_WN_PITCH * 4) + e * TC_WN_CLASS_BYTES + ((w_shift >> (8 * e)) & 0xffu) * 4, x[e]);
    }
}

// One k-step (16 consecutive k of column n) of one row, scaled by sc -> hl[0..7] packed high parts, hl[8..15] packed low parts.
// Keeps the running packed largest and smallest |high part|: 0x7c00 means that a value left fp16's range, less than
// tc_safe_f16 that its parts may leave something (or that it is a zero).
template <bool MODE3X, int WK>
__device__ __forceinline__ void tc_convert_step(uint32_t base, uint32_t w_shift, int step, uint64_t sc2, uint32_t (&hl)[16], uint32_t &top, uint32_t &low)
{
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float4 v = tc_read4<WK>(base, step * 4 + c, w_shift);
        tc_split2<MODE3X>(tc_mul2(tc_pack2(v.x, v.y), sc2), hl[2 * c], hl[8 + 2 * c]);
        tc_split2<MODE3X>(tc_mul2(tc_pack2(v.z, v.w), sc2), hl[2 * c + 1], hl[8 + 2 * c + 1]);
        asm("max.xorsign.abs.f16x2 %0, %0, %1;" : "+r"(top) : "r"(hl[2 * c]));
        asm("max.xorsign.abs.f16x2 %0, %0, %1;" : "+r"(top) : "r"(hl[2 * c + 1]));
        asm("min.xorsign.abs.f16x2 %0, %0, %1;" : "+r"(low) : "r"(hl[2 * c]));
        asm("min.xorsign.abs.f16x2 %0, %0, %1;" : "+r"(low) : "r"(hl[2 * c + 1]));
    }
}

template <int WK>
__device__ __forceinline__ uint32_t tc_row_amax(uint32_t base, uint32_t w_shift)
{
    uint32_t amax = 0u;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float4 v = tc_read4<WK>(base, c, w_shift);
        amax = max(max(amax, __float_as_uint(v.x) & 0x7fffffffu), max(__float_as_uint(v.y) & 0x7fffffffu, __float_as_uint(v.z) & 0x7fffffffu));
        amax = max(amax, __float_as_uint(v.w) & 0x7fffffffu);
    }
    return amax;
}

// Whether the parts of this row's 32 values leave something: the smallest nonzero magnitude tells that they do not, else every
// value's parts are made once more.
template <bool MODE3X, int WK>
__device__ __forceinline__ bool tc_row_left(uint32_t base, uint32_t w_shift, float sc)
{
    uint32_t amin = 0xffffffffu;   // of 2 |bits| - 1, in which a zero is the largest
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float4 v = tc_read4<WK>(base, c, w_shift);
        amin = min(min(amin, __float_as_uint(v.x) * 2u - 1u), min(__float_as_uint(v.y) * 2u - 1u, __float_as_uint(v.z) * 2u - 1u));
        amin = min(amin, __float_as_uint(v.w) * 2u - 1u);
    }
    if (amin == 0xffffffffu || __uint_as_float((amin + 1u) >> 1) * sc >= (MODE3X ? 0.03125f : 6.103515625e-5f)) return false;
    bool left = false;
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
        const float4 v = tc_read4<WK>(base, c, w_shift);
        uint32_t h, l;
        float r[4];
        tc_split2_left<MODE3X>(v.x * sc, v.y * sc, h, l, r[0], r[1]);
        tc_split2_left<MODE3X>(v.z * sc, v.w * sc, h, l, r[2], r[3]);
        left |= r[0] != 0.0f || r[1] != 0.0f || r[2] != 0.0f || r[3] != 0.0f;
    }
    return left;
}

// Tensor maps of the weights: one, or one per class of rows (W_K_ANY, W_N_ANY).
struct WMaps {
    CUtensorMap map[TC_CLASSES];
};

// Warp roles (warpgroups of 4 warps so that register budgets can be moved between them):
//   WG0  warp 0: TMA producer for W, warp 1: MMA issuer of W tile 0 + TMEM owner, warp 2: TMA producer for the
//        activations, warp 3: MMA issuer of W tile 1 (NT == 2)
//   then one warpgroup of converters per W tile (raw W block in shared memory -> scaled fp16 hi / lo parts in TMEM)
//   and one warpgroup for accumulator drain + epilogue per W tile.
// The two W tiles of a CTA share the W and activation rings and are otherwise independent of each other.  One converter
// warpgroup for both tiles was short of registers (their spills went through the shared-memory pipe) and of warps to hide
// the latency of its conversions: 3.8 ms for 128 x 100000 x 40000 against 3.2 ms with the conversion left out.
//
// Accumulation chains.  The tensor core adds into its fp32 accumulator with truncation, so a long chain of
// accumulating MMAs drifts (about 6e-8 of the running sum per step, all in one direction).  The K loop is therefore
// cut into chains of at most 512 k, which end where the activations' scale groups end: each chain starts a fresh TMEM
// accumulator, and when it ends the drain warps read it with tcgen05.ld, remove both scales and add it, in round-to-nearest
// fp32, to running sums that they keep in registers (one thread = one output column n, 128 sums = 128 rows m).
// SHARED: the CTAs of a cluster share a tile's K and add its parts themselves (an instance of its own: as a branch it cost the others 0.6 us).
template <int NT, bool MODE3X, int WK, bool SHARED>
__global__ void __launch_bounds__(TcCfg<NT, MODE3X, WK>::THREADS, 1)
cn_gemm_tc_kernel(const __grid_constant__ WMaps tm_w, const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ TcParams p)
{
    using Cfg = TcCfg<NT, MODE3X, WK>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    constexpr int B_WFULL = 0, B_WEMPTY = B_WFULL + Cfg::W_STAGES, B_AFULL = B_WEMPTY + Cfg::W_STAGES,
                  B_AEMPTY = B_AFULL + Cfg::A_STAGES, B_TFULL = B_AEMPTY + Cfg::A_STAGES, B_TEMPTY = B_TFULL + NT * Cfg::TMEM_STAGES,
                  B_ACCFULL = B_TEMPTY + NT * Cfg::TMEM_STAGES, B_ACCEMPTY = B_ACCFULL + NT * Cfg::ACC_BUFS;
    constexpr int B_XFULL = B_ACCEMPTY + NT * Cfg::ACC_BUFS, B_XEMPTY = B_XFULL + NT * 4;   // left-overs of the weights, per converter warp
    constexpr int B_PART = B_XEMPTY + NT * 4;   // this CTA's rows of the partial tiles of its cluster have arrived
    static_assert(B_PART + 1 == Cfg::BARS, "barrier count");
    auto bar = [&](int idx) { return smem_base + Cfg::BAR_OFF + 8u * idx; };
    auto wfull_bar = [&](int s) { return bar(B_WFULL + s); };
    auto wempty_bar = [&](int s) { return bar(B_WEMPTY + s); };
    auto afull_bar = [&](int s) { return bar(B_AFULL + s); };
    auto aempty_bar = [&](int s) { return bar(B_AEMPTY + s); };
    auto tfull_bar = [&](int w, int t) { return bar(B_TFULL + w * Cfg::TMEM_STAGES + t); };
    auto tempty_bar = [&](int w, int t) { return bar(B_TEMPTY + w * Cfg::TMEM_STAGES + t); };
    auto accfull_bar = [&](int w, int b) { return bar(B_ACCFULL + w * Cfg::ACC_BUFS + b); };
    auto accempty_bar = [&](int w, int b) { return bar(B_ACCEMPTY + w * Cfg::ACC_BUFS + b); };
    auto xfull_bar = [&](int w, int q) { return bar(B_XFULL + w * 4 + q); };
    auto xempty_bar = [&](int w, int q) { return bar(B_XEMPTY + w * 4 + q); };
    const uint32_t tmem_holder = smem_base + Cfg::HOLD_OFF, abort_flag = tmem_holder + 4;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    cn_pdl_launch_dependents();
    if (p.cond) {
        cn_pdl_wait();
        if (blockIdx.x == 0 && threadIdx.x == 0) p.cond[CN_STATUS_OVERFLOW - CN_STATUS_MANY] = 0u;   // for the next product
        // one thread looks at the word: the reads of every warp of all CTAs meet in one line
        if (!__syncthreads_or(threadIdx.x == 0 && __ldcg(p.cond) != 0u)) return;
    }

    // Fused all-gather: everything queued earlier on this GPU's stream has finished, so this rank's copy of C may now be
    // overwritten by its peers: tell them (slot 0 of their flag block).
    if (p.npeers > 0 && blockIdx.x == 0 && threadIdx.x < p.nranks && (int)threadIdx.x != p.my_rank) {
        cn_pdl_wait();
        __threadfence_system();
        volatile unsigned int *f = p.peer_flags[threadIdx.x] + p.my_rank;
        *f = p.epoch;
    }

    if (threadIdx.x == 0) {
        for (int s = 0; s < Cfg::W_STAGES; ++s) { mbar_init(wfull_bar(s), 1); mbar_init(wempty_bar(s), 4 * NT); }
        for (int s = 0; s < Cfg::A_STAGES; ++s) { mbar_init(afull_bar(s), 1); mbar_init(aempty_bar(s), NT); }
        for (int w = 0; w < NT; ++w) {
            for (int t = 0; t < Cfg::TMEM_STAGES; ++t) { mbar_init(tfull_bar(w, t), 4); mbar_init(tempty_bar(w, t), 1); }
            for (int b = 0; b < Cfg::ACC_BUFS; ++b) { mbar_init(accfull_bar(w, b), 2); mbar_init(accempty_bar(w, b), 4); }
            for (int q = 0; q < 4; ++q) { mbar_init(xfull_bar(w, q), 1); mbar_init(xempty_bar(w, q), 1); }
        }
        if (SHARED) mbar_init(bar(B_PART), 1);
        if (SHARED) {
            const TcShare s(p);
            if (s.mine > 0) mbar_expect_tx(bar(B_PART), (uint32_t)((p.cluster - 1) * s.mine * (16 * 4) * (NT * TC_BN)));
        }
        sts1u(abort_flag, 0u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {   // this warp owns the tensor-memory allocation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_holder), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = lds1u(tmem_holder);

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::REGS_WG0));
        if (warp == 0) {
            // ------------------------------------------------------------ TMA producer of W
            if (lane == 0) {
                TcWalk walk(p);
                TcSeg seg;
                if (!p.w_ready) cn_pdl_wait();
                uint32_t it = 0;
                bool ok = true;
                while (ok && walk.next(p, seg)) {
                    const int32_t n0 = (seg.tile / p.tiles_m) * (NT * TC_BN);
                    for (int kb = seg.k0; kb < seg.k1; ++kb, ++it) {
                        const int s = it % Cfg::W_STAGES;
                        ok = mbar_wait(wempty_bar(s), ((it / Cfg::W_STAGES) & 1u) ^ 1u, abort_flag, p.status, 1u);
                        if (!ok) break;
                        const uint32_t stage = smem_base + Cfg::W_RING + s * Cfg::W_STAGE_BYTES;
                        mbar_expect_tx(wfull_bar(s), (uint32_t)(NT * w_box_bytes(WK)));
#pragma unroll
                        for (int t = 0; t < NT; ++t) {
                            const uint32_t dst = stage + t * Cfg::W_TILE_BYTES;
                            const int32_t n = n0 + t * TC_BN;
                            if (WK == W_K) tma_load_2d(dst, &tm_w.map[0], wfull_bar(s), kb * TC_WK, n);
                            if (WK == W_N) tma_load_2d(dst, &tm_w.map[0], wfull_bar(s), n, kb * TC_WK);
                            if (w_any(WK)) {
#pragma unroll
                                for (int r = 0; r < TC_CLASSES; ++r) {
                                    if (WK == W_K_ANY) tma_load_2d(dst + r * TC_WK_CLASS_BYTES, &tm_w.map[r], wfull_bar(s), kb * TC_WK, n / TC_CLASSES);
                                    else               tma_load_2d(dst + r * TC_WN_CLASS_BYTES, &tm_w.map[r], wfull_bar(s), n, kb * (TC_WK / TC_CLASSES));
                                }
                            }
                        }
                    }
                }
                if (lds1u(abort_flag) != 0u) {
                    // give copies that are still in flight a bounded chance to land before the CTA exits
                    for (uint32_t i = it > Cfg::W_STAGES ? it - Cfg::W_STAGES : 0; i < it; ++i) {
                        const long long t0 = clock64();
                        while (!mbar_try(wfull_bar(i % Cfg::W_STAGES), (i / Cfg::W_STAGES) & 1u) && clock64() - t0 < 20000000LL) {}
                    }
                }
            }
            __syncwarp();
        } else if (warp == 2) {
            // ------------------------------------------------------------ TMA producer of the activations
            if (lane == 0) {
                TcWalk walk(p);
                TcSeg seg;
                tma_prefetch_map(&tm_a);
                cn_pdl_wait();
                uint32_t it = 0;
                bool ok = true;
                while (ok && walk.next(p, seg)) {
                    const int32_t m0 = (seg.tile % p.tiles_m) * TC_BM;
                    const uint2 *bands = reinterpret_cast<const uint2 *>(p.a_bands) + (int64_t)(seg.tile % p.tiles_m) * p.a_stages;
                    uint2 b8 = __ldcg(bands + (seg.k0 >> 1));   // bands of the eight blocks of 16 rows, a byte each
                    for (int kb = seg.k0 & ~1; kb < seg.k1 && ok; kb += 2) {
                        const uint2 now = b8;
                        if (kb + 2 < seg.k1) b8 = __ldcg(bands + (kb >> 1) + 1);
                        uint32_t masks = 0u;                        // byte b - 1, and b + 1 for the second 32 k: the blocks that have something in band b
                        if ((now.x | now.y) != 0u) {
                            for (int j = 0; j < 16; ++j) {
                                const uint32_t n = ((j < 8 ? now.x : now.y) >> (4 * (j & 7))) & 0xfu;
                                for (uint32_t b = 0; b < n; ++b) masks |= 1u << (16 * (j & 1) + 8 * b + (j >> 1));
                            }
                        }
                        const int bands_here = 1 + (masks != 0u) + ((masks & 0xff00ff00u) != 0u);
                        for (int band = 0; band < bands_here; ++band, ++it) {
                            const int s = it % Cfg::A_STAGES;
                            ok = mbar_wait(aempty_bar(s), ((it / Cfg::A_STAGES) & 1u) ^ 1u, abort_flag, p.status, 8u);
                            if (!ok) break;
                            const uint32_t stage = smem_base + Cfg::A_RING + s * Cfg::A_STAGE_BYTES;
                            if (band == 0) sts1u(smem_base + Cfg::BAND_OFF + s * 4, masks);
                            mbar_expect_tx(afull_bar(s), (uint32_t)((MODE3X ? 2 : 1) * TC_A_TILE_BYTES));
                            tma_load_3d(stage, &tm_a, afull_bar(s), kb * TC_WK, m0, band * (MODE3X ? 2 : 1));
                            if (MODE3X) tma_load_3d(stage + TC_A_TILE_BYTES, &tm_a, afull_bar(s), kb * TC_WK, m0, 2 * band + 1);
                        }
                    }
                }
                // the last stages' releases (commits of the MMA issuers) must have arrived before the CTA may exit; on the way out
                // after a wait that ran out, copies in flight get a bounded chance to land
                const bool aborted = lds1u(abort_flag) != 0u;
                for (uint32_t i = it > Cfg::A_STAGES ? it - Cfg::A_STAGES : 0; i < it; ++i) {
                    const int s = i % Cfg::A_STAGES;
                    const uint32_t ph = (i / Cfg::A_STAGES) & 1u;
                    if (!aborted) {
                        if (!mbar_wait(aempty_bar(s), ph, abort_flag, p.status, 11u)) break;
                    } else {
                        const long long t0 = clock64();
                        while (!mbar_try(afull_bar(s), ph) && clock64() - t0 < 20000000LL) {}
                    }
                }
            }
            __syncwarp();
        } else if (warp == 1 || (NT == 2 && warp == 3)) {
            // ------------------------------------------------------------ MMA issuers: one thread per W tile
            if (lane == 0) {
                TcWalk walk(p);
                TcSeg seg;
                const int w = warp == 1 ? 0 : 1;
                constexpr uint32_t idesc = make_idesc_f16(TC_BN, TC_BM);
                uint32_t it = 0, a_it = 0;       // W blocks and activation stages so far
                int ab = 0;                      // accumulator buffer and its phase
                uint32_t aph = 0, xph = 0;       // ... of the left-overs, a bit per converter warp
                bool open = false, ok = true;    // a chain is accumulating
                // Ends the open chain: the drain warps learn where its scales are and which blocks of 16 rows m it has (mask, from bit
                // 16), for left-overs of the weights how often they were scaled (from bit 9) and which quarters of the rows n have
                // any (from bit 24), and that it is complete when its MMAs retire
                constexpr uint32_t WHOLE = 0x0fff0000u;
                auto close_chain = [&](uint32_t last_it, int a_scales, uint32_t what, bool last_of_run) {
                    const uint32_t q = smem_base + Cfg::INFO_OFF + (w * Cfg::ACC_BUFS + ab) * 8;
                    sts1u(q, (last_it % Cfg::WS_SLOTS) | (last_of_run ? 0x100u : 0u) | what);
                    sts1u(q + 4, (uint32_t)a_scales);
                    mbar_arrive(accfull_bar(w, ab));
                    tc_commit(accfull_bar(w, ab));
                    if (++ab == Cfg::ACC_BUFS) { ab = 0; aph ^= 1u; }
                    open = false;
                };
                auto open_chain = [&]() {   // the drain warps must have emptied this accumulator
                    if (!mbar_wait(accempty_bar(w, ab), aph ^ 1u, abort_flag, p.status, 7u)) return false;
                    tc_fence_after();
                    open = true;
                    return true;
                };
                auto wait_weights = [&](uint32_t i) { return mbar_wait(tfull_bar(w, i % Cfg::TMEM_STAGES), (i / Cfg::TMEM_STAGES) & 1u, abort_flag, p.status, 3u); };
                auto wait_stage = [&](uint32_t a) { return mbar_wait(afull_bar(a % Cfg::A_STAGES), (a / Cfg::A_STAGES) & 1u, abort_flag, p.status, 2u); };
                // operands of one W block: the activation stage where it opens one, and the converted W rows
                auto wait_block = [&](uint32_t i, uint32_t a, bool opens_stage) { return (!opens_stage || wait_stage(a)) && wait_weights(i); };
                // what the converters say of a block of weights, a byte per warp: 1 = a row's scale had to change, the chain ends before
                // it; 2 = something is left of it.  And what is left of the activations of a stage, see their producer.
                auto block_word = [&](uint32_t i) { return lds1u(smem_base + Cfg::BRK_OFF + ((i % Cfg::TMEM_STAGES) * NT + w) * 4); };
                auto stage_masks = [&](uint32_t a) { return lds1u(smem_base + Cfg::BAND_OFF + (a % Cfg::A_STAGES) * 4); };
                while (ok && walk.next(p, seg)) {
                    ok = wait_block(it, a_it, true);
                    uint32_t word = block_word(it), masks = stage_masks(a_it);
                    for (int kb = seg.k0; kb < seg.k1 && ok; ++kb, ++it) {
                        const int s = a_it % Cfg::A_STAGES, t = it % Cfg::TMEM_STAGES;
                        const bool last_block = kb == seg.k1 - 1, ends_stage = (kb & 1) || last_block;
                        tc_fence_after();
                        if (open && (word & 0x01010101u) != 0u) close_chain(it - 1, (kb - 1) / TC_GROUP_KB, WHOLE, false);
                        const bool first = !open;
                        if (!open && !(ok = open_chain())) break;
                        const uint32_t rare = (word & 0x02020202u) | masks;
                        const uint32_t stage = smem_base + Cfg::A_RING + s * Cfg::A_STAGE_BYTES + (uint32_t)(kb & 1) * (TC_WK * 2);
                        const uint64_t bhi = make_kmajor_sw128_desc(stage), blo = make_kmajor_sw128_desc(stage + TC_A_TILE_BYTES);
                        const uint32_t bhi_lo = (uint32_t)bhi, bhi_hi = (uint32_t)(bhi >> 32), blo_lo = (uint32_t)blo, blo_hi = (uint32_t)(blo >> 32);
                        const uint32_t acc = tmem_base + Cfg::ACC_COL + (w * Cfg::ACC_BUFS + ab) * TC_BM;
                        const uint32_t w_hi = tmem_base + Cfg::OP_COL + t * Cfg::OP_STAGE_COLS + w * Cfg::OP_COLS;
                        // 16 fp16 per k-step: 8 TMEM columns of W, 32 bytes (descriptor units of 16 B) of the activations
                        tc_mma_ts(acc, w_hi, bhi_lo, bhi_hi, idesc, first ? 0u : 1u);
                        if (MODE3X) {
                            tc_mma_ts(acc, w_hi + 8, bhi_lo, bhi_hi, idesc, 1u);
                            tc_mma_ts(acc, w_hi, blo_lo, blo_hi, idesc, 1u);
                        }
                        // Look ahead: make sure the operands of the next block are there BEFORE the last MMAs of this one are
                        // issued.  Issue is back-pressured by the tensor pipe, so once those are in, only the commits stand
                        // between them and the next block's first MMA.
                        uint32_t next_word = 0u, next_masks = masks;
                        if (rare == 0u && !last_block) {
                            ok = wait_block(it + 1, a_it + 1, ends_stage);
                            next_word = block_word(it + 1);
                            if (ends_stage) next_masks = stage_masks(a_it + 1);
                        }
                        tc_mma_ts(acc, w_hi + Cfg::STEP_COLS, bhi_lo + 2, bhi_hi, idesc, 1u);
                        if (MODE3X) {
                            tc_mma_ts(acc, w_hi + 24, bhi_lo + 2, bhi_hi, idesc, 1u);
                            tc_mma_ts(acc, w_hi + 16, blo_lo + 2, blo_hi, idesc, 1u);
                        }
                        if (rare != 0u || last_block || ((kb + 1) & p.chain_mask) == 0) close_chain(it, kb / TC_GROUP_KB, WHOLE, last_block && (word & 0x02020202u) == 0u && (masks >> (16 * (kb & 1)) & 0xffffu) == 0u);
                        if (rare == 0u) {
                            if (ends_stage) {   // the activation stage may be refilled once these MMAs retire
                                tc_commit(aempty_bar(s));
                                ++a_it;
                            }
                            tc_commit(tempty_bar(w, t));   // and the TMEM operand stage rewritten
                        } else {
                            // chains of the left-overs.  Level 0 multiplies the weights' parts with what is left of the
                            // activations, the others what is left of the weights with both.
                            const uint32_t here = masks >> (16 * (kb & 1)) & 0xffffu;
                            uint32_t more = 0u, quarters = 0xfu, wt = w_hi;
                            for (int q = 0; q < 4; ++q) more |= (word >> (8 * q + 1) & 1u) << q;
#pragma unroll 1
                            for (uint32_t level = 0;; ++level) {
                                if (level > 0) {
                                    quarters = more;
                                    more = 0u;
#pragma unroll 1
                                    for (int q = 0; q < 4 && ok; ++q) {
                                        if ((quarters >> q & 1u) == 0u) continue;
                                        ok = mbar_wait(xfull_bar(w, q), xph >> q & 1u, abort_flag, p.status, 18u);
                                        more |= (lds1u(smem_base + Cfg::LEFT_OFF + w * 4) >> (8 * q) & 1u) << q;
                                    }
                                    xph ^= quarters;
                                    if (!ok) break;
                                    tc_fence_after();
                                    wt = tmem_base + Cfg::LEFT_COL + w * Cfg::OP_COLS;
                                }
#pragma unroll 1
                                for (int band = level == 0 ? 1 : 0; band < TC_BANDS; ++band) {
                                    const uint32_t mask = band == 0 ? 0xffu : here >> (8 * (band - 1)) & 0xffu;
                                    if (mask == 0u) break;
                                    ok = (band == 0 || wait_stage(a_it + band)) && open_chain();
                                    if (!ok) break;
                                    constexpr uint32_t idesc16 = make_idesc_f16(TC_BN, TC_SUB);
                                    uint32_t at = (smem_base + Cfg::A_RING + ((a_it + band) % Cfg::A_STAGES) * Cfg::A_STAGE_BYTES + (uint32_t)(kb & 1) * (TC_WK * 2)) >> 4;
                                    uint32_t d = tmem_base + Cfg::ACC_COL + (w * Cfg::ACC_BUFS + ab) * TC_BM;
#pragma unroll 1
                                    for (uint32_t rows = mask; rows != 0u; rows >>= 1, d += TC_SUB, at += TC_SUB * 128 / 16) {
                                        if ((rows & 1u) == 0u) continue;
#pragma unroll 1
                                        for (uint32_t step = 0; step < 2; ++step) {
                                            const uint32_t a = wt + Cfg::STEP_COLS * step, h = (bhi_lo & ~0x3fffu) | (at + 2 * step);
                                            tc_mma_ts(d, a, h, bhi_hi, idesc16, step);
                                            if (MODE3X) {
                                                tc_mma_ts(d, a + 8, h, bhi_hi, idesc16, 1u);
                                                tc_mma_ts(d, a, h + (TC_A_TILE_BYTES >> 4), bhi_hi, idesc16, 1u);
                                            }
                                        }
                                    }
                                    const bool last_band = band == TC_BANDS - 1 || (here >> (8 * band) & 0xffu) == 0u;
                                    close_chain(it, band * p.groups + kb / TC_GROUP_KB, level << 9 | mask << 16 | quarters << 24, last_block && more == 0u && last_band);
                                }
                                if (!ok) break;
                                if (level == 0) {
                                    tc_commit(tempty_bar(w, t));
                                } else {
                                    for (int q = 0; q < 4; ++q)
                                        if (quarters >> q & 1u) tc_commit(xempty_bar(w, q));
                                }
                                if (more == 0u) break;
                            }
                            // The bands' stages may be refilled, too.  Where a run begins or ends inside a stage, its half may have nothing
                            // in a band that the other half has: the copy has to have landed all the same before its slot and its
                            // barrier are given away, or the CTA ends.
                            if (ok && ends_stage)
                                for (uint32_t n = 1u + (masks != 0u) + ((masks & 0xff00ff00u) != 0u); n > 0 && ok; --n, ++a_it)
                                    if ((ok = wait_stage(a_it))) tc_commit(aempty_bar(a_it % Cfg::A_STAGES));
                            if (ok && !last_block) {
                                ok = wait_block(it + 1, a_it, ends_stage);
                                next_word = block_word(it + 1);
                                next_masks = stage_masks(a_it);
                            }
                        }
                        word = next_word;
                        masks = next_masks;
                    }
                }
            }
            __syncwarp();
        }
    } else if (warp < 4 + 4 * NT) {
        // ---------------------------------------------------------------- converter warps, one warpgroup per W tile
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::REGS_CONV));
        const int w = (warp - 4) >> 2;                // W tile of this warpgroup
        const int q = warp & 3;                       // TMEM lane quarter this warp may touch
        const int row = q * 32 + lane;                // row of the W tile = TMEM lane
        const uint32_t dst0 = tmem_base + ((uint32_t)(q * 32) << 16) + Cfg::OP_COL + w * Cfg::OP_COLS;
        TcWalk walk(p);
        TcSeg seg;
        float sc = 1.0f, inv = 1.0f;                  // this row's scale in the open chain
        bool set = false;                             // ... is fixed: the row has had a nonzero element
        uint32_t it = 0;
        bool ok = true;
        // What is left of this warp's rows of a block, 2^38 times the scale, replaces the raw values; its parts go to the left-overs'
        // stage, and once more what those leave.
        uint32_t x_it = 0;
        auto left_overs = [&](uint32_t rowp) {
            const uint32_t dst = tmem_base + ((uint32_t)(q * 32) << 16) + Cfg::LEFT_COL + w * Cfg::OP_COLS;
            bool again = true;
#pragma unroll 1
            for (bool raw = true; again; raw = false, ++x_it) {
                ok = mbar_wait(xempty_bar(w, q), (x_it & 1u) ^ 1u, abort_flag, p.status, 17u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) return;
                tc_fence_after();
                again = false;
#pragma unroll 1
                for (int c = 0; c < 8; ++c) {
                    float4 v = tc_read4<WK>(rowp, c, p.w_shift);
                    uint32_t h[2], l[2];
                    if (raw) {
                        tc_split2_left<MODE3X>(v.x * sc, v.y * sc, h[0], l[0], v.x, v.y);
                        tc_split2_left<MODE3X>(v.z * sc, v.w * sc, h[0], l[0], v.z, v.w);
                    }
                    tc_split2_left<MODE3X>(v.x * TC_LEFT_SCALE, v.y * TC_LEFT_SCALE, h[0], l[0], v.x, v.y);
                    tc_split2_left<MODE3X>(v.z * TC_LEFT_SCALE, v.w * TC_LEFT_SCALE, h[1], l[1], v.z, v.w);
                    tc_write4<WK>(rowp, c, p.w_shift, v);
                    again |= v.x != 0.0f || v.y != 0.0f || v.z != 0.0f || v.w != 0.0f;
                    __syncwarp();
                    const uint32_t at = dst + (c >> 2) * Cfg::STEP_COLS + 2 * (c & 3);
                    tc_st2(at, h[0], h[1]);
                    if (MODE3X) tc_st2(at + 8, l[0], l[1]);
                }
                again = __any_sync(0xffffffffu, again);
                if (lane == 0) sts1b(smem_base + Cfg::LEFT_OFF + w * 4 + q, again ? 1u : 0u);
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(xfull_bar(w, q));
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the slot's next contents come through TMA
            __syncwarp();
        };
        while (ok && walk.next(p, seg)) {
            for (int kb = seg.k0; kb < seg.k1; ++kb, ++it) {
                const int s = it % Cfg::W_STAGES, t = it % Cfg::TMEM_STAGES;
                ok = mbar_wait(wfull_bar(s), (it / Cfg::W_STAGES) & 1u, abort_flag, p.status, 4u) &&
                     mbar_wait(tempty_bar(w, t), ((it / Cfg::TMEM_STAGES) & 1u) ^ 1u, abort_flag, p.status, 5u);
                ok = __all_sync(0xffffffffu, ok);   // the tcgen05 stores below need the whole warp
                if (!ok) break;
                tc_fence_after();
                const uint32_t rowp = tc_row_base<WK>(smem_base + Cfg::W_RING + s * Cfg::W_STAGE_BYTES + w * Cfg::W_TILE_BYTES, row, p.w_shift);
                const bool chain_start = kb == seg.k0 || (kb & p.chain_mask) == 0;
                if (chain_start) set = false;
                if (!set) {
                    // nothing but zeros of this row is in the accumulator: any scale is right for what is there
                    const uint32_t amax = tc_row_amax<WK>(rowp, p.w_shift);
                    tc_scale<TC_W_EXP>(amax, sc, inv);
                    set = amax != 0u && amax < 0x7f800000u;   // (a row that is not finite any more may have any scale, too)
                }
                __syncwarp();
                const uint32_t dst = dst0 + t * Cfg::OP_STAGE_COLS;
                bool grew = false, left = false;
                for (;;) {
                    uint32_t top = 0u, low = 0x7bff7bffu;
                    const uint64_t sc2 = tc_pack2(sc, sc);
#pragma unroll 1
                    for (int step = 0; step < 2; ++step) {
                        uint32_t hl[16];
                        tc_convert_step<MODE3X, WK>(rowp, p.w_shift, step, sc2, hl, top, low);
                        if (MODE3X) tc_st16(dst + step * 16, hl);
                        else        tc_st8(dst + step * Cfg::STEP_COLS, hl);
                    }
                    top &= 0x7fff7fffu;
                    low &= 0x7fff7fffu;
                    const bool over = (top >> 16) >= 0x7c00u || (top & 0xffffu) >= 0x7c00u;
                    const bool small = set && ((low >> 16) < tc_safe_f16<MODE3X>() || (low & 0xffffu) < tc_safe_f16<MODE3X>());
                    if (!__any_sync(0xffffffffu, over || small)) break;
                    if (!grew && __any_sync(0xffffffffu, over)) {
                        // rare: a row's magnitudes grew more than fourfold since its chain began: new scale, and once more
                        grew = true;
                        if (over) {
                            const uint32_t amax = tc_row_amax<WK>(rowp, p.w_shift);
                            tc_scale<TC_W_EXP>(amax, sc, inv);
                            set = amax < 0x7f800000u;
                        }
                        tc_wait_st();
                        __syncwarp();
                        continue;
                    }
                    // zeros, or elements too small for this scale
                    left = __any_sync(0xffffffffu, small && tc_row_left<MODE3X, WK>(rowp, p.w_shift, sc));
                    break;
                }
                sts1(smem_base + Cfg::WS_OFF + (((it % Cfg::WS_SLOTS) * NT + w) * TC_BN + row) * 4, inv);
                if (lane == 0) sts1b(smem_base + Cfg::BRK_OFF + (t * NT + w) * 4 + q, (grew && !chain_start ? 1u : 0u) | (left ? 2u : 0u));
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tfull_bar(w, t));
                if (left) left_overs(rowp);
                if (lane == 0) mbar_arrive(wempty_bar(s));   // the raw block now lives in TMEM: its ring slot may be refilled
            }
        }
        // the last operand stages' releases must have arrived before the CTA may exit
        for (uint32_t i = it > Cfg::TMEM_STAGES ? it - Cfg::TMEM_STAGES : 0; i < it && ok; ++i)
            ok = mbar_wait(tempty_bar(w, i % Cfg::TMEM_STAGES), (i / Cfg::TMEM_STAGES) & 1u, abort_flag, p.status, 13u);
    } else {
        // ---------------------------------------------------------------- drain + epilogue warps, one warpgroup per W tile
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::REGS_DRAIN));
        const int w = (warp - 4 - 4 * NT) >> 2;       // W tile of this warpgroup
        const int q = warp & 3;
        const int row = q * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        TcWalk walk(p);
        TcSeg seg;
        cn_pdl_wait();
        uint32_t chains = 0;
        bool ok = true;
        while (ok && walk.next(p, seg)) {
            const float *a_inv = p.a_inv + (int64_t)(seg.tile % p.tiles_m) * TC_BM + row;
            uint64_t sum[TC_BM / 2];   // pairs of rows
#pragma unroll
            for (int i = 0; i < TC_BM / 2; ++i) sum[i] = 0ull;
            // the inverse scales of the activation rows: thread `row` fetches row m0 + row of the group it expects next
            int have = seg.k0 / TC_GROUP_KB;   // scales: band * groups + group
            float my_inv = a_inv[have * p.m_pad];
            for (bool last = false; !last; ++chains) {
                const int ab = chains % Cfg::ACC_BUFS;
                ok = mbar_wait<TC_DRAIN_SLEEP_NS>(accfull_bar(w, ab), (chains / Cfg::ACC_BUFS) & 1u, abort_flag, p.status, 6u);
                {   // all 128 threads of the warpgroup go on together or not at all
                    uint32_t all_ok;
                    asm volatile(
                        "{\n\t.reg .pred pi, po;\n\t"
                        "setp.ne.u32 pi, %1, 0;\n\t"
                        "bar.red.and.pred po, %2, 128, pi;\n\t"
                        "selp.u32 %0, 1, 0, po;\n\t}"
                        : "=r"(all_ok) : "r"((uint32_t)ok), "r"(1 + w) : "memory");
                    ok = all_ok != 0;
                }
                if (!ok) break;
                tc_fence_after();
                const uint32_t what = lds1u(smem_base + Cfg::INFO_OFF + (w * Cfg::ACC_BUFS + ab) * 8);
                const int scales = (int)lds1u(smem_base + Cfg::INFO_OFF + (w * Cfg::ACC_BUFS + ab) * 8 + 4);
                last = (what & 0x100u) != 0u;
                if (scales != have) my_inv = a_inv[scales * p.m_pad];
                const uint32_t as = smem_base + Cfg::AS_OFF + ((chains & 1u) * NT + w) * (TC_BM * 4);
                sts1(as + row * 4, my_inv);
                float wi = lds1(smem_base + Cfg::WS_OFF + (((what & 0xffu) * NT + w) * TC_BN + row) * 4);
                for (uint32_t level = what >> 9 & 7u; level > 0; --level) wi *= 1.0f / TC_LEFT_SCALE;
                asm volatile("bar.sync %0, 128;" ::"r"(1 + w) : "memory");
                have = scales;
                if (!last && scales < (seg.k1 - 1) / TC_GROUP_KB) {   // most likely the next chain's group
                    have = scales + 1;
                    my_inv = a_inv[have * p.m_pad];
                }
                const uint32_t src = tmem_base + lane_addr + Cfg::ACC_COL + (w * Cfg::ACC_BUFS + ab) * TC_BM;
                // Remove both scales and add.  (The product of the two inverse scales is finite unless the product of the segment's
                // largest magnitudes is beyond fp32's range by 2^27.)
                const uint64_t wi2 = tc_pack2(wi, wi);
                auto add16 = [&](int cc) {
                    uint32_t r[16];
                    tc_ld16(src + cc * 16, r);
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const float4 f = lds4(as + (cc * 16 + i) * 4);
                        uint64_t &s0 = sum[(cc * 16 + i) / 2], &s1 = sum[(cc * 16 + i) / 2 + 1];
                        s0 = tc_fma2(tc_pack2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), tc_mul2(tc_pack2(f.x, f.y), wi2), s0);
                        s1 = tc_fma2(tc_pack2(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])), tc_mul2(tc_pack2(f.z, f.w), wi2), s1);
                    }
                };
                if ((what & 0x00ff0e00u) == 0x00ff0000u) {
#pragma unroll
                    for (int cc = 0; cc < TC_BM / TC_SUB; ++cc) add16(cc);
                } else {
                    // left-overs: the blocks of 16 rows m, and the quarters of the rows n, that have some
                    uint32_t mask = (what >> (24 + q) & 1u) ? what >> 16 & 0xffu : 0u;
#pragma unroll
                    for (int cc = 0; cc < TC_BM / TC_SUB; ++cc) {
                        const bool in_chain = (mask & 1u) != 0u;
                        asm volatile("shr.u32 %0, %0, 1;" : "+r"(mask));   // one test at a time: eight predicates held together are too many
                        if (in_chain) add16(cc);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(accempty_bar(w, ab));
            }
            if (!ok) break;
            const int64_t m0 = (int64_t)(seg.tile % p.tiles_m) * TC_BM, n = (int64_t)(seg.tile / p.tiles_m) * (NT * TC_BN) + w * TC_BN + row;
            if (SHARED) {
                // The rings are idle in every CTA of the cluster: each unit of 16 rows goes to the CTA that finishes it, [sender][quad of m][column n]
                // float4, which adds the parts in K order.  A lane's own share stays where it is, and it reads what it wrote itself.
                cluster_arrive();
                cluster_wait();
                chains = ~0u;   // done
                const TcShare share(p);
                const int per = share.per, rank = share.rank, mine = share.mine;
                constexpr uint32_t QUAD = NT * TC_BN * 16;
                const uint32_t column = (uint32_t)(w * TC_BN + row) * 16u;
                int to = 0, at_unit = 0;
#pragma unroll
                for (int u = 0; u < TC_BM / 16; ++u) {
                    if (u >= share.units) break;
                    const uint32_t at = smem_base + (uint32_t)((rank * per + at_unit) * 4) * QUAD + column;
                    if (to == rank) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) sts2l(at + j * QUAD, sum[8 * u + 2 * j], sum[8 * u + 2 * j + 1]);
                    } else {
                        const uint32_t there = in_cta(at, to), counted = in_cta(bar(B_PART), to);
#pragma unroll
                        for (int j = 0; j < 4; ++j) st_async2(there + j * QUAD, counted, sum[8 * u + 2 * j], sum[8 * u + 2 * j + 1]);
                    }
                    if (++at_unit == per) { at_unit = 0; ++to; }
                }
                if (mine <= 0) break;
                ok = mbar_wait(bar(B_PART), 0u, abort_flag, p.status, 24u) && mbar_try_cluster(bar(B_PART), 0u) != 0u;
                if (!ok) break;
                if (n >= p.N) break;
                const float bias = p.bias ? p.bias[n] : 0.0f;
                const bool vec = (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15u) == 0;
                int64_t m = m0 + 16 * (rank * per);
                float *q = p.C + n * p.ldc + m;
#pragma unroll 1
                for (int i = 0; i < 4 * mine && m < p.M; ++i, m += 4, q += 4) {
                    float4 part[CN_TC_MAX_CLUSTER];
#pragma unroll
                    for (int s = 0; s < CN_TC_MAX_CLUSTER; ++s)
                        if (s < p.cluster) part[s] = lds4(smem_base + (uint32_t)(s * per * 4 + i) * QUAD + column);
                    float v[4] = {part[0].x, part[0].y, part[0].z, part[0].w};
#pragma unroll
                    for (int s = 1; s < CN_TC_MAX_CLUSTER; ++s)
                        if (s < p.cluster) { v[0] += part[s].x; v[1] += part[s].y; v[2] += part[s].z; v[3] += part[s].w; }
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = cn_apply_activation(p.bias ? v[e] + bias : v[e], p.act);
                    if (vec && m + 4 <= p.M) {
                        *reinterpret_cast<float4 *>(q) = make_float4(v[0], v[1], v[2], v[3]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (m + e < p.M) q[e] = v[e];
                    }
                }
                break;
            }
            if (seg.slot >= 0) {
                // Partial tile: float4 number i of 32 for all 128 columns, then the next, so that a warp writes 512 contiguous bytes.  Rows that
                // do not exist are neither written nor read: 20 x 9000 . 9000 x 4000 48.4 -> 43.8 us (46.7 where only the reduction leaves
                // them), 203 x 4001 . 4001 x 3001 47.2 -> 46.0.  Leaving them out of the multiplication and the sums, too, cost full tiles 2 %.
                const int64_t rows = p.M - m0;
                ulonglong2 *P = reinterpret_cast<ulonglong2 *>(p.partials) + ((int64_t)seg.slot * NT + w) * (TC_BM * TC_BN / 4) + row;
#pragma unroll
                for (int i = 0; i < TC_BM / 4; ++i)
                    if (i * 4 < rows) P[i * TC_BN] = make_ulonglong2(sum[2 * i], sum[2 * i + 1]);
                continue;
            }
            const int L = p.maxout_level;
            const float bias = (p.bias && n < p.N) ? p.bias[n] : 0.0f;
            float *dst = p.C + n * p.ldc + m0;
            if (L <= 1) {
                // every lane writes a column of its own: 32 bytes at a time fill whole sectors of L2, 16 half of one.  Product of
                // 4096^3 alone: 475 us with 16-byte stores, 455 us with these.
                // Rows beyond M are left out, and the logistic function, whose code is long, has a copy of the loop to itself: a pass
                // through the other one is 128 additions and 16 stores, not a walk over 128 branches around it (16 x 248 . 248 x 35720 with
                // logistic units: 36 us, 20 now; linear ones of 128 rows 27, 22).
                const uintptr_t at = reinterpret_cast<uintptr_t>(dst);
                const bool whole = m0 + TC_BM <= p.M, vec8 = whole && (at & 31u) == 0, vec4 = whole && (at & 15u) == 0;
                auto store8 = [&](int i, const float (&v)[8]) {
                    if (n >= p.N) return;
                    if (vec8) {
                        stg8(dst + i, v);
                    } else if (vec4) {
                        *reinterpret_cast<float4 *>(dst + i) = make_float4(v[0], v[1], v[2], v[3]);
                        *reinterpret_cast<float4 *>(dst + i + 4) = make_float4(v[4], v[5], v[6], v[7]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (m0 + i + e < p.M) dst[i + e] = v[e];
                    }
                };
                if (p.act == CN_ACT_LOGISTIC) {
#pragma unroll
                    for (int i = 0; i < TC_BM; i += 8) {
                        if (m0 + i >= p.M) break;
                        float v[8];
#pragma unroll
                        for (int e = 0; e < 8; e += 2) tc_unpack2(sum[(i + e) / 2], v[e], v[e + 1]);
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] = cn_apply_activation(p.bias ? v[e] + bias : v[e], CN_ACT_LOGISTIC);
                        store8(i, v);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < TC_BM; i += 8) {
                        if (m0 + i >= p.M) break;
                        float v[8];
#pragma unroll
                        for (int e = 0; e < 8; e += 2) tc_unpack2(sum[(i + e) / 2], v[e], v[e + 1]);
                        if (p.bias) {
#pragma unroll
                            for (int e = 0; e < 8; ++e) v[e] += bias;
                        }
                        if (p.act != CN_ACT_LINEAR) {
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                v[e] = v[e] > 0.0f ? v[e] : 0.0f;
                                if (p.act == CN_ACT_DOUBLE_RELU) v[e] = v[e] < 1.0f ? v[e] : 1.0f;
                            }
                        }
                        store8(i, v);
                    }
                }
                __syncwarp();   // the next tile's tensor-memory loads need the whole warp
                continue;
            }
#pragma unroll
            for (int i = 0; i < TC_BM; i += 4) {
                float v[4];
                tc_unpack2(sum[i / 2], v[0], v[1]);
                tc_unpack2(sum[i / 2 + 1], v[2], v[3]);
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = cn_apply_activation(p.bias ? v[e] + bias : v[e], p.act);
                // maxout over L consecutive columns = L adjacent lanes (L is a power of two <= 32).
                // Same comparison tree as the reference's 32-slot reduction: at offsets L/2 .. 1 slot t
                // takes slot t+offset when strictly smaller; larger offsets only meet -FLT_MAX padding.
                const int tl = lane & (L - 1);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float val = v[e], idx = (float)n;
                    for (int off = L >> 1; off > 0; off >>= 1) {
                        const float ov = __shfl_down_sync(0xffffffffu, val, off, L);
                        const float oi = __shfl_down_sync(0xffffffffu, idx, off, L);
                        if (tl < off && val < ov) { val = ov; idx = oi; }
                    }
                    if (tl == 0 && n < p.N && m0 + i + e < p.M) {
                        const int64_t g = n / L;
                        p.C[g * p.ldc + m0 + i + e] = val;
                        if (p.argmax) p.argmax[g * p.ldc + m0 + i + e] = idx;
                    }
                }
            }
            __syncwarp();   // as above
        }
        __syncwarp();
        if (SHARED && chains != ~0u) { cluster_arrive(); cluster_wait(); }   // gave up before
    }
    if (SHARED && warp < 4 + 4 * NT) {   // this CTA's loads and products are over, once all warps say so
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    }

    tc_fence_before();
    __syncthreads();
    if (SHARED) {
        // no CTA leaves before the others have sent; after a wait that ran out, what is under way gets a bounded chance to land
        if (lds1u(abort_flag) != 0u) {
            const long long t0 = clock64();
            while (clock64() - t0 < 20000000LL) {}
        }
        __syncwarp();
        cluster_arrive_relaxed();
        cluster_wait();
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ------------------------------------------------------------------------------------------ reduction of the runs
// One CTA per COLS columns of one W tile: adds the partial tiles of all runs in K order (a fixed order, so the result does not
// depend on scheduling), applies bias and activation, turns the block through shared memory so that a warp stores 512
// contiguous bytes of a column, and stores to C and, for the fused all-gather, to every peer's C (full NVLink packets).
//
// Few tiles, and tiles that are cut into many runs, are bound by how many loads are in flight: 8 columns per CTA, eight partial tiles at a time,
// where 32 would leave SMs without a CTA, and from three CTAs per tile on; else 32.  us of the whole product, 32 columns / 8: 203 x 4001 . 4001 x 3001
// (six CTAs per tile) 50.5 / 44.7, 500 x 3000 . 3000 x 3000 (three) 59.5 / 56.1; 2304 x 512 . 512 x 2304 (seven tiles of 256 x 256 by 18 pairs) 43.4 /
// 40.1, 4850 x 512 . 512 x 1024 (two by five) 48.2 / 44.5; 300 x 6000 . 6000 x 6000 (72 by two CTAs each) 117.6 / 120.1, 1000 x 4096 . 4096 x 2048 (32 by two
// pairs each) 71 / 73.6.
template <int COLS>
__global__ void __launch_bounds__(256)
cn_splitk_reduce_kernel(const __grid_constant__ ReduceParams p)
{
    constexpr int QSTEP = 256 / COLS, QUADS = 32 / QSTEP, UNROLL = 8 / QUADS;   // quads of m per thread; partial tiles in flight
    __shared__ float turn[COLS][TC_BM + 4];
    cn_pdl_launch_dependents();
    // where this CTA's partial tiles are, worked out (divisions of 64 bits) while the product still runs
    const int chunk = blockIdx.x % (TC_BN / COLS);
    const int tw = blockIdx.x / (TC_BN / COLS), rm = tw / p.nt, w = tw - rm * p.nt, r = rm / p.mt, mh = rm - r * p.mt, tile = p.full_tiles + r;
    const int64_t m0 = ((int64_t)(tile % p.tiles_m) * p.mt + mh) * p.rows, n0 = ((int64_t)(tile / p.tiles_m) * p.nt + w) * TC_BN + chunk * COLS;
    // the CTAs whose runs hold K blocks of this tile: run c is [total c / ctas, total (c + 1) / ctas)
    const int64_t total = (int64_t)p.tail_tiles * p.kb_total, first = (int64_t)r * p.kb_total, last = first + p.kb_total - 1;
    auto owner = [&](int64_t x) {
        int64_t c = x * p.tail_ctas / total;
        while (total * (c + 1) / p.tail_ctas <= x) ++c;
        while (total * c / p.tail_ctas > x) --c;
        return c;
    };
    const int64_t c0 = owner(first), c1 = owner(last);
    cn_pdl_wait();
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
        __syncthreads();
    }
    if (p.cond && !__syncthreads_or(threadIdx.x == 0 && __ldcg(p.cond) != 0u)) return;
    if (n0 >= p.N || m0 >= p.M) return;
    const int row = threadIdx.x % COLS, quad = threadIdx.x / COLS;   // column of the chunk; quads of m: quad + QSTEP j
    constexpr int64_t TILE4 = TC_BM * TC_BN / 4;
    const float4 *src = reinterpret_cast<const float4 *>(p.partials) + (((c0 + r) * p.mt + mh) * p.nt + w) * TILE4 + quad * TC_BN + chunk * COLS + row;
    const int64_t step = p.mt * p.nt * TILE4;
    float4 acc[QUADS];
#pragma unroll
    for (int j = 0; j < QUADS; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    // Rows that do not exist have not been written.  Reading what memory holds in their place cost more than reading what had just been written: 192 x
    // 1048 . 1048 x 10532 44.7 us as long as they were written, 45.0 read all the same, 42.6 left alone.
    int64_t left = m0 + quad * 4 < p.M ? c1 - c0 + 1 : 0;
    const int quads = QUADS == 1 || p.M - m0 >= TC_BM ? QUADS : (int)(p.M - m0 - quad * 4 + 4 * QSTEP - 1) / (4 * QSTEP);   // of this thread, that exist
    // the additions stay in K order, so the sum does not depend on the grouping; what is left of a group is loaded together, too
    for (; left > 0; left -= UNROLL, src += UNROLL * step) {
        float4 v[UNROLL][QUADS];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u)
#pragma unroll
            for (int j = 0; j < QUADS; ++j)
                if (u < left && (QUADS == 1 || j < quads)) v[u][j] = __ldcs(src + u * step + j * QSTEP * TC_BN);
#pragma unroll
        for (int u = 0; u < UNROLL; ++u)
#pragma unroll
            for (int j = 0; j < QUADS; ++j)
                if (u < left && (QUADS == 1 || j < quads)) { acc[j].x += v[u][j].x; acc[j].y += v[u][j].y; acc[j].z += v[u][j].z; acc[j].w += v[u][j].w; }
    }
#pragma unroll
    for (int j = 0; j < QUADS; ++j) *reinterpret_cast<float4 *>(&turn[row][(quad + QSTEP * j) * 4]) = acc[j];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t m = m0 + lane * 4;
    const bool vec = (m + 4 <= p.M) && ((p.ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15u) == 0);
#pragma unroll
    for (int j = 0; j < COLS / 8; ++j) {
        const int nl = (threadIdx.x >> 5) + 8 * j;
        const int64_t n = n0 + nl;
        if (n >= p.N || m >= p.M || lane * 4 >= p.rows) continue;
        const float b = p.bias ? p.bias[n] : 0.0f;
        const float4 a = *reinterpret_cast<const float4 *>(&turn[nl][lane * 4]);
        float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = cn_apply_activation(p.bias ? v[i] + b : v[i], p.act);
        const int64_t off = n * p.ldc + m;
        for (int d = 0; d <= p.npeers; ++d) {
            float *dst = (d == 0 ? p.C : p.peerC[d - 1]) + off;
            if (vec) {
                *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (m + i < p.M) dst[i] = v[i];
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------------ host
int cn_splitk_reduce_launch(cn_context *ctx, const ReduceParams &rp, cudaStream_t s)
{
    const int64_t blocks = (int64_t)rp.tail_tiles * rp.nt * rp.mt;
    if (rp.tail_ctas >= 3LL * rp.tail_tiles || blocks * 4 <= ctx->sm_count) CN_CUDA(cn_launch_pdl(cn_splitk_reduce_kernel<8>, dim3((unsigned)(blocks * (TC_BN / 8))), 256, 0, s, rp));
    else CN_CUDA(cn_launch_pdl(cn_splitk_reduce_kernel<32>, dim3((unsigned)(blocks * (TC_BN / 32))), 256, 0, s, rp));
    cn_count_launch();
    return CN_OK;
}

int cn_get_encode_fn(cn_context *ctx, EncodeTiledFn *out)
{
    if (!ctx->gemm) ctx->gemm = cn_gemm_workspace_new();
    if (!ctx->gemm->encode_fn) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        CN_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
        CN_REQUIRE(fn && qres == cudaDriverEntryPointSuccess, CN_ERR_CUDA, "cuTensorMapEncodeTiled is not available in this driver");
        ctx->gemm->encode_fn = fn;
    }
    *out = (EncodeTiledFn)ctx->gemm->encode_fn;
    return CN_OK;
}

// Weight map: fp32, inner extent `inner`, outer extent `outer`, row pitch in elements, box in elements.  The 128-byte swizzle for
// 128-byte box rows that the converters read in 16-byte chunks (W_K), none otherwise.
static int make_w_map(EncodeTiledFn enc, CUtensorMap *map, const float *base, int64_t inner, int64_t outer, int64_t pitch, int box_inner, int box_outer,
                      bool swizzle)
{
    cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
    cuuint64_t strides[1] = {(cuuint64_t)pitch * sizeof(float)};
    cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CN_REQUIRE(r == CUDA_SUCCESS, CN_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d (inner %lld outer %lld pitch %lld)", (int)r,
               (long long)inner, (long long)outer, (long long)pitch);
    return CN_OK;
}

// The maps of a stored matrix of `outer` rows of `inner` elements, and the offsets of the classes of rows.
static int make_w_maps(EncodeTiledFn enc, WMaps *m, uint32_t *shift, const float *base, int64_t inner, int64_t outer, int64_t pitch, int wk)
{
    const bool n_inner = wk == W_N || wk == W_N_ANY;
    const int box_inner = n_inner ? TC_BN : TC_WK, box_outer = n_inner ? TC_WK : TC_BN;
    *shift = 0;
    if (!w_any(wk)) {
        int st = make_w_map(enc, &m->map[0], base, inner, outer, pitch, box_inner, box_outer, wk == W_K);
        for (int r = 1; r < TC_CLASSES; ++r) m->map[r] = m->map[0];
        return st;
    }
    for (int r = 0; r < TC_CLASSES; ++r) {
        const uintptr_t row = reinterpret_cast<uintptr_t>(base + r * pitch);
        const int64_t d = (int64_t)((row & 15u) / sizeof(float));
        int st = make_w_map(enc, &m->map[r], reinterpret_cast<const float *>(row & ~(uintptr_t)15), inner + d, (outer - r + TC_CLASSES - 1) / TC_CLASSES,
                            pitch * TC_CLASSES, box_inner + 4, box_outer / TC_CLASSES, false);
        if (st != CN_OK) return st;
        *shift |= (uint32_t)d << (8 * r);
    }
    return CN_OK;
}

bool cn_gemm_tc_can_fuse_maxout(int L) { return L == 2 || L == 4 || L == 8 || L == 16 || L == 32; }

// Rows that TMA can read as they are.
static bool w_aligned(const float *B, int64_t ldb) { return (ldb & 3) == 0 && (reinterpret_cast<uintptr_t>(B) & 15u) == 0; }

// short dimensions are zero-filled by TMA up to the tile; its coordinates are 32-bit
static bool tc_dims(int64_t M, int64_t N, int64_t K)
{
    return M >= 1 && N >= 1 && K >= 1 && K < (1LL << 31) - 64 && N < (1LL << 31) - 256 && M < (1LL << 31) - 256;
}

bool cn_gemm_tc_any_supported(int transB, int64_t M, int64_t N, int64_t K, const float *B)
{
    if ((transB ? K : N) < TC_CLASSES) return false;   // every class of rows has at least one
    return tc_dims(M, N, K) && (reinterpret_cast<uintptr_t>(B) & 3u) == 0;
}

bool cn_gemm_tc_supported(cn_context *, int transA, int transB, int64_t M, int64_t N, int64_t K, const float *,
                          int64_t, const float *B, int64_t ldb, const float *, int64_t)
{
    (void)transA;   // a transposed activation operand only changes the pre-pass
    (void)transB;   // a transposed weight only changes the TMA box and the converter's read pattern
    return tc_dims(M, N, K) && w_aligned(B, ldb);
}

// K blocks per accumulation chain for weights of any pitch.  They were multiplied on the fp32 kernel before, whose error grows with
// the square root of K: relative to an fp64 product (uniform operands) 2.1e-7 at K = 130, 5.0e-7 at 785, 1.13e-6 at 4001, 3.6e-6 at
// 39999.  Here it grows with the chain: 2.1e-7 with one block, 3.2e-7 with 2, 5.2e-7 with 4, 9.0e-7 with 8, 1.8e-6 with 16.  The
// longest chain that is no less exact than the fp32 kernel was:
int cn_gemm_any_chain(int64_t K) { return K < 384 ? 1 : K < 1024 ? 2 : K < 3072 ? 4 : K < 12288 ? 8 : TC_GROUP_KB; }

template <class Kernel>
static cudaError_t tc_launch_clusters(Kernel kernel, unsigned grid, int cluster, int block, size_t smem, cudaStream_t s, const WMaps &mw, const CUtensorMap &ma,
                                      const TcParams &prm)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, mw, ma, prm);
}

// Clusters of c CTAs of an SM each that the device holds at once: their SMs have to lie in one GPC.
static int tc_max_clusters(const cn_context *ctx, int c)
{
    using Cfg = TcCfg<2, true, W_K>;
    static int known[64][CN_TC_MAX_CLUSTER + 1] = {};
    const int dev = ctx->device;
    if (dev >= 0 && dev < 64 && known[dev][c] > 0) return known[dev][c];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ctx->sm_count / c * c));
    cfg.blockDim = dim3(Cfg::THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(cn_gemm_tc_kernel<2, true, W_K, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, cn_gemm_tc_kernel<2, true, W_K, true>, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = 1;
    }
    if (dev >= 0 && dev < 64) known[dev][c] = n;
    return n;
}

template <int NT, bool MODE3X, int WK, bool SHARED>
static int launch_cfg(const WMaps &mw, const CUtensorMap &ma, const TcParams &prm, int64_t grid, int dev, cudaStream_t s)
{
    using Cfg = TcCfg<NT, MODE3X, WK>;
    static bool attr_set[64] = {};   // per device: the attribute belongs to the device's copy of the function
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        CN_CUDA(cudaFuncSetAttribute(cn_gemm_tc_kernel<NT, MODE3X, WK, SHARED>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    if (SHARED) CN_CUDA(tc_launch_clusters(cn_gemm_tc_kernel<NT, MODE3X, WK, SHARED>, (unsigned)grid, prm.cluster, Cfg::THREADS, Cfg::SMEM_BYTES, s, mw, ma, prm));
    else CN_CUDA(cn_launch_pdl(cn_gemm_tc_kernel<NT, MODE3X, WK, SHARED>, dim3((unsigned)grid), Cfg::THREADS, Cfg::SMEM_BYTES, s, mw, ma, prm));
    cn_count_launch();
    return CN_OK;
}

size_t cn_tc_cut::partial_bytes() const { return rest() > 0 && cluster == 1 ? (size_t)(tail_ctas + rest()) * nt * TC_BM * TC_BN * sizeof(float) : 0; }

// Clusters in place of runs that leave partial tiles, for products of one tile of rows.  A run's partial tiles go to memory and a reduction reads
// them, a launch later: 17 us, 8 more where all SMs leave some, and 0.9 per K block of a CTA for the whole product, by a fit to what
// follows.  A cluster's CTAs exchange the parts through distributed shared memory (20 bytes per clock from a CTA), in one launch less: 15 us
// and 0.66 per block with one tile of 128 columns per CTA, 20 and 0.74 with two; but K is cut into as many parts as CTAs find room in the GPCs
// for every tile, not one per SM.  us, runs / clusters: 24 x 560 . 560 x 5192 23.8 / 14.5; 100 x 1500 . 1500 x 2500 30.6 / 19.6; 48 x 1568 . 1568 x 11448 39.4
// / 28.7; 128 x 2348 . 2348 x 8289 40.4 / 38.5; 128 x 100000 . 100000 x 1000 131 / 299.  With two tiles of rows a few gain (256 x 4096 . 4096 x 4096 55.5 /
// 49.7), others lose (150 x 2344 . 2344 x 2208 33 / 38).  The fit is older than the reduction's CTAs of eight columns and than
// runs that leave out rows which do not exist: of 238 products drawn where this rule takes clusters, which take 0.94 of the runs' time on average,
// 70 are more than 3 % faster by runs today, 54 of them among the 102 of up to 32 rows (32 x 3888 . 3888 x 3000 23.7 / 30.3 the worst of them).
//
// Runs are short, and so are their accumulation chains; clusters' chains are cut as short, so that no product is less exact: relative to fp64,
// runs of 28 blocks 1.6e-6, of 14 1.3e-6, of 6 7e-7; chains of 8 blocks 9.8e-7, of 4 5.4e-7.  That costs long runs more than the launch
// (25 blocks per CTA, 128 x 6400 . 6400 x 448 23.2 / 30.0; 32, 128 x 4064 . 4064 x 6702 47.6 / 51.1): at most 24 blocks.
static void tc_share_tiles(const cn_context *ctx, int64_t N, cn_tc_cut *cut)
{
    if (cut->rest() == 0 || cut->full > 0 || cut->tiles_m > 1) return;   // with whole tiles besides, no two CTAs per tile find room
    const double run = (double)cut->rest() * cut->kb_total / cut->tail_ctas;
    const double runs = 17.0 + 8.0 * (double)cut->tail_ctas / ctx->sm_count + 0.9 * run;
    double best = 0.95 * runs;
    for (int nt = 1; nt <= (N > TC_BN ? 2 : 1); ++nt) {
        const int64_t tiles = (N + nt * TC_BN - 1) / (nt * TC_BN);
        for (int c = 2; c <= CN_TC_MAX_CLUSTER && cut->kb_total >= 2 * c; ++c) {
            const int per = (TC_BM / 16 + c - 1) / c;
            // room for the parts in the rings' shared memory
            if (c * per * 16 * nt * TC_BN * (int)sizeof(float) > (nt == 1 ? TcCfg<1, true, W_K>::RING_BYTES : TcCfg<2, true, W_K>::RING_BYTES)) continue;
            const double t = (nt == 1 ? 15.0 : 20.0) + (nt == 1 ? 0.66 : 0.74) * (double)((cut->kb_total + c - 1) / c);
            if (t >= best || (cut->kb_total + c - 1) / c > 24 || tiles > tc_max_clusters(ctx, c)) continue;
            best = t;
            cut->nt = nt;
            cut->cluster = c;
        }
    }
    if (cut->cluster == 1) return;
    cut->tiles = (N + cut->nt * TC_BN - 1) / (cut->nt * TC_BN);
    cut->tail_ctas = cut->tiles * cut->cluster;
    cut->max_chain = run >= 12.0 ? 8 : run >= 6.0 ? 4 : 2;
}

cn_tc_cut cn_tc_decompose(const cn_context *ctx, int64_t M, int64_t N, int64_t K, int kind, bool push)
{
    const cn_gemm_workspace *ws = ctx->gemm;
    cn_tc_cut c;
    c.nt = N > TC_BN ? 2 : 1;
    if (ws && (ws->force_nt == 1 || ws->force_nt == 2)) c.nt = ws->force_nt;
    const int64_t tiles_n = (N + c.nt * TC_BN - 1) / (c.nt * TC_BN);
    c.tiles_m = (M + TC_BM - 1) / TC_BM;
    c.tiles = tiles_n * c.tiles_m;
    c.kb_total = (int)((K + TC_WK - 1) / TC_WK);
    const int64_t sms = ctx->sm_count;
    c.full = c.tail_ctas = 0;
    c.cluster = 1;
    c.max_chain = TC_GROUP_KB;
    if (kind == CN_TC_WHOLE) {
        c.full = c.tiles;   // the reduction kernel has no maxout; such layers are small
    } else if (ws && ws->force_splits >= 1) {
        const int64_t splits = ws->force_splits <= c.kb_total ? ws->force_splits : c.kb_total;
        if (splits == 1 && !push) c.full = c.tiles; else c.tail_ctas = c.tiles * splits;
    } else {
        // Whole tiles only, where the last round over the SMs is nearly full or cutting it would cost more than it saves: the
        // reduction of a cut tail takes as long as about 12 K blocks of a CTA (8 us).  Peers take their tiles from the reduction.
        // Behind the planes kernel the reduction is one more launch in every product (600 x 4000 . 4000 x 4096: 73 us, 76 with it; 1023 x
        // 33200 . 33200 x 1659 in the single pass 273, 286), for the few whose lists overflow: only where those would take more than four
        // times as long without it.
        const int64_t rounds = (c.tiles + sms - 1) / sms, even = c.tiles * c.kb_total / sms + 12;
        if (!push && rounds * c.kb_total <= (kind == CN_TC_BEHIND ? 4 * even : even)) {
            c.full = c.tiles;
        } else {
            c.full = push ? 0 : c.tiles / sms * sms;
            c.tail_ctas = c.rest() * c.kb_total / 6;   // at least six K blocks per CTA: shorter runs cost more in partial tiles than they save
            if (c.tail_ctas > sms) c.tail_ctas = sms;
            if (c.tail_ctas < c.rest()) c.tail_ctas = c.rest() < sms ? c.rest() : sms;
        }
    }
    if (kind == CN_TC_CLUSTERS && !push) tc_share_tiles(ctx, N, &c);
    return c;
}

int cn_gemm_tc_launch(cn_context *ctx, int64_t M, int64_t N, int64_t K, const float *A, int64_t lda, const float *B,
                      int64_t ldb, float *C, int64_t ldc, const cn_epilogue *epi, int mode, cudaStream_t s, const cn_peer_out *peers,
                      int transA, int transB, const cn_tc_cond *cond, bool clusters)
{
    EncodeTiledFn enc = nullptr;
    int st = cn_get_encode_fn(ctx, &enc);
    if (st != CN_OK) return st;
    cn_gemm_workspace *ws = ctx->gemm;
    {
        unsigned int *d_status = nullptr;
        if ((st = cn_status_block(ctx, &d_status)) != CN_OK) return st;
    }
    const bool mode3x = mode == CN_GEMM_3XTF32;
    CN_REQUIRE(mode3x || w_aligned(B, ldb), CN_ERR_UNSUPPORTED, "cn_gemm_f32: weights of any alignment take the 3x mode");

    // 1. activations -> K-major hi / lo planes (made here, or ahead of the call by cn_gemm_prepare)
    cn_planes pl;
    cn_plane_layout(M, K, mode, &pl);
    uint8_t *planes = nullptr;
    const bool ahead = ws->prepared != nullptr;
    if (cond) {
        planes = (uint8_t *)cond->planes;
    } else if (ahead) {
        const cn_prepared *pr = ws->prepared;
        ws->prepared = nullptr;
        CN_REQUIRE(pr->filled && pr->M == M && pr->K == K && pr->mode == mode, CN_ERR_SHAPE,
                   "prepared activations are %lld x %lld for mode %d, the product wants %lld x %lld for mode %d", (long long)pr->M,
                   (long long)pr->K, pr->mode, (long long)M, (long long)K, mode);
        planes = (uint8_t *)pr->planes;
    } else {
        void *buf = nullptr;
        if ((st = cn_gemm_scratch(ctx, CN_GEMM_SLOT_ASPLIT, pl.bytes, &buf)) != CN_OK) return st;
        planes = (uint8_t *)buf;
        const cn_coded_src *cs = ws->coded_src;
        ws->coded_src = nullptr;
        CN_REQUIRE(!cs || (!transA && lda == M), CN_ERR_UNSUPPORTED, "coded activations must be untransposed with ld = rows");
        if ((st = cn_make_planes(ctx, transA != 0, M, K, A, lda, cs, pl, planes, s)) != CN_OK) return st;
    }

    // 2. work decomposition
    const int maxout = epi ? epi->maxout_level : 1;
    const cn_tc_cut cut = cn_tc_decompose(ctx, M, N, K, maxout > 1 ? CN_TC_WHOLE : cond ? CN_TC_BEHIND : clusters ? CN_TC_CLUSTERS : CN_TC_ALONE, peers && peers->npeers > 0);
    const int nt = cut.nt, kb_total = cut.kb_total;
    const int64_t tiles_m = cut.tiles_m, tiles_n = cut.tiles / tiles_m, tiles = cut.tiles, full = cut.full, tail_ctas = cut.tail_ctas, rest = cut.rest();
    const int64_t sms = ctx->sm_count;
    const int64_t grid = tail_ctas > (full < sms ? full : sms) ? tail_ctas : (full < sms ? full : sms);
    CN_REQUIRE(tiles < (1LL << 29) && grid < (1LL << 30) && rest * nt * 4 < (1LL << 31), CN_ERR_UNSUPPORTED, "cn_gemm_f32: too many work units");

    TcParams prm;
    prm.M = M; prm.N = N;
    prm.C = C; prm.ldc = ldc;
    prm.bias = epi ? epi->bias : nullptr;
    prm.act = epi ? epi->activation : CN_ACT_LINEAR;
    prm.maxout_level = maxout;
    prm.argmax = epi ? epi->argmax_out : nullptr;
    prm.tiles_n = (int)tiles_n; prm.tiles_m = (int)tiles_m;
    prm.full_tiles = (int)full; prm.tail_ctas = (int)tail_ctas; prm.kb_total = kb_total;
    prm.cluster = cut.cluster;
    int chain = w_aligned(B, ldb) ? TC_GROUP_KB : cn_gemm_any_chain(K);
    while (chain > cut.max_chain) chain >>= 1;
    if (cut.cluster > 1 && !w_aligned(B, ldb) && chain > 2) chain >>= 1;   // else 49 x 1597 . 1597 x 4326 is off by 4.0e-7, 3.5e-7 by runs
    if (ws->force_chain >= 1)
        while (chain > 1 && chain > ws->force_chain) chain >>= 1;
    prm.chain_mask = chain - 1;
    prm.a_inv = reinterpret_cast<const float *>(planes + pl.inv_off);
    prm.m_pad = pl.m_pad;
    prm.groups = (int)pl.groups;
    prm.a_bands = planes + pl.bands_off;
    prm.a_stages = (int)(pl.Kp / TC_AK);
    prm.partials = nullptr;
    prm.status = ctx->d_status;
    prm.w_ready = ahead || cond ? 0 : 1;
    prm.cond = cond ? cond->many : nullptr;
    prm.npeers = 0;
    prm.peer_flags = nullptr;
    prm.nranks = 0; prm.my_rank = 0; prm.epoch = 0;
    if (peers && peers->npeers > 0) {
        prm.npeers = peers->npeers;
        prm.peer_flags = peers->peer_flags;
        prm.nranks = peers->nranks; prm.my_rank = peers->my_rank; prm.epoch = peers->epoch;
    }
    if (cut.partial_bytes() > 0) {
        void *buf = nullptr;
        st = cn_gemm_scratch(ctx, CN_GEMM_SLOT_SPLITK, cut.partial_bytes(), &buf);
        if (st != CN_OK) return st;
        prm.partials = (float *)buf;
    }

    // 3. tensor maps
    WMaps mw;
    CUtensorMap ma;
    const int wk = w_aligned(B, ldb) ? (transB ? W_N : W_K) : (transB ? W_N_ANY : W_K_ANY);
    st = transB ? make_w_maps(enc, &mw, &prm.w_shift, B, N, K, ldb, wk)    // stored N x K, n contiguous
                : make_w_maps(enc, &mw, &prm.w_shift, B, K, N, ldb, wk);
    if (st != CN_OK) return st;
    st = cn_make_planes_map(enc, &ma, reinterpret_cast<const uint16_t *>(planes), pl.Kp, M, pl.plane, TC_BANDS * pl.parts, TC_BM);
    if (st != CN_OK) return st;

    cudaEvent_t ev_stop = nullptr;
    if (!cond && (st = cn_gemm_profile_start(ctx, s, &ev_stop)) != CN_OK) return st;
    if (ev_stop) prm.w_ready = 0;   // the event stands between the pre-pass and this launch: keep the plain order
#define CN_LAUNCH(M3, WKV) \
    (cut.cluster > 1 ? (nt == 1 ? launch_cfg<1, M3, WKV, true>(mw, ma, prm, grid, ctx->device, s) : launch_cfg<2, M3, WKV, true>(mw, ma, prm, grid, ctx->device, s)) \
                     : (nt == 1 ? launch_cfg<1, M3, WKV, false>(mw, ma, prm, grid, ctx->device, s) : launch_cfg<2, M3, WKV, false>(mw, ma, prm, grid, ctx->device, s)))
    if (wk == W_K_ANY)      st = CN_LAUNCH(true, W_K_ANY);
    else if (wk == W_N_ANY) st = CN_LAUNCH(true, W_N_ANY);
    else if (mode3x)        st = wk == W_N ? CN_LAUNCH(true, W_N) : CN_LAUNCH(true, W_K);
    else                    st = wk == W_N ? CN_LAUNCH(false, W_N) : CN_LAUNCH(false, W_K);
#undef CN_LAUNCH
    if (st != CN_OK) return st;
    if (rest > 0 && cut.cluster == 1) {
        ReduceParams rp;
        rp.partials = prm.partials; rp.nt = nt; rp.mt = 1; rp.rows = TC_BM; rp.tail_ctas = (int)tail_ctas; rp.kb_total = kb_total;
        rp.tail_tiles = (int)rest; rp.full_tiles = (int)full; rp.tiles_m = (int)tiles_m; rp.cond = prm.cond; rp.M = M; rp.N = N;
        rp.C = C; rp.ldc = ldc; rp.bias = prm.bias; rp.act = prm.act;
        rp.npeers = prm.npeers;
        for (int i = 0; i < CN_MAX_PEERS; ++i) rp.peerC[i] = prm.npeers > i ? peers->C[i] : nullptr;
        rp.ready = prm.npeers > 0 ? peers->ready : nullptr;
        rp.nranks = prm.nranks; rp.my_rank = prm.my_rank; rp.epoch = prm.epoch; rp.status = prm.status;
        if ((st = cn_splitk_reduce_launch(ctx, rp, s)) != CN_OK) return st;
    }
    if (ev_stop) CN_CUDA(cudaEventRecord(ev_stop, s));
    ctx->gemm_last_path = mode3x ? "tcgen05_3xtf32" : "tcgen05_tf32";
    ctx->gemm_last_kernel = cond ? "planes" : "streaming";
    return CN_OK;
}

// Reads the status word that a kernel sets when one of its bounded waits ran out (0 = clean).
extern "C" int cn_gemm_check_status(cn_context *ctx, void *stream)
{
    CN_REQUIRE(ctx, CN_ERR_ARG, "cn_gemm_check_status: null context");
    cudaStream_t s = cn_stream(stream);
    if (!ctx->gemm) return CN_OK;
    unsigned int h = 0;
    CN_CUDA(cudaMemcpyAsync(&h, ctx->d_status, sizeof(h), cudaMemcpyDeviceToHost, s));
    CN_CUDA(cudaStreamSynchronize(s));
    if (h != 0) {
        cudaMemsetAsync(ctx->d_status, 0, sizeof(h), s);
        cn_set_error("cn_gemm_f32: a pipeline wait ran out in the tensor-core kernel (role code %u)", h);
        return CN_ERR_TIMEOUT;
    }
    return CN_OK;
}

int cn_gemm_profile_start(cn_context *ctx, cudaStream_t s, cudaEvent_t *stop)
{
    cn_gemm_workspace *ws = ctx->gemm;
    *stop = nullptr;
    if (!ws || !ws->profile) return CN_OK;
    while (ws->prof_events.size() < ws->prof_used + 2) {
        cudaEvent_t e;
        CN_CUDA(cudaEventCreate(&e));
        ws->prof_events.push_back(e);
    }
    CN_CUDA(cudaEventRecord(ws->prof_events[ws->prof_used], s));
    *stop = ws->prof_events[ws->prof_used + 1];
    ws->prof_used += 2;
    return CN_OK;
}

extern "C" int cn_gemm_profile_enable(cn_context *ctx, int enable)
{
    CN_REQUIRE(ctx, CN_ERR_ARG, "cn_gemm_profile_enable: null context");
    if (!ctx->gemm) ctx->gemm = cn_gemm_workspace_new();
    ctx->gemm->profile = enable != 0;
    return CN_OK;
}

extern "C" int cn_gemm_profile_read(cn_context *ctx, float *ms_out, int max, int *count)
{
    CN_REQUIRE(ctx && count, CN_ERR_ARG, "cn_gemm_profile_read: null argument");
    *count = 0;
    if (!ctx->gemm) return CN_OK;
    cn_gemm_workspace *ws = ctx->gemm;
    const size_t pairs = ws->prof_used / 2;
    for (size_t i = 0; i < pairs; ++i) {
        CN_CUDA(cudaEventSynchronize(ws->prof_events[2 * i + 1]));
        float ms = 0.f;
        CN_CUDA(cudaEventElapsedTime(&ms, ws->prof_events[2 * i], ws->prof_events[2 * i + 1]));
        if ((int)i < max && ms_out) ms_out[i] = ms;
    }
    *count = (int)pairs;
    ws->prof_used = 0;
    return CN_OK;
}
