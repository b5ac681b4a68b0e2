// Host-side pieces that the two tensor-core kernels over planes share (cn_gemm_tc.cu, cn_gemm_planes.cu).
#pragma once
#include <cuda.h>
#include "cn_gemm.h"

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
int cn_get_encode_fn(cn_context *ctx, EncodeTiledFn *out);
// Planes of an operand: fp16, k contiguous with pitch Kp, `plane` elements apart, box 64 k x box_rows rows of one, 128-byte swizzle.
int cn_make_planes_map(EncodeTiledFn enc, CUtensorMap *map, const uint16_t *base, int64_t Kp, int64_t rows, int64_t plane, int planes, int box_rows);
// The pre-pass: planes of an operand whose rows lie k contiguous (`k_contiguous`) or row contiguous; pl says how many bands.
int cn_make_planes(cn_context *ctx, bool k_contiguous, int64_t rows, int64_t K, const float *src, int64_t ld, const cn_coded_src *cs, const cn_planes &pl,
                   void *planes, cudaStream_t s);

// Reduction of the runs of K blocks that tiles were cut into (cn_splitk_reduce_kernel).
struct ReduceParams {
    const float *partials;       // [slot][mt][nt][32 quads of m][128 n] float4
    int nt, mt;                  // blocks of 128 columns n, and of `rows` rows m, per tile
    int rows;
    int tail_ctas, kb_total;
    int tail_tiles;              // tiles cut into runs, [full_tiles, full_tiles + tail_tiles)
    int full_tiles, tiles_m;
    const unsigned int *cond;    // add them only where this word is not zero; null: always
    int64_t M, N;
    float *C;
    int64_t ldc;
    const float *bias;
    int act;
    int npeers;
    float *peerC[CN_MAX_PEERS];
    const unsigned int *ready;
    int nranks, my_rank;
    unsigned int epoch;
    unsigned int *status;
};
int cn_splitk_reduce_launch(cn_context *ctx, const ReduceParams &rp, cudaStream_t s);

// The streaming kernel's decomposition of a product: nt tiles of 128 columns n per CTA, whole tiles, then tiles cut into runs; or, cluster > 1,
// every tile's K shared by the CTAs of a cluster.
struct cn_tc_cut {
    int nt, kb_total, cluster;
    int max_chain;   // K blocks per accumulation chain, at most
    int64_t tiles_m, tiles, full, tail_ctas;
    int64_t rest() const { return tiles - full; }
    size_t partial_bytes() const;   // of CN_GEMM_SLOT_SPLITK
};
// CN_TC_WHOLE: whole tiles only; CN_TC_BEHIND: the launch behind the planes kernel; CN_TC_CLUSTERS: clusters, where they are faster
enum { CN_TC_ALONE, CN_TC_WHOLE, CN_TC_BEHIND, CN_TC_CLUSTERS };
cn_tc_cut cn_tc_decompose(const cn_context *ctx, int64_t M, int64_t N, int64_t K, int kind, bool push);

// The streaming kernel behind the one that multiplies planes: it runs where the word at `many` (CN_STATUS_MANY) is not zero, on these
// planes of the activations, and so does the reduction of its runs.
struct cn_tc_cond {
    unsigned int *many;
    void *planes;
};
