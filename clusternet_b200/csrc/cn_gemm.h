// Internal interface between the GEMM entry point (cn_gemm.cu) and the tensor-core kernel (cn_gemm_tc.cu).
#pragma once
#include "cn_internal.h"

enum {
    CN_GEMM_SLOT_MAXOUT = 0,   // full product ahead of an un-fused maxout
    CN_GEMM_SLOT_ASPLIT = 1,   // activations re-laid K-major as hi / lo planes with their scales
    CN_GEMM_SLOT_SPLITK = 2,   // partial tiles of the runs of K blocks of a launch
    CN_GEMM_SLOT_EXCHANGE = 3, // codes + scales of the 8-bit exchange in dotMPI
    CN_GEMM_SLOT_WSPLIT = 4,   // weights as hi / lo planes, for products with many rows
    CN_GEMM_SLOTS = 5
};

// Words of the status block.  OVERFLOW: raised by the pre-pass of a product of planes by planes where a list overflows, taken back by the
// streaming kernel behind that product.  MANY: what the product found there, for the kernels behind it.
#define CN_STATUS_MANY 1
#define CN_STATUS_OVERFLOW 2

// Activations that exist only as gathered 8-bit codes (plus this rank's own block in fp32): set by
// cn_dotmpi_from_coded_f32 right before the dispatch, consumed by the tensor-core launch, whose pre-pass then decodes
// while it transposes and splits.
struct cn_coded_src {
    const uint8_t *codes = nullptr;
    const float *scales = nullptr;
    const float *own_fp32 = nullptr;
    int nranks = 1, own_rank = 0;
};

// Planes of an M x K activation operand, in one allocation: per band fp16 hi [M][Kp] and, in the 3x mode, lo, `plane` elements apart;
// inverse scales [band][group of CN_PLANE_GROUP_K k][m_pad]; bands behind the first that a block of 16 rows x 64 k has, a byte each
// [tile of 128 rows][64 k][8] (see cn_gemm_tc.cu); cells of left-overs [block of 16 rows][group]: how many elements of the 16 x 512
// band 0 leaves something of, a byte each, and up to CN_CELL of them, {row << 16 | k, value}.
#define CN_PLANE_GROUP_K 512
#define CN_PLANE_BANDS 3
#define CN_CELL 8
struct cn_planes {
    int64_t Kp, plane, m_pad, groups;
    int parts, bands;
    size_t inv_off, bands_off, counts_off, cells_off, bytes;
};
void cn_plane_layout(int64_t M, int64_t K, int mode, cn_planes *pl, int bands = CN_PLANE_BANDS);

// The planes of an activation operand made ahead of the product that consumes them (cn_gemm_prepare): the product's own
// pre-pass is then skipped.
struct cn_prepared {
    cn_context *ctx = nullptr;
    void *planes = nullptr;
    float *raw = nullptr;       // K-major fp32 copy with pitch raw_ld, for products small enough for the one-launch kernel
    int64_t M = 0, K = 0, raw_ld = 0;
    int mode = 0;
    bool filled = false;
};

struct cn_tc_cond;

struct cn_gemm_workspace {
    void *ptr[CN_GEMM_SLOTS] = {nullptr, nullptr, nullptr, nullptr};
    size_t bytes[CN_GEMM_SLOTS] = {0, 0, 0, 0};
    void *encode_fn = nullptr;          // cuTensorMapEncodeTiled, resolved once
    const cn_coded_src *coded_src = nullptr;   // one-shot: see cn_coded_src
    const cn_prepared *prepared = nullptr;   // one-shot: planes made ahead of the launch (cn_gemm_prepare)
    // test and sweep knobs (0 = automatic choice): W tiles per CTA, K splits, K blocks per accumulation chain.  Seeded once,
    // when the workspace is made, from CN_GEMM_NT / CN_GEMM_SPLITS / CN_GEMM_CHAIN; changed with cn_gemm_set_tuning.
    int force_nt = 0, force_splits = 0, force_chain = 0;
    bool wsplit_recorded = false;       // a recorded graph may read CN_GEMM_SLOT_WSPLIT
    bool profile = false;               // bracket main-kernel launches with events
    std::vector<cudaEvent_t> prof_events;   // start, stop, start, stop, ...
    size_t prof_used = 0;
};

// The only way a workspace is made: reads the environment knobs once.
cn_gemm_workspace *cn_gemm_workspace_new();

// Where products are profiled (cn_gemm_profile_enable): records the start of one, behind its pre-pass, and hands out the event for its end.
int cn_gemm_profile_start(cn_context *ctx, cudaStream_t s, cudaEvent_t *stop);
// Grow-only scratch buffers owned by the context.
int cn_gemm_scratch(cn_context *ctx, int slot, size_t bytes, void **out);
// cudaMalloc that gives back the planes of the weights, which products can do without, before it fails for want of memory.
cudaError_t cn_gemm_malloc(cn_context *ctx, void **p, size_t bytes);

// Peer windows of the output for the fused all-gather: the tensor-core kernel's epilogue stores each finished tile into
// the same window of every peer's C (plain stores to peer memory over NVLink) in addition to the local C.
#define CN_MAX_PEERS 7
struct cn_peer_out {
    int npeers = 0;
    float *C[CN_MAX_PEERS] = {};          // peer addresses of the window that d_C points to locally
    const unsigned int *ready = nullptr;  // local flags, one per rank, raised by the peers when they may be written to
    unsigned int *const *peer_flags = nullptr;   // device table: flag block of every rank (this kernel raises its own "ready")
    int nranks = 0;
    int my_rank = 0;
    unsigned int epoch = 0;
};

bool cn_gemm_tc_supported(cn_context *ctx, int transA, int transB, int64_t M, int64_t N, int64_t K,
                          const float *A, int64_t lda, const float *B, int64_t ldb, const float *C, int64_t ldc);
// Weights of any pitch and alignment: the same kernel in its 3x mode, no peers, no prepared or coded activations.
bool cn_gemm_tc_any_supported(int transB, int64_t M, int64_t N, int64_t K, const float *B);
bool cn_gemm_tc_can_fuse_maxout(int level);
// the activation pre-pass alone, into caller-owned planes of cn_plane_layout's size
int cn_gemm_tc_split_activations(cn_context *ctx, int transA, int64_t M, int64_t K, const float *A, int64_t lda, int mode, void *planes,
                                 cudaStream_t s);
int cn_gemm_tc_launch(cn_context *ctx, int64_t M, int64_t N, int64_t K, const float *A, int64_t lda,
                      const float *B, int64_t ldb, float *C, int64_t ldc, const cn_epilogue *epi, int mode, cudaStream_t s,
                      const cn_peer_out *peers = nullptr, int transA = 0, int transB = 0, const cn_tc_cond *cond = nullptr, bool clusters = false);
// Products of planes by planes (cn_gemm_planes.cu), any layout and alignment of both operands: whether it is the faster kernel for a
// shape, and the launch.  `fine`: the shape is one for the small products' kernel,
// whose error must not be exceeded, and which is the one to record in a graph.  *done = false: no room for the planes of the weights, or that;
// nothing was launched.
bool cn_gemm_planes_shape(const cn_context *ctx, int64_t M, int64_t N, int64_t K, int mode, bool w_aligned, bool fine);
int cn_gemm_planes_launch(cn_context *ctx, int64_t M, int64_t N, int64_t K, const float *A, int64_t lda, const float *B, int64_t ldb, float *C, int64_t ldc,
                          const cn_epilogue *epi, int mode, cudaStream_t s, int transA, int transB, bool w_aligned, bool fine, bool *done);
// Small products in one launch (cn_gemm_small.cu): whether a shape is one, and the launch.  Takes any layout and alignment.
bool cn_gemm_small_shape(const cn_context *ctx, int64_t M, int64_t N, int64_t K, bool w_aligned, int max_rounds);
#define CN_SMALL_MAX_K 3072   // no product of aligned weights with a longer inner dimension is small: eight CTAs of twelve blocks of 32
// K blocks of 32 per accumulation chain for weights whose rows TMA cannot read (cn_gemm_tc.cu)
int cn_gemm_any_chain(int64_t K);
int cn_gemm_small_launch(cn_context *ctx, int transA, int transB, int64_t M, int64_t N, int64_t K, const float *A, int64_t lda, const float *B, int64_t ldb,
                         float *C, int64_t ldc, const cn_epilogue *epi, int mode, cudaStream_t s, const cn_peer_out *peers);
// Weight gradients with a short inner dimension in one launch (cn_gemm_outer.cu): A (K x M) transposed, B (K x N), any alignment.  `fine`: the shape
// is one for the small products' kernel, whose error must not be exceeded.
bool cn_gemm_outer_shape(int64_t M, int64_t N, int64_t K);
int cn_gemm_outer_launch(cn_context *ctx, int64_t M, int64_t N, int64_t K, const float *A, int64_t lda, const float *B, int64_t ldb, float *C, int64_t ldc,
                         cudaStream_t s, bool fine);
// cn_gemm_f32 with optional peer windows; *used_peers tells whether the launch took them (tensor-core path only).  planes_ok: the
// kernel for many rows may be taken.  The products with a column-sharded weight (cn_dotmpi_f32 and its forms) do not take it: their bits may
// not depend on whether the activations' planes were made ahead, the activations are codes, or the output goes to peers, and those
// forms are the streaming kernel's.
int cn_gemm_dispatch(cn_context *ctx, int transA, int transB, int64_t M, int64_t N, int64_t K, const float *d_A, int64_t lda,
                     const float *d_B, int64_t ldb, float *d_C, int64_t ldc, const cn_epilogue *epi, int mode, void *stream,
                     const cn_peer_out *peers, bool *used_peers, bool planes_ok = false);
