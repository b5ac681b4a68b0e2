// Stand-alone bias/activation and maxout kernels over a column-major matrix: the un-fused forms of
// addMatrixVector + activation (source/basicOps.cu:966-974; source/clusterKernels.cu:706-718) and of
// maxout (source/basicOps.cu:1287-1299; kMaxout source/clusterKernels.cu:1432-1458).
#include "cn_epilogue.cuh"

// Blocks of rows of one column: the column's bias is read once and no element needs a division to find its column.
__global__ void __launch_bounds__(256)
cn_bias_act_kernel(const float *A, const float *bias, int act, float *out, int64_t rows, int64_t cols, int64_t row_blocks)
{
    cn_pdl_launch_dependents();
    cn_pdl_wait();
    for (int64_t b = blockIdx.x; b < row_blocks * cols; b += gridDim.x) {
        const int64_t col = b / row_blocks, r0 = (b - col * row_blocks) * 1024;
        const float bj = bias ? bias[col] : 0.0f;   // kAddMatrixVector: one bias value per column
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t r = r0 + u * 256 + threadIdx.x;
            if (r < rows) {
                float v = A[col * rows + r];
                if (bias) v += bj;
                out[col * rows + r] = cn_apply_activation(v, act);
            }
        }
    }
}

// Any number of rows, an element at a time: with few rows per column the blocks above would be nearly empty (16 x 40000: 34 rounds of
// blocks with 16 of 256 threads at work).
template <typename I>
__global__ void __launch_bounds__(256)
cn_bias_act_flat_kernel(const float *A, const float *bias, int act, float *out, I rows, I n)
{
    cn_pdl_launch_dependents();
    cn_pdl_wait();
    const I stride = (I)gridDim.x * 256;
    for (I i0 = (I)blockIdx.x * 256 + threadIdx.x; i0 < n;) {
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const I i = i0 + u * stride;
            if (i < n) {
                v[u] = A[i];
                if (bias) v[u] += bias[i / rows];
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const I i = i0 + u * stride;
            if (i < n) out[i] = cn_apply_activation(v[u], act);
        }
        if (n - i0 <= 4 * stride) break;   // (the next index may not fit the type)
        i0 += 4 * stride;
    }
}

// One warp per (row, output column).  The reference reduces 32 shared-memory slots (slot t = column
// g*L + t for t < L, -FLT_MAX with index -1 otherwise) with a fixed tree: at offsets 16, 8, 4, 2, 1 slot t
// takes slot t+offset when its own value is strictly smaller (reduceToMaxAndArgMax,
// source/clusterKernels.cu:563-604).  The same tree is walked here with shuffles so that ties resolve
// to the same column.
__global__ void cn_maxout_kernel(const float *A, float *out, float *argmax, int64_t rows, int64_t out_cols, int L)
{
    cn_pdl_launch_dependents();
    cn_pdl_wait();
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t total = rows * out_cols;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < total; w += warps) {
        const int64_t g = w / rows, row = w % rows;
        float v = -FLT_MAX, idx = -1.0f;
        if (lane < L) {
            v = A[row + (g * L + lane) * rows];
            idx = (float)(g * L + lane);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float ov = __shfl_down_sync(0xffffffffu, v, off);
            const float oi = __shfl_down_sync(0xffffffffu, idx, off);
            if (lane < off && v < ov) { v = ov; idx = oi; }
        }
        if (lane == 0) {
            out[row + g * rows] = v;
            if (argmax) argmax[row + g * rows] = idx;
        }
    }
}

extern "C" int cn_bias_activation(cn_context *ctx, const float *d_A, const float *d_bias, int activation,
                                  float *d_out, int64_t rows, int64_t cols, void *stream)
{
    CN_REQUIRE(ctx && rows >= 0 && cols >= 0, CN_ERR_ARG, "cn_bias_activation: bad argument");
    const int64_t n = rows * cols;
    if (n == 0) return CN_OK;
    CN_REQUIRE(d_A && d_out, CN_ERR_ARG, "cn_bias_activation: null buffer");
    CN_REQUIRE(activation >= CN_ACT_LINEAR && activation <= CN_ACT_DOUBLE_RELU, CN_ERR_ARG, "cn_bias_activation: unknown activation %d", activation);
    const int64_t row_blocks = (rows + 1023) / 1024, cap = (int64_t)ctx->sm_count * 8;
    if (rows < 1024) {
        const int64_t want = (n + 1023) / 1024;
        const dim3 grid((unsigned)(want < cap ? want : cap));
        if (n < (1LL << 31)) CN_CUDA(cn_launch_pdl(cn_bias_act_flat_kernel<uint32_t>, grid, 256, 0, cn_stream(stream), d_A, d_bias, activation, d_out, (uint32_t)rows, (uint32_t)n));
        else CN_CUDA(cn_launch_pdl(cn_bias_act_flat_kernel<int64_t>, grid, 256, 0, cn_stream(stream), d_A, d_bias, activation, d_out, rows, n));
        cn_count_launch();
        return CN_OK;
    }
    int64_t blocks = row_blocks * cols;
    CN_CUDA(cn_launch_pdl(cn_bias_act_kernel, dim3((unsigned)(blocks < cap ? blocks : cap)), 256, 0, cn_stream(stream), d_A, d_bias, activation, d_out,
                          rows, cols, row_blocks));
    cn_count_launch();
    return CN_OK;
}

extern "C" int cn_maxout(cn_context *ctx, const float *d_A, float *d_out, float *d_argmax, int64_t rows, int64_t cols,
                         int maxout_level, void *stream)
{
    CN_REQUIRE(ctx && rows >= 0 && cols >= 0, CN_ERR_ARG, "cn_maxout: bad argument");
    // the reference asserts cols % level == 0 and level <= 64, and its 32-slot reduction covers level <= 32
    CN_REQUIRE(maxout_level >= 1 && maxout_level <= 32, CN_ERR_ARG, "cn_maxout: level %d outside 1..32", maxout_level);
    CN_REQUIRE(cols % maxout_level == 0, CN_ERR_SHAPE, "cn_maxout: %lld columns are not a multiple of level %d", (long long)cols, maxout_level);
    const int64_t out_cols = cols / maxout_level, total = rows * out_cols;
    if (total == 0) return CN_OK;
    CN_REQUIRE(d_A && d_out, CN_ERR_ARG, "cn_maxout: null buffer");
    int64_t blocks = (total + 7) / 8, cap = (int64_t)ctx->sm_count * 8;
    CN_CUDA(cn_launch_pdl(cn_maxout_kernel, dim3((unsigned)(blocks < cap ? blocks : cap)), 256, 0, cn_stream(stream), d_A, d_out, d_argmax, rows, out_cols,
                          maxout_level));
    cn_count_launch();
    return CN_OK;
}
