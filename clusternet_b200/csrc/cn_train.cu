// Elementwise kernels of the data-parallel training step and the 8-bit gradient exchange.
// They take the place of the kernels the reference's Layer class strings together per step
// (source/Layer.cpp:147-178,180-200,314-339,341-437,439-471):
//   kSoftMax source/clusterKernels.cu:651-688, kCreate_t_matrix :775-790, kSub :332-339, kMul :323-330, kAdd :313-320,
//   kScalarMul, kRectifiedLinear_Derivative :813-821, kLogisticGrad, kDoubleRectifiedLinear_Derivative,
//   kRMSprop_with_weight_update :1306-1325,
// and fuse the per-peer decompression_8bit + add loop of Layer::wait_for_synchronization into one pass.
#include <float.h>
#include "cn_gemm.h"

// ---- softmax over the columns of a column-major rows x cols matrix: one thread per row, the row's maximum, sum and
// quotient taken in the reference's order with the same fast exponential, so results match it bit for bit.  Up to
// SOFTMAX_REGS columns the row lives in registers: its loads are all in flight at once and each exponential is taken once
// (bound by latency: 128 x 10 took 3.3 us with three passes over memory).
#define SOFTMAX_REGS 32
#define SOFTMAX_THREADS 64

// ERROR: the output layer's error softmax - onehot(label) in the same pass (the three launches softmax / create_t_matrix / sub
// of the reference's step, source/Layer.cpp:163-165,318-322).  A and prob may be the same matrix.
template <bool ERROR, bool SHORT_ROWS>
__global__ void __launch_bounds__(SOFTMAX_THREADS)
cn_softmax_kernel(const float *A, const float *labels, float *prob, float *err, int64_t rows, int64_t cols)
{
    cn_pdl_launch_dependents();
    cn_pdl_wait();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < rows; row += stride) {
        const int64_t hot = ERROR ? (int64_t)(int)labels[row] : -1;
        float mx = -FLT_MAX, sum = 0.0f;
        if (SHORT_ROWS) {
            float v[SOFTMAX_REGS];
#pragma unroll
            for (int i = 0; i < SOFTMAX_REGS; ++i) v[i] = i < cols ? A[i * rows + row] : -FLT_MAX;
#pragma unroll
            for (int i = 0; i < SOFTMAX_REGS; ++i)
                if (v[i] > mx) mx = v[i];
#pragma unroll
            for (int i = 0; i < SOFTMAX_REGS; ++i)
                if (i < cols) { v[i] = __expf(v[i] - mx); sum += v[i]; }
#pragma unroll
            for (int i = 0; i < SOFTMAX_REGS; ++i)
                if (i < cols) {
                    const float pr = v[i] / sum;
                    prob[i * rows + row] = pr;
                    if (ERROR) err[i * rows + row] = pr - (i == hot ? 1.0f : 0.0f);
                }
        } else {
            for (int64_t i = 0; i < cols; ++i) {
                const float v = A[i * rows + row];
                if (v > mx) mx = v;
            }
            for (int64_t i = 0; i < cols; ++i) sum += __expf(A[i * rows + row] - mx);
            for (int64_t i = 0; i < cols; ++i) {
                const float pr = __expf(A[i * rows + row] - mx) / sum;
                prob[i * rows + row] = pr;
                if (ERROR) err[i * rows + row] = pr - (i == hot ? 1.0f : 0.0f);
            }
        }
    }
}

// Few rows of up to 32 columns: a warp per row, a lane per column.  The maximum is the same in any order; the sum is taken in the reference's
// order, an addition and a shuffle per column.  Bound by latency: the kernel above is straight code for 32 columns, which a launch fetches
// whole whatever their number.  us in a series, with the error: 128 x 10 4.3 -> 1.5, 128 x 32 8.4 -> 2.1,
// 4000 x 10 4.4 -> 2.6, 4000 x 32 8.8 -> 5.4.  Beyond, that kernel's whole lines of a column per warp are worth more.
#define SOFTMAX_WARP_ROWS 4096
template <bool ERROR>
__global__ void __launch_bounds__(128)
cn_softmax_warp_kernel(const float *A, const float *labels, float *prob, float *err, int rows, int cols)
{
    cn_pdl_launch_dependents();
    const int lane = threadIdx.x & 31, row = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int64_t at = (int64_t)lane * rows + row;
    cn_pdl_wait();
    if (row >= rows) return;
    const bool mine = lane < cols;
    const int64_t hot = ERROR ? (int64_t)(int)labels[row] : -1;
    const float v = mine ? A[at] : -FLT_MAX;
    float mx = v > -FLT_MAX ? v : -FLT_MAX;   // a NaN is no maximum
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float e = mine ? __expf(v - mx) : 0.0f;
    float sum = 0.0f;
#pragma unroll 1
    for (int i = 0; i < cols; ++i) sum += __shfl_sync(0xffffffffu, e, i);
    if (!mine) return;
    const float pr = e / sum;
    prob[at] = pr;
    if (ERROR) err[at] = pr - (lane == hot ? 1.0f : 0.0f);
}

// err_out = err_in * f'(activation), and optionally grad_out = f'(activation) (the reference writes the derivative into
// the layer's `out` matrix and multiplies in a second kernel, source/Layer.cpp:323-329)
//
// Elementwise kernels below: bound by HBM on large matrices and by launch latency on a layer's activations.  Four elements per
// thread with 16-byte accesses where every buffer is 16-byte aligned (n4 > 0), the rest one by one.
template <int ACT>
__device__ __forceinline__ float act_derivative(float a)
{
    if (ACT == CN_ACT_RELU) return a > 0.0f ? 1.0f : 0.0f;
    if (ACT == CN_ACT_LOGISTIC) return a * (1.0f - a);
    return (a > 0.0f && a < 1.0f) ? 1.0f : 0.0f;
}

template <int ACT>
__global__ void __launch_bounds__(256)
cn_mul_grad_kernel(const float *err_in, const float *act, float *grad_out, float *err_out, int64_t n, int64_t n4)
{
    cn_pdl_launch_dependents();
    cn_pdl_wait();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t v = t0; v < n4; v += stride) {
        const float4 a = reinterpret_cast<const float4 *>(act)[v], e = reinterpret_cast<const float4 *>(err_in)[v];
        const float4 g = make_float4(act_derivative<ACT>(a.x), act_derivative<ACT>(a.y), act_derivative<ACT>(a.z), act_derivative<ACT>(a.w));
        if (grad_out) reinterpret_cast<float4 *>(grad_out)[v] = g;
        reinterpret_cast<float4 *>(err_out)[v] = make_float4(e.x * g.x, e.y * g.y, e.z * g.z, e.w * g.w);
    }
    for (int64_t i = (n4 << 2) + t0; i < n; i += stride) {
        const float g = act_derivative<ACT>(act[i]);
        if (grad_out) grad_out[i] = g;
        err_out[i] = err_in[i] * g;
    }
}

// out = one-hot(labels): zero fill and scatter in one pass over the output
__global__ void cn_t_matrix_kernel(const float *labels, float *out, int64_t rows, int64_t n)
{
    cn_pdl_launch_dependents();
    cn_pdl_wait();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int64_t row = i % rows, col = i / rows;
        out[i] = ((int64_t)(int)labels[row] == col) ? 1.0f : 0.0f;
    }
}

enum { EW_ADD = 0, EW_SUB = 1, EW_MUL = 2, EW_SCALAR_MUL = 3, EW_GRAD_RELU = 4, EW_GRAD_LOGISTIC = 5, EW_GRAD_DOUBLE_RELU = 6,
       EW_ABS = 7, EW_DIV = 8, EW_SCALAR_ADD = 9, EW_SQUARE = 10 };

template <int OP>
__device__ __forceinline__ float ew_op(float a, float b, float s)
{
    if (OP == EW_ADD) return a + b;
    if (OP == EW_SUB) return a - b;
    if (OP == EW_MUL) return a * b;
    if (OP == EW_SCALAR_MUL) return a * s;
    if (OP == EW_GRAD_RELU) return act_derivative<CN_ACT_RELU>(a);
    if (OP == EW_GRAD_LOGISTIC) return act_derivative<CN_ACT_LOGISTIC>(a);
    if (OP == EW_ABS) return fabsf(a);
    if (OP == EW_DIV) return fdividef(a, b);   // kDiv divides with fdividef (source/clusterKernels.cu:341-348)
    if (OP == EW_SCALAR_ADD) return a + s;
    if (OP == EW_SQUARE) return a * a;         // kSquare calls powf(a, 2) (source/clusterKernels.cu:420-427): the product is its correctly rounded value
    return act_derivative<CN_ACT_DOUBLE_RELU>(a);
}

template <int OP>
__global__ void __launch_bounds__(256)
cn_ew_kernel(const float *A, const float *B, float s, float *out, int64_t n, int64_t n4)
{
    constexpr bool TWO = OP == EW_ADD || OP == EW_SUB || OP == EW_MUL || OP == EW_DIV;
    cn_pdl_launch_dependents();
    cn_pdl_wait();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t v = t0; v < n4; v += stride) {
        const float4 a = reinterpret_cast<const float4 *>(A)[v];
        float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
        if (TWO) b = reinterpret_cast<const float4 *>(B)[v];
        reinterpret_cast<float4 *>(out)[v] = make_float4(ew_op<OP>(a.x, b.x, s), ew_op<OP>(a.y, b.y, s), ew_op<OP>(a.z, b.z, s), ew_op<OP>(a.w, b.w, s));
    }
    for (int64_t i = (n4 << 2) + t0; i < n; i += stride) out[i] = ew_op<OP>(A[i], TWO ? B[i] : 0.f, s);
}

// kNesterov_weight_update (source/clusterKernels.cu:1064-1077): g = lr * grad / batch_size; m = momentum * m - g; w -= g
__device__ __forceinline__ void nesterov_step(float grad, float &w, float &m, float lr, float batch_size, float momentum)
{
    const float g = lr * fdividef(grad, batch_size);
    m = (momentum * m) - g;
    w -= g;
}

__global__ void __launch_bounds__(256)
cn_nesterov_kernel(const float *grad, float *w, float *m, float lr, float batch_size, float momentum, int64_t n, int64_t n4)
{
    cn_pdl_launch_dependents();
    cn_pdl_wait();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t v = t0; v < n4; v += stride) {
        const float4 g = reinterpret_cast<const float4 *>(grad)[v];
        float4 x = reinterpret_cast<const float4 *>(w)[v], q = reinterpret_cast<const float4 *>(m)[v];
        nesterov_step(g.x, x.x, q.x, lr, batch_size, momentum);
        nesterov_step(g.y, x.y, q.y, lr, batch_size, momentum);
        nesterov_step(g.z, x.z, q.z, lr, batch_size, momentum);
        nesterov_step(g.w, x.w, q.w, lr, batch_size, momentum);
        reinterpret_cast<float4 *>(m)[v] = q;
        reinterpret_cast<float4 *>(w)[v] = x;
    }
    for (int64_t i = (n4 << 2) + t0; i < n; i += stride) {
        float x = w[i], q = m[i];
        nesterov_step(grad[i], x, q, lr, batch_size, momentum);
        m[i] = q;
        w[i] = x;
    }
}

// kRMSprop_with_weight_update: RMS = m*RMS + (1-m)*g^2 ; w -= lr * g / (sqrt(RMS) + 1e-8).  The reference divides with fdividef,
// reproduced as written, and squares with powf(g, 2.0f), whose correctly rounded value is the product.
__device__ __forceinline__ void rmsprop_step(float g, float &rms, float &w, float rms_mult, float rec, float lr)
{
    const float r = (rms_mult * rms) + ((g * g) * rec);
    rms = r;
    w -= lr * fdividef(g, sqrtf(r) + 1.0e-08f);
}

// 20 bytes per element.  With one element per thread and powf it took 77 us on 4096 x 4096, against 51 us for the bytes at the
// measured copy rate.
__global__ void __launch_bounds__(256)
cn_rmsprop_kernel(float *RMS, const float *grad, float *w, float rms_mult, float lr, int64_t n, int64_t n4)
{
    cn_pdl_launch_dependents();
    cn_pdl_wait();
    const float rec = 1.0f - rms_mult;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t v = t0; v < n4; v += stride) {
        const float4 g = reinterpret_cast<const float4 *>(grad)[v];
        float4 q = reinterpret_cast<const float4 *>(RMS)[v], x = reinterpret_cast<const float4 *>(w)[v];
        rmsprop_step(g.x, q.x, x.x, rms_mult, rec, lr);
        rmsprop_step(g.y, q.y, x.y, rms_mult, rec, lr);
        rmsprop_step(g.z, q.z, x.z, rms_mult, rec, lr);
        rmsprop_step(g.w, q.w, x.w, rms_mult, rec, lr);
        reinterpret_cast<float4 *>(RMS)[v] = q;
        reinterpret_cast<float4 *>(w)[v] = x;
    }
    for (int64_t i = (n4 << 2) + t0; i < n; i += stride) {
        float r = RMS[i], x = w[i];
        rmsprop_step(grad[i], r, x, rms_mult, rec, lr);
        RMS[i] = r;
        w[i] = x;
    }
}

// grad[i] += sum over peers r != me of decode_r(codes_r[i]); decode tables as kDecompression_8bit builds them, one per
// rank with that rank's scale; peers are added in rank order (the order of the reference's loop).  The gradients of
// several tensors (segments) lie back to back in one buffer, each coded with its own scale per rank.  A rank's block of
// the gathered buffer is [codes of all segments][one scale per segment]; seg_end[s] is the end offset of segment s.
#define CN_SYNC_MAX_SEGMENTS 8
struct SegParams {
    int nseg;
    int64_t seg_end[CN_SYNC_MAX_SEGMENTS];
};

// UPDATE: the RMSprop step of cn_rmsprop_kernel on the summed gradient in the same pass (same arithmetic, one launch less).
// Four elements per thread where the buffers allow 16-byte accesses (vec_ok) and the four lie in one segment.
template <bool UPDATE>
__global__ void __launch_bounds__(512)
cn_decode_sum_multi_kernel(float *grad, const uint8_t *blocks, size_t block_bytes, size_t scales_off,
                           const float *g_tbl, int64_t n, int nranks, int my_rank, const SegParams sp,
                           float *RMS, float *w, float rms_mult, float lr, int vec_ok)
{
    extern __shared__ float lut[];   // (segment, rank) x 256
    cn_pdl_launch_dependents();
    cn_pdl_wait();
    for (int e = threadIdx.x; e < sp.nseg * nranks * 256; e += blockDim.x) {
        const int sr = e >> 8, c = e & 255, i = c & 127;
        const int seg = sr / nranks, r = sr - seg * nranks;
        const float p = reinterpret_cast<const float *>(blocks + (size_t)r * block_bytes + scales_off)[seg];
        float v;
        if (i < CN_CODEBOOK_N) {
            v = __fmul_rn(g_tbl[i], p);
            if (c >= 128) v = -v;
        } else {
            v = (c == 255) ? -p : p;
        }
        lut[e] = v;
    }
    __syncthreads();
    const float rec = 1.0f - rms_mult;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, tid0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    auto one = [&](int64_t i) {
        int seg = 0;
        while (seg + 1 < sp.nseg && i >= sp.seg_end[seg]) ++seg;
        const float *l = lut + (size_t)seg * nranks * 256;
        float g = grad[i];
        for (int r = 0; r < nranks; ++r)
            if (r != my_rank) g += l[(r << 8) + blocks[(size_t)r * block_bytes + i]];
        grad[i] = g;
        if (UPDATE) {
            float q = RMS[i], x = w[i];
            rmsprop_step(g, q, x, rms_mult, rec, lr);
            RMS[i] = q;
            w[i] = x;
        }
    };
    const int64_t n4 = vec_ok ? (n >> 2) : 0;
    for (int64_t v = tid0; v < n4; v += stride) {
        const int64_t i = v << 2;
        int seg = 0;
        while (seg + 1 < sp.nseg && i >= sp.seg_end[seg]) ++seg;
        if (i + 3 >= sp.seg_end[seg] && seg + 1 < sp.nseg) {   // the four straddle a segment boundary
            for (int k = 0; k < 4; ++k) one(i + k);
            continue;
        }
        const float *l = lut + (size_t)seg * nranks * 256;
        float4 g = reinterpret_cast<const float4 *>(grad)[v];
        for (int r = 0; r < nranks; ++r) {
            if (r == my_rank) continue;
            const uint32_t c = *reinterpret_cast<const uint32_t *>(blocks + (size_t)r * block_bytes + i);
            const float *lr_ = l + (r << 8);
            g.x += lr_[c & 0xffu];
            g.y += lr_[(c >> 8) & 0xffu];
            g.z += lr_[(c >> 16) & 0xffu];
            g.w += lr_[c >> 24];
        }
        reinterpret_cast<float4 *>(grad)[v] = g;
        if (UPDATE) {
            float4 q = reinterpret_cast<const float4 *>(RMS)[v], x = reinterpret_cast<const float4 *>(w)[v];
            rmsprop_step(g.x, q.x, x.x, rms_mult, rec, lr);
            rmsprop_step(g.y, q.y, x.y, rms_mult, rec, lr);
            rmsprop_step(g.z, q.z, x.z, rms_mult, rec, lr);
            rmsprop_step(g.w, q.w, x.w, rms_mult, rec, lr);
            reinterpret_cast<float4 *>(RMS)[v] = q;
            reinterpret_cast<float4 *>(w)[v] = x;
        }
    }
    for (int64_t i = (n4 << 2) + tid0; i < n; i += stride) one(i);
}

// blocks of 256 threads, `per_thread` elements each, at most eight per SM
static dim3 ew_grid(const cn_context *ctx, int64_t n, int per_thread)
{
    const int64_t cap = (int64_t)ctx->sm_count * 8;
    int64_t blocks = (n + 256 * per_thread - 1) / (256 * per_thread);
    if (blocks < 1) blocks = 1;
    return dim3((unsigned)(blocks < cap ? blocks : cap));
}

static bool aligned16(const void *a, const void *b = nullptr, const void *c = nullptr, const void *d = nullptr)
{
    return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 15u) == 0;
}

template <bool ERROR>
static int softmax_launch(cn_context *ctx, const float *A, const float *labels, float *prob, float *err, int64_t rows, int64_t cols, void *stream)
{
    const int64_t blocks = (rows + SOFTMAX_THREADS - 1) / SOFTMAX_THREADS;
    const dim3 grid((unsigned)(blocks < 4096 ? blocks : 4096));
    if (cols <= 32 && rows < SOFTMAX_WARP_ROWS)
        CN_CUDA(cn_launch_pdl(cn_softmax_warp_kernel<ERROR>, dim3((unsigned)((rows + 3) / 4)), 128, 0, cn_stream(stream), A, labels, prob, err, (int)rows, (int)cols));
    else if (cols <= SOFTMAX_REGS)
        CN_CUDA(cn_launch_pdl(cn_softmax_kernel<ERROR, true>, grid, SOFTMAX_THREADS, 0, cn_stream(stream), A, labels, prob, err, rows, cols));
    else
        CN_CUDA(cn_launch_pdl(cn_softmax_kernel<ERROR, false>, grid, SOFTMAX_THREADS, 0, cn_stream(stream), A, labels, prob, err, rows, cols));
    cn_count_launch();
    return CN_OK;
}

extern "C" int cn_softmax(cn_context *ctx, const float *d_A, float *d_out, int64_t rows, int64_t cols, void *stream)
{
    CN_REQUIRE(ctx && rows >= 0 && cols >= 0 && (rows * cols == 0 || (d_A && d_out)), CN_ERR_ARG, "cn_softmax: bad argument");
    if (rows * cols == 0) return CN_OK;
    return softmax_launch<false>(ctx, d_A, nullptr, d_out, nullptr, rows, cols, stream);
}

extern "C" int cn_softmax_error(cn_context *ctx, const float *d_A, const float *d_labels, float *d_softmax_out, float *d_error_out,
                                int64_t rows, int64_t cols, void *stream)
{
    CN_REQUIRE(ctx && rows >= 0 && cols >= 0 && (rows * cols == 0 || (d_A && d_labels && d_softmax_out && d_error_out)), CN_ERR_ARG,
               "cn_softmax_error: bad argument");
    if (rows * cols == 0) return CN_OK;
    return softmax_launch<true>(ctx, d_A, d_labels, d_softmax_out, d_error_out, rows, cols, stream);
}

extern "C" int cn_create_t_matrix(cn_context *ctx, const float *d_labels, float *d_out, int64_t rows, int64_t cols, void *stream)
{
    CN_REQUIRE(ctx && rows >= 0 && cols >= 0 && (rows * cols == 0 || (d_labels && d_out)), CN_ERR_ARG, "cn_create_t_matrix: bad argument");
    if (rows * cols == 0) return CN_OK;
    CN_CUDA(cn_launch_pdl(cn_t_matrix_kernel, ew_grid(ctx, rows * cols, 1), 256, 0, cn_stream(stream), d_labels, d_out, rows, rows * cols));
    cn_count_launch();
    return CN_OK;
}

template <int OP>
static int ew_launch(cn_context *ctx, const float *A, const float *B, float s, float *out, int64_t n, void *stream, bool needs_b)
{
    CN_REQUIRE(ctx && n >= 0 && (n == 0 || (A && out && (!needs_b || B))), CN_ERR_ARG, "elementwise op: bad argument");
    if (n == 0) return CN_OK;
    const int64_t n4 = aligned16(A, needs_b ? B : nullptr, out) ? n >> 2 : 0;
    CN_CUDA(cn_launch_pdl(cn_ew_kernel<OP>, ew_grid(ctx, n, n4 ? 4 : 1), 256, 0, cn_stream(stream), A, B, s, out, n, n4));
    cn_count_launch();
    return CN_OK;
}

extern "C" int cn_add(cn_context *ctx, const float *a, const float *b, float *out, int64_t n, void *stream) { return ew_launch<EW_ADD>(ctx, a, b, 0.f, out, n, stream, true); }
extern "C" int cn_sub(cn_context *ctx, const float *a, const float *b, float *out, int64_t n, void *stream) { return ew_launch<EW_SUB>(ctx, a, b, 0.f, out, n, stream, true); }
extern "C" int cn_mul(cn_context *ctx, const float *a, const float *b, float *out, int64_t n, void *stream) { return ew_launch<EW_MUL>(ctx, a, b, 0.f, out, n, stream, true); }
extern "C" int cn_scalar_mul(cn_context *ctx, const float *a, float s, float *out, int64_t n, void *stream) { return ew_launch<EW_SCALAR_MUL>(ctx, a, nullptr, s, out, n, stream, false); }

extern "C" int cn_div(cn_context *ctx, const float *a, const float *b, float *out, int64_t n, void *stream) { return ew_launch<EW_DIV>(ctx, a, b, 0.f, out, n, stream, true); }
extern "C" int cn_scalar_add(cn_context *ctx, const float *a, float s, float *out, int64_t n, void *stream) { return ew_launch<EW_SCALAR_ADD>(ctx, a, nullptr, s, out, n, stream, false); }
extern "C" int cn_abs(cn_context *ctx, const float *a, float *out, int64_t n, void *stream) { return ew_launch<EW_ABS>(ctx, a, nullptr, 0.f, out, n, stream, false); }
extern "C" int cn_square(cn_context *ctx, const float *a, float *out, int64_t n, void *stream) { return ew_launch<EW_SQUARE>(ctx, a, nullptr, 0.f, out, n, stream, false); }

extern "C" int cn_nesterov_update(cn_context *ctx, const float *d_grad, float *d_w, float *d_m, float learning_rate, int64_t batch_size,
                                  float momentum, int64_t n, void *stream)
{
    CN_REQUIRE(ctx && n >= 0 && batch_size > 0 && (n == 0 || (d_grad && d_w && d_m)), CN_ERR_ARG, "cn_nesterov_update: bad argument");
    if (n == 0) return CN_OK;
    const int64_t n4 = aligned16(d_grad, d_w, d_m) ? n >> 2 : 0;
    CN_CUDA(cn_launch_pdl(cn_nesterov_kernel, ew_grid(ctx, n, n4 ? 4 : 1), 256, 0, cn_stream(stream), d_grad, d_w, d_m, learning_rate, (float)batch_size,
                          momentum, n, n4));
    cn_count_launch();
    return CN_OK;
}

extern "C" int cn_activation_gradient(cn_context *ctx, const float *d_activation, int activation, float *d_out, int64_t n, void *stream)
{
    switch (activation) {
        case CN_ACT_RELU: return ew_launch<EW_GRAD_RELU>(ctx, d_activation, nullptr, 0.f, d_out, n, stream, false);
        case CN_ACT_LOGISTIC: return ew_launch<EW_GRAD_LOGISTIC>(ctx, d_activation, nullptr, 0.f, d_out, n, stream, false);
        case CN_ACT_DOUBLE_RELU: return ew_launch<EW_GRAD_DOUBLE_RELU>(ctx, d_activation, nullptr, 0.f, d_out, n, stream, false);
    }
    cn_set_error("cn_activation_gradient: no derivative for activation %d (the reference throws 'Unknown unit')", activation);
    return CN_ERR_ARG;
}

extern "C" int cn_mul_activation_gradient(cn_context *ctx, const float *d_error_in, const float *d_activation, int activation,
                                          float *d_gradient_out, float *d_error_out, int64_t n, void *stream)
{
    CN_REQUIRE(ctx && n >= 0 && (n == 0 || (d_error_in && d_activation && d_error_out)), CN_ERR_ARG, "cn_mul_activation_gradient: bad argument");
    if (n == 0) return CN_OK;
    const int64_t n4 = aligned16(d_error_in, d_activation, d_gradient_out, d_error_out) ? n >> 2 : 0;
    const dim3 grid = ew_grid(ctx, n, n4 ? 4 : 1);
#define CN_MUL_GRAD(ACT) \
    CN_CUDA(cn_launch_pdl(cn_mul_grad_kernel<ACT>, grid, 256, 0, cn_stream(stream), d_error_in, d_activation, d_gradient_out, d_error_out, n, n4))
    switch (activation) {
        case CN_ACT_RELU: CN_MUL_GRAD(CN_ACT_RELU); break;
        case CN_ACT_LOGISTIC: CN_MUL_GRAD(CN_ACT_LOGISTIC); break;
        case CN_ACT_DOUBLE_RELU: CN_MUL_GRAD(CN_ACT_DOUBLE_RELU); break;
        default:
            cn_set_error("cn_mul_activation_gradient: no derivative for activation %d (the reference throws 'Unknown unit')", activation);
            return CN_ERR_ARG;
    }
#undef CN_MUL_GRAD
    cn_count_launch();
    return CN_OK;
}

extern "C" int cn_rmsprop_update(cn_context *ctx, float *d_rms, const float *d_grad, float *d_w, float rms_multiplier, float learning_rate,
                                 int64_t n, void *stream)
{
    CN_REQUIRE(ctx && n >= 0 && (n == 0 || (d_rms && d_grad && d_w)), CN_ERR_ARG, "cn_rmsprop_update: bad argument");
    if (n == 0) return CN_OK;
    const int64_t n4 = aligned16(d_rms, d_grad, d_w) ? n >> 2 : 0;
    CN_CUDA(cn_launch_pdl(cn_rmsprop_kernel, ew_grid(ctx, n, n4 ? 4 : 1), 256, 0, cn_stream(stream), d_rms, d_grad, d_w, rms_multiplier, learning_rate, n,
                          n4));
    cn_count_launch();
    return CN_OK;
}

// comm-side pieces live in cn_comm.cu
int cn_comm_info(cn_context *ctx, int *rank, int *nranks, float **d_scales);

int cn_comm_gather_blocks(cn_context *ctx, uint8_t *d_blocks, size_t block_bytes, void *stream);
int cn_comm_push_area(cn_context *ctx, size_t block_bytes, void *stream, uint8_t **blocks);
int cn_comm_push_blocks(cn_context *ctx, uint8_t *blocks, size_t block_bytes, void *stream);

// Several tensors that lie back to back in one buffer (the gradients of all layers of a step), each coded with its own
// scale exactly as cn_grad_sync_8bit would code it alone, but exchanged with ONE all-gather and summed in ONE pass.
extern "C" int cn_grad_sync_8bit(cn_context *ctx, float *d_grad, int64_t n, float fixed_precision, void *stream);

static int grad_sync_multi_impl(cn_context *ctx, float *d_grad, const int64_t *segment_sizes, int num_segments, float fixed_precision,
                                float *d_rms, float *d_w, float rms_multiplier, float learning_rate, void *stream)
{
    const bool update = d_rms != nullptr;
    CN_REQUIRE(ctx && segment_sizes && num_segments >= 1, CN_ERR_ARG, "cn_grad_sync_8bit_multi: bad argument");
    int rank = 0, G = 1;
    float *unused = nullptr;
    cn_comm_info(ctx, &rank, &G, &unused);
    int64_t n = 0;
    for (int s = 0; s < num_segments; ++s) {
        CN_REQUIRE(segment_sizes[s] >= 0, CN_ERR_ARG, "cn_grad_sync_8bit_multi: negative segment size");
        n += segment_sizes[s];
    }
    if (n == 0) return CN_OK;
    CN_REQUIRE(d_grad, CN_ERR_ARG, "cn_grad_sync_8bit_multi: null buffer");
    if (G == 1) return update ? cn_rmsprop_update(ctx, d_rms, d_grad, d_w, rms_multiplier, learning_rate, n, stream) : CN_OK;
    if (num_segments > CN_SYNC_MAX_SEGMENTS || (size_t)num_segments * G * 1024 > 48 * 1024) {
        // too many tables for one pass: segment by segment
        int64_t off = 0;
        for (int s = 0; s < num_segments; ++s) {
            int st = cn_grad_sync_8bit(ctx, d_grad + off, segment_sizes[s], fixed_precision, stream);
            if (st != CN_OK) return st;
            off += segment_sizes[s];
        }
        return update ? cn_rmsprop_update(ctx, d_rms, d_grad, d_w, rms_multiplier, learning_rate, n, stream) : CN_OK;
    }
    const size_t scales_off = ((size_t)n + 15) & ~(size_t)15;
    const size_t block_bytes = scales_off + (((size_t)num_segments * sizeof(float) + 15) & ~(size_t)15);
    // the blocks travel by direct stores into the peers' memory where the communicator can do that (one process per
    // GPU), else through the library's all-gather
    uint8_t *blocks = nullptr;
    int st = cn_comm_push_area(ctx, block_bytes, stream, &blocks);
    if (st != CN_OK) return st;
    const bool pushed = blocks != nullptr;
    if (!pushed) {
        void *buf = nullptr;
        if ((st = cn_gemm_scratch(ctx, CN_GEMM_SLOT_EXCHANGE, (size_t)G * block_bytes, &buf)) != CN_OK) return st;
        blocks = (uint8_t *)buf;
    }
    uint8_t *mine = blocks + (size_t)rank * block_bytes;
    float *my_scales = reinterpret_cast<float *>(mine + scales_off);
    SegParams sp;
    sp.nseg = num_segments;
    int64_t off = 0;
    bool exchanged = false;
    if (pushed && num_segments == 1 && fixed_precision <= 0.0f) {
        // one tensor, scale = its absmax: code and push in ONE launch where the tensor is small enough for that form
        cn_codec_push cp;
        if ((st = cn_comm_push_params(ctx, block_bytes, scales_off, &cp)) != CN_OK) return st;
        int done = 0;
        if ((st = cn_absmax_compress_push(ctx, d_grad, n, my_scales, mine, &cp, stream, &done)) != CN_OK) return st;
        exchanged = done != 0;
    }
    for (int s = 0; s < num_segments; ++s) {
        const int64_t sz = segment_sizes[s];
        if (exchanged) {
            // done above
        } else if (fixed_precision > 0.0f) {
            st = cn_fill_f32(ctx, my_scales + s, 1, fixed_precision, stream);
            if (st == CN_OK && sz > 0) st = cn_compress_8bit_dp(ctx, d_grad + off, my_scales + s, sz, mine + off, stream);
        } else {
            st = cn_absmax_compress_8bit(ctx, d_grad + off, sz, my_scales + s, mine + off, stream);   // one launch per tensor
        }
        if (st != CN_OK) return st;
        off += sz;
        sp.seg_end[s] = off;
    }
    for (int s = num_segments; s < CN_SYNC_MAX_SEGMENTS; ++s) sp.seg_end[s] = off;
    if (!exchanged) {
        st = pushed ? cn_comm_push_blocks(ctx, blocks, block_bytes, stream) : cn_comm_gather_blocks(ctx, blocks, block_bytes, stream);
        if (st != CN_OK) return st;
    }
    const int vec_ok = ((uintptr_t)d_grad % 16 == 0) && ((uintptr_t)blocks % 16 == 0) &&
                       (!update || ((uintptr_t)d_rms % 16 == 0 && (uintptr_t)d_w % 16 == 0));
    const int64_t work = vec_ok ? (n + 3) / 4 : n;
    int64_t nblocks = (work + 511) / 512, cap = (int64_t)ctx->sm_count * 4;
    const unsigned grid = (unsigned)(nblocks < cap ? nblocks : cap);
    const size_t smem = (size_t)num_segments * G * 256 * sizeof(float);
    if (update)
        cn_decode_sum_multi_kernel<true><<<grid, 512, smem, cn_stream(stream)>>>(d_grad, blocks, block_bytes, scales_off, ctx->d_tbl, n, G, rank, sp,
                                                                                 d_rms, d_w, rms_multiplier, learning_rate, vec_ok);
    else
        cn_decode_sum_multi_kernel<false><<<grid, 512, smem, cn_stream(stream)>>>(d_grad, blocks, block_bytes, scales_off, ctx->d_tbl, n, G, rank, sp,
                                                                                  nullptr, nullptr, 0.f, 0.f, vec_ok);
    CN_CUDA(cudaGetLastError());
    cn_count_launch();
    return CN_OK;
}

extern "C" int cn_grad_sync_8bit(cn_context *ctx, float *d_grad, int64_t n, float fixed_precision, void *stream)
{
    CN_REQUIRE(ctx && n >= 0 && (n == 0 || d_grad), CN_ERR_ARG, "cn_grad_sync_8bit: bad argument");
    return grad_sync_multi_impl(ctx, d_grad, &n, 1, fixed_precision, nullptr, nullptr, 0.f, 0.f, stream);
}

extern "C" int cn_grad_sync_8bit_multi(cn_context *ctx, float *d_grad, const int64_t *segment_sizes, int num_segments,
                                       float fixed_precision, void *stream)
{
    return grad_sync_multi_impl(ctx, d_grad, segment_sizes, num_segments, fixed_precision, nullptr, nullptr, 0.f, 0.f, stream);
}

// cn_grad_sync_8bit_multi followed by cn_rmsprop_update over the same elements, with the update done in the pass that sums
// the decoded gradients: the results (gradient, RMS state, weights) are those of the two calls bit for bit.
extern "C" int cn_grad_sync_8bit_rmsprop(cn_context *ctx, float *d_grad, const int64_t *segment_sizes, int num_segments,
                                         float fixed_precision, float *d_rms, float *d_w, float rms_multiplier, float learning_rate,
                                         void *stream)
{
    CN_REQUIRE(d_rms && d_w, CN_ERR_ARG, "cn_grad_sync_8bit_rmsprop: null state or weight buffer");
    return grad_sync_multi_impl(ctx, d_grad, segment_sizes, num_segments, fixed_precision, d_rms, d_w, rms_multiplier, learning_rate, stream);
}
