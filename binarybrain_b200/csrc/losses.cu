// Neighbours of the LUT path in a training step: the two losses the reference's LUT samples use and the node-group mean
// (bb::Reduce) that maps the last LUT layer to class scores.  Tiny next to the LUT layers (10 class rows against
// thousands of LUT rows); they exist so that a whole step -- forward, loss, backward, Adam -- stays on the device.
//
// Semantics follow the reference's CPU branches:
//   LossSoftmaxCrossEntropy  include/bb/LossSoftmaxCrossEntropy.h:151-205   (operator: include/bbcu/bbcu.h:1507-1519)
//   LossMeanSquaredError     include/bb/LossMeanSquaredError.h:153-172      (operator: include/bbcu/bbcu.h:1487-1500)
//   Reduce                   include/bb/Reduce.h:200-220, 250-268           (no CUDA counterpart in the reference)
#include "common.cuh"

namespace bb200 {

// The mean loss over frames in one go: work[0] = sum of all targets, work[1] = sum of the per-frame losses, *loss = -work[1] / work[0].
// Up to kOneCta target values a single CTA does everything in one launch; above, three kernels share it and the sums go through `work`, which
// the caller clears (the clear and the launches are 14 us whatever the size).  One CTA / general on B200: 10 classes 8192 values 8.9 / 14.0 us,
// 16384 13.5 / 14.0, 24576 18.7 / 14.1, 32768 24.0 / 14.1; 2 classes 8192 9.5 / 13.9, 16384 16.1 / 13.7; 100 classes 16384 34.2 / 39.0, 24576
// 42.5 / 40.8.  (Before there was either, a read of the target sum by the host, three reductions and a kernel took 58 us of host time.)
constexpr int kOneCta = 1 << 14;

__device__ __forceinline__ double cta_sum(double v, double *red)
{
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const unsigned warps = blockDim.x >> 5;
    v = (threadIdx.x & 31) < warps ? red[threadIdx.x & 31] : 0.0;
#pragma unroll
    for (unsigned m = 16; m > 0; m >>= 1)
        if (m < warps) v += __shfl_xor_sync(0xffffffffu, v, m);
    return __shfl_sync(0xffffffffu, v, 0);
}

// one frame: softmax over the channel rows of every pixel, dy, and the frame's loss
__device__ __forceinline__ double softmax_frame(const float *__restrict__ y, const float *__restrict__ t, float *dy, float t_sum, int pix_size, int ch_size,
                                                int f, long long stride)
{
    const float eps = 1.0e-7f;
    double loss = 0.0;
    for (int pix = 0; pix < pix_size; ++pix) {
        float c = -3.402823466e+38f;
        for (int ch = 0; ch < ch_size; ++ch) c = fmaxf(c, y[(size_t)(ch * pix_size + pix) * stride + f]);
        float y_sum = 0.0f, t_max = 0.0f;
        for (int ch = 0; ch < ch_size; ++ch) {
            const size_t o = (size_t)(ch * pix_size + pix) * stride + f;
            y_sum += expf(y[o] - c);
            t_max += t[o];                       // one-hot targets: the sum is the frame's weight
        }
        if (y_sum <= eps) y_sum = eps;
        for (int ch = 0; ch < ch_size; ++ch) {
            const size_t o = (size_t)(ch * pix_size + pix) * stride + f;
            const float softmax = expf(y[o] - c) / y_sum;
            const float tv = t[o];
            if (tv > 0.0f) loss += (double)(logf(softmax + eps) * t_max);
            dy[o] = (t_max * softmax - tv) / t_sum;
        }
    }
    return loss;
}

__global__ void k_softmax_cross_entropy(const float *__restrict__ y, const float *__restrict__ t, float *dy, double *loss_buf, float t_sum,
                                        int pix_size, int ch_size, int F, long long stride)
{
    grid_dependency();
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f < F) loss_buf[f] = softmax_frame(y, t, dy, t_sum, pix_size, ch_size, f, stride);
}

__global__ void __launch_bounds__(1024)
k_softmax_cross_entropy_one(const float *__restrict__ y, const float *__restrict__ t, float *dy, double *loss, int pix_size, int ch_size, int F,
                            long long stride)
{
    grid_dependency();
    __shared__ double red[32];
    double s = 0.0;
    for (int row = threadIdx.x / 128; row < pix_size * ch_size; row += blockDim.x / 128)
        for (int f = threadIdx.x % 128; f < F; f += 128) s += (double)t[(size_t)row * stride + f];
    const double t_total = cta_sum(s, red);
    double l = 0.0;
    for (int f = threadIdx.x; f < F; f += blockDim.x) l += softmax_frame(y, t, dy, (float)t_total, pix_size, ch_size, f, stride);
    l = cta_sum(l, red);
    if (threadIdx.x == 0) *loss = -l / t_total;
}

// The same for one pixel, up to ROWS classes and a frame per thread: everything is read once, all loads of a frame in flight together, and a frame
// with one target above 0 takes one logarithm.  Latency is all there is to it (k_softmax_cross_entropy_one -> this, in us: 10 classes, 100 frames
// 6.7 -> 5.8, 512 7.8 -> 6.8, 1000 11.4 -> 9.3; 16 classes, 1000 frames 15.1 -> 12.2).  Every thread walks through all ROWS, so there are kernels
// for 4, 8 and 16: 3 classes, 1024 frames 5.5, with 16 rows 6.0, with 4 rows 5.1; 5 classes 6.6, 7.0, with 8 rows 5.5.
template <int ROWS>
__global__ void __launch_bounds__(1024)
k_softmax_cross_entropy_frames(const float *__restrict__ y, const float *__restrict__ t, float *dy, double *loss, int ch_size, int F, long long stride)
{
    grid_dependency();
    __shared__ double red[32];
    const float eps = 1.0e-7f;
    const int f = threadIdx.x;
    const bool live = f < F;
    float yv[ROWS], tv[ROWS];
#pragma unroll
    for (int ch = 0; ch < ROWS; ++ch) {
        const bool has = live && ch < ch_size;
        yv[ch] = has ? y[(size_t)ch * stride + f] : -3.402823466e+38f;
        tv[ch] = has ? t[(size_t)ch * stride + f] : 0.0f;
    }
    float c = -3.402823466e+38f, t_max = 0.0f;
    double s = 0.0;
    int above = 0;
#pragma unroll
    for (int ch = 0; ch < ROWS; ++ch) {
        c = fmaxf(c, yv[ch]);
        if (ch < ch_size) { t_max += tv[ch]; s += (double)tv[ch]; }
        above += tv[ch] > 0.0f ? 1 : 0;
    }
    const double t_total = cta_sum(s, red);
    const float t_sum = (float)t_total;
    float y_sum = 0.0f;
#pragma unroll
    for (int ch = 0; ch < ROWS; ++ch) {
        yv[ch] = ch < ch_size ? expf(yv[ch] - c) : 0.0f;
        if (ch < ch_size) y_sum += yv[ch];
    }
    if (y_sum <= eps) y_sum = eps;
    double l = 0.0;
    float picked = 1.0f;
#pragma unroll
    for (int ch = 0; ch < ROWS; ++ch) {
        if (ch >= ch_size) break;
        const float softmax = yv[ch] / y_sum;
        if (tv[ch] > 0.0f) {
            picked = softmax;
            if (above > 1) l += (double)(logf(softmax + eps) * t_max);
        }
        if (live) dy[(size_t)ch * stride + f] = (t_max * softmax - tv[ch]) / t_sum;
    }
    if (above == 1) l = (double)(logf(picked + eps) * t_max);
    l = cta_sum(l, red);
    if (threadIdx.x == 0) *loss = -l / t_total;
}

__global__ void __launch_bounds__(256)
k_target_sum(const float *__restrict__ t, double *work, int rows, int F, long long stride)
{
    grid_dependency();
    __shared__ double red[8];
    double s = 0.0;
    for (int row = blockIdx.y; row < rows; row += gridDim.y)
        for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < F; f += gridDim.x * blockDim.x) s += (double)t[(size_t)row * stride + f];
    s = cta_sum(s, red);
    if (threadIdx.x == 0) atomicAdd(work, s);
}

__global__ void __launch_bounds__(128)
k_softmax_cross_entropy_sums(const float *__restrict__ y, const float *__restrict__ t, float *dy, double *work, int pix_size, int ch_size, int F,
                             long long stride)
{
    grid_dependency();
    __shared__ double red[4];
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    double l = f < F ? softmax_frame(y, t, dy, (float)work[0], pix_size, ch_size, f, stride) : 0.0;
    l = cta_sum(l, red);
    if (threadIdx.x == 0) atomicAdd(work + 1, l);
}

__global__ void k_mean_loss(const double *__restrict__ work, double *loss) { grid_dependency(); *loss = -work[1] / work[0]; }

// dy = grad_reduction * (y - t);  loss_buf[block % loss_buf_size] += sum (y - t)^2 * loss_reduction  (NaN terms skipped)
__global__ void __launch_bounds__(256)
k_mean_squared_error(const float *__restrict__ y, const float *__restrict__ t, float *dy, double *loss_buf, int loss_buf_size, int F,
                     long long stride, float grad_reduction, double loss_reduction, int chunks)
{
    grid_dependency();
    __shared__ double red[8];
    const int node = blockIdx.x / chunks, chunk = blockIdx.x % chunks;
    const size_t row = (size_t)node * stride;
    const int f0 = chunk * 8192, f1 = min(F, f0 + 8192);
    double acc = 0.0;
    for (int f = f0 + threadIdx.x; f < f1; f += 256) {
        const float g = y[row + f] - t[row + f];
        dy[row + f] = g * grad_reduction;
        const float e = g * g;
        if (e == e) acc += (double)e;
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) s += red[w];
        atomicAdd(loss_buf + (blockIdx.x % loss_buf_size), s * loss_reduction);
    }
}

// y[o] = mean_i x[out_nodes * i + o]    /    dx[out_nodes * i + o] = dy[o] / mux
__global__ void k_reduce_forward(const float *__restrict__ x, float *y, int out_nodes, int mux, int F, long long xs, long long ys)
{
    grid_dependency();
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    const int o = blockIdx.y;
    if (f >= F) return;
    float sum = 0.0f;
    for (int i = 0; i < mux; ++i) sum += x[(size_t)(out_nodes * i + o) * xs + f];
    y[(size_t)o * ys + f] = sum / (float)mux;
}

__global__ void k_reduce_backward(const float *__restrict__ dy, float *dx, int out_nodes, int mux, int F, long long dys, long long dxs)
{
    grid_dependency();
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    const int o = blockIdx.y;
    if (f >= F) return;
    const float g = dy[(size_t)o * dys + f] / (float)mux;
    for (int i = 0; i < mux; ++i) dx[(size_t)(out_nodes * i + o) * dxs + f] = g;
}

}   // namespace bb200

using namespace bb200;

extern "C" int bbcu_fp32_LossSoftmaxCrossEntropy(const float *y, const float *t, float *dy, double *loss_buf, float t_sum, int pix_size,
                                                 int ch_size, int frame_size, int frame_stride, bbcu_stream_t stream)
{
    BB200_REQUIRE_PTR(y); BB200_REQUIRE_PTR(t); BB200_REQUIRE_PTR(dy); BB200_REQUIRE_PTR(loss_buf);
    BB200_REQUIRE(pix_size > 0 && ch_size > 0 && frame_size >= 0, BBCU_ERR_BAD_SIZE);
    BB200_REQUIRE(frame_stride >= frame_size, BBCU_ERR_BAD_STRIDE);
    if (frame_size == 0) return BBCU_OK;
    launch(k_softmax_cross_entropy, (frame_size + 127) / 128, 128, 0, as_stream(stream), y, t, dy, loss_buf, t_sum, pix_size, ch_size, frame_size,
                                                                                   frame_stride);
    return launch_status();
}

extern "C" int bbcu_fp32_LossSoftmaxCrossEntropyMean(const float *y, const float *t, float *dy, double *loss, int pix_size, int ch_size, int frame_size,
                                                     int frame_stride, bbcu_stream_t stream)
{
    BB200_REQUIRE_PTR(y); BB200_REQUIRE_PTR(t); BB200_REQUIRE_PTR(dy); BB200_REQUIRE_PTR(loss);
    BB200_REQUIRE(pix_size > 0 && ch_size > 0 && frame_size >= 0, BBCU_ERR_BAD_SIZE);
    BB200_REQUIRE(frame_stride >= frame_size, BBCU_ERR_BAD_STRIDE);
    cudaStream_t st = as_stream(stream);
    const long long rows = (long long)pix_size * ch_size;
    BB200_REQUIRE(rows < (1LL << 31), BBCU_ERR_TOO_LARGE);
    double *work = rows * frame_size <= kOneCta ? nullptr : static_cast<double *>(stream_scratch(st, 2 * sizeof(double)));
    if (pix_size == 1 && ch_size <= 16 && frame_size <= 1024) {
        const int threads = frame_size > 32 ? (frame_size + 31) / 32 * 32 : 32;
        auto kern = ch_size <= 4 ? k_softmax_cross_entropy_frames<4> : ch_size <= 8 ? k_softmax_cross_entropy_frames<8> : k_softmax_cross_entropy_frames<16>;
        launch(kern, 1, threads, 0, st, y, t, dy, loss, ch_size, frame_size, frame_stride);
        return launch_status();
    }
    if (work == nullptr) {                                    // (a heap that declines it: slower, not an error)
        launch(k_softmax_cross_entropy_one, 1, 1024, 0, st, y, t, dy, loss, pix_size, ch_size, frame_size, frame_stride);
        return launch_status();
    }
    BB200_CUDA(cudaMemsetAsync(work, 0, 2 * sizeof(double), st));
    const unsigned bx = (unsigned)((frame_size + 2047) / 2048);
    launch(k_target_sum, dim3(bx, (unsigned)(rows < 64 ? rows : 64)), 256, 0, st, t, work, (int)rows, frame_size, frame_stride);
    BB200_CUDA(cudaPeekAtLastError());
    launch(k_softmax_cross_entropy_sums, (frame_size + 127) / 128, 128, 0, st, y, t, dy, work, pix_size, ch_size, frame_size, frame_stride);
    BB200_CUDA(cudaPeekAtLastError());
    launch(k_mean_loss, 1, 1, 0, st, work, loss);
    return launch_status();
}

extern "C" int bbcu_fp32_LossMeanSquaredError(const float *y, const float *t, float *dy, double *loss_buf, int loss_buf_size, int node_size,
                                              int frame_size, int frame_stride, float grad_reduction, double loss_reduction,
                                              bbcu_stream_t stream)
{
    BB200_REQUIRE_PTR(y); BB200_REQUIRE_PTR(t); BB200_REQUIRE_PTR(dy); BB200_REQUIRE_PTR(loss_buf);
    BB200_REQUIRE(loss_buf_size > 0 && node_size >= 0 && frame_size >= 0, BBCU_ERR_BAD_SIZE);
    BB200_REQUIRE(frame_stride >= frame_size, BBCU_ERR_BAD_STRIDE);
    if (node_size == 0 || frame_size == 0) return BBCU_OK;
    const int chunks = (frame_size + 8191) / 8192;
    BB200_REQUIRE((long long)node_size * chunks < (1LL << 31), BBCU_ERR_TOO_LARGE);
    launch(k_mean_squared_error, node_size * chunks, 256, 0, as_stream(stream), y, t, dy, loss_buf, loss_buf_size, frame_size, frame_stride,
                                                                          grad_reduction, loss_reduction, chunks);
    return launch_status();
}

extern "C" int bbcu_fp32_Reduce_Forward(const float *x, float *y, int input_node_size, int output_node_size, int frame_size,
                                        int x_frame_stride, int y_frame_stride, bbcu_stream_t stream)
{
    BB200_REQUIRE_PTR(x); BB200_REQUIRE_PTR(y);
    BB200_REQUIRE(output_node_size > 0 && input_node_size >= output_node_size && input_node_size % output_node_size == 0 && frame_size >= 0 &&
                  output_node_size <= 65535, BBCU_ERR_BAD_SIZE);
    BB200_REQUIRE(x_frame_stride >= frame_size && y_frame_stride >= frame_size, BBCU_ERR_BAD_STRIDE);
    if (frame_size == 0) return BBCU_OK;
    launch(k_reduce_forward, dim3((frame_size + 255) / 256, output_node_size), 256, 0, as_stream(stream),
        x, y, output_node_size, input_node_size / output_node_size, frame_size, x_frame_stride, y_frame_stride);
    return launch_status();
}

extern "C" int bbcu_fp32_Reduce_Backward(const float *dy, float *dx, int input_node_size, int output_node_size, int frame_size,
                                         int dy_frame_stride, int dx_frame_stride, bbcu_stream_t stream)
{
    BB200_REQUIRE_PTR(dy); BB200_REQUIRE_PTR(dx);
    BB200_REQUIRE(output_node_size > 0 && input_node_size >= output_node_size && input_node_size % output_node_size == 0 && frame_size >= 0 &&
                  output_node_size <= 65535, BBCU_ERR_BAD_SIZE);
    BB200_REQUIRE(dy_frame_stride >= frame_size && dx_frame_stride >= frame_size, BBCU_ERR_BAD_STRIDE);
    if (frame_size == 0) return BBCU_OK;
    launch(k_reduce_backward, dim3((frame_size + 255) / 256, output_node_size), 256, 0, as_stream(stream),
        dy, dx, output_node_size, input_node_size / output_node_size, frame_size, dy_frame_stride, dx_frame_stride);
    return launch_status();
}
