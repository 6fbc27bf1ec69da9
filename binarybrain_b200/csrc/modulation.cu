// Binary modulation around a LUT network: RealToBinary turns one fp32 frame into frame_mod
// bit frames by comparing against a threshold per output frame, BinaryToReal integrates bit frames back into fp32.
//
// Semantics follow the reference's CPU branches:
//   RealToBinary  include/bb/RealToBinary.h:309-345 (deterministic thresholds), :352-398 (thresholds from a value generator;
//                 here the caller passes them, because the reference draws them on the host)
//   BinaryToReal  include/bb/BinaryToReal.h:247-276 (forward), :312-330 (backward)
#include "common.cuh"

namespace bb200 {

// Block = one output node x kR2bFrames output frames; a thread takes every 256th frame, a warp's ballot is one word of bits.  The
// thresholds (4 bytes per output frame) are the traffic; everything that depends on the node only, and the division of an output frame
// into (input frame, modulation step), is done once per thread and advanced by addition, because one thread per output
// frame with its own divisions was bound by them (3072 nodes x 1792 frames: 35 us, floor 3.6 us).  PLAIN: thresholds given, no depth
// modulation -- the usual call; without the code of the others 17 -> 14 us.
constexpr int kR2bSteps = 8, kR2bFrames = 256 * kR2bSteps;

template <bool PLAIN>
__global__ void __launch_bounds__(256)
k_real_to_binary_bit(const float *__restrict__ x, uint32_t *y, const float *__restrict__ th, unsigned depth_mod, unsigned frame_mod, float lo,
                     float hi, unsigned point_size, unsigned x_frame_size, long long xs, long long ys, long long ths)
{
    grid_dependency();
    const unsigned node = blockIdx.y;                                  // output node = (input_depth * depth_mod + d) * point_size + p
    const unsigned out_frames = x_frame_size * frame_mod;
    unsigned of = blockIdx.x * kR2bFrames + threadIdx.x;               // output frame = fi * frame_mod + f
    unsigned d = 0, row = node;
    if (!PLAIN) {
        const unsigned p = node % point_size, od = node / point_size, in_depth = od / depth_mod;
        d = od % depth_mod;
        row = in_depth * point_size + p;
    }
    const float *xrow = x + (size_t)row * xs;
    const float *trow = th == nullptr ? nullptr : th + (size_t)row * ths;
    const float depth_step = 1.0f / (float)depth_mod, frame_step = 1.0f / (float)frame_mod, scale = 1.0f / (hi - lo);
    unsigned fi = of / frame_mod, f = of - fi * frame_mod;
    const unsigned di = 256u / frame_mod, df = 256u - di * frame_mod;
    float xv[kR2bSteps], tv[kR2bSteps];
    unsigned fs[kR2bSteps];
#pragma unroll
    for (int k = 0; k < kR2bSteps; ++k) {
        const bool live = of + 256u * k < out_frames;
        xv[k] = live ? __ldg(xrow + fi) : 0.0f;
        tv[k] = live && (PLAIN || trow != nullptr) ? __ldg(trow + of + 256u * k) : 0.0f;
        fs[k] = f;
        fi += di;
        f += df;
        if (f >= frame_mod) { f -= frame_mod; ++fi; }
    }
#pragma unroll
    for (int k = 0; k < kR2bSteps; ++k, of += 256u) {
        bool bit = false;
        if (of < out_frames) {
            float v = (xv[k] - lo) * scale;
            if (!PLAIN) v = (v - (float)d * depth_step) * (float)depth_mod;
            if (PLAIN || th != nullptr) {
                bit = v > tv[k];
            } else {
                v = (v - (float)fs[k] * frame_step) * (float)frame_mod;
                v = fmaxf(0.0f, fminf(1.0f, v));
                bit = v > 0.5f;
            }
        }
        const unsigned word = __ballot_sync(0xffffffffu, bit);
        if ((threadIdx.x & 31) == 0 && of < out_frames) y[(size_t)node * ys + (of >> 5)] = word;
    }
}

// y[f][n] = mean over i < node_mux, j < frame_mux of bit x[f * frame_mux + j][n + i * y_nodes]
// Block = one output node x 32 output frames, i.e. 32 * frame_mux consecutive input frames of node_mux rows; its warps share the rows, a
// lane counts its input frames (lane + 32 m) over the warp's rows in registers, and the counts meet in shared memory.  The counts are whole
// numbers, so the order of addition does not show.  (One thread per output value walked its node_mux * frame_mux inputs alone: 1020 x 1792 ->
// 10 x 256 took 43 us on 2560 threads; the rows are 7.3 MB.)  8 to 32 warps, a row each while there are enough: there are few blocks, and 13
// rows one after the other took a warp 14 us for that size, 8.6 us now.
constexpr int kB2rSteps = 8;

template <bool XBIT>
__global__ void __launch_bounds__(1024)
k_binary_to_real_forward(const void *x, float *y, int node_mux, int frame_mux, int y_nodes, long long xs, int y_frames, long long ys)
{
    grid_dependency();
    __shared__ int s_cnt[32 * kB2rSteps];                              // counts of a run of input frames
    __shared__ int s_out[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int n = blockIdx.y, f0 = blockIdx.x * 32;
    const long long x_begin = (long long)f0 * frame_mux, x_end = (long long)min(y_frames, f0 + 32) * frame_mux;
    if (threadIdx.x < 32) s_out[threadIdx.x] = 0;
    for (int m0 = 0; m0 < frame_mux; m0 += kB2rSteps) {
        const int m_end = min(kB2rSteps, frame_mux - m0);
        if (threadIdx.x < 32 * kB2rSteps) s_cnt[threadIdx.x] = 0;
        __syncthreads();
        int acc[kB2rSteps];
#pragma unroll
        for (int m = 0; m < kB2rSteps; ++m) acc[m] = 0;
        for (int i = warp; i < node_mux; i += warps) {
            const size_t row = (size_t)(n + (size_t)i * y_nodes) * xs;
#pragma unroll
            for (int m = 0; m < kB2rSteps; ++m) {
                const long long xf = x_begin + 32 * (m0 + m) + lane;
                if (m < m_end && xf < x_end) {
                    if (XBIT) acc[m] += (__ldg(static_cast<const uint32_t *>(x) + row + (xf >> 5)) >> lane) & 1u;      // x_begin is a multiple of 32
                    else      acc[m] += __ldg(static_cast<const float *>(x) + row + xf) > 0.0f ? 1 : 0;
                }
            }
        }
#pragma unroll
        for (int m = 0; m < kB2rSteps; ++m)
            if (acc[m]) atomicAdd(&s_cnt[32 * m + lane], acc[m]);
        __syncthreads();
        const int k = 32 * m0 + (int)threadIdx.x;                      // input frame relative to x_begin
        if ((int)threadIdx.x < 32 * m_end && s_cnt[threadIdx.x]) atomicAdd(&s_out[k / frame_mux], s_cnt[threadIdx.x]);
        __syncthreads();
    }
    if (threadIdx.x < 32 && f0 + (int)threadIdx.x < y_frames)
        y[(size_t)n * ys + f0 + threadIdx.x] = (float)s_out[threadIdx.x] / (float)(node_mux * frame_mux);
}

// dx[f * frame_mux + j][n + i * y_nodes] = dy[f][n] * y_nodes / (x_nodes * frame_mux)
// Four consecutive input frames per thread: one division, and one 128-bit store where the rows are aligned (`vec`).
__global__ void __launch_bounds__(256)
k_binary_to_real_backward(const float *__restrict__ dy, float *dx, int node_mux, int frame_mux, int y_nodes, long long xs, int y_frames, long long ys,
                          int vec)
{
    grid_dependency();
    const long long x_frames = (long long)y_frames * frame_mux;
    const long long xf = 4 * ((long long)blockIdx.x * blockDim.x + threadIdx.x);
    const int xn = blockIdx.y;
    if (xf >= x_frames) return;
    const float gain = (float)y_nodes / ((float)(y_nodes * node_mux) * (float)frame_mux);
    const float *row = dy + (size_t)(xn % y_nodes) * ys;
    unsigned f = (unsigned)xf / (unsigned)frame_mux, j = (unsigned)xf - f * (unsigned)frame_mux;       // x strides are ints: xf fits
    float g[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        g[i] = f < (unsigned)y_frames ? __ldg(row + f) * gain : 0.0f;
        if (++j == (unsigned)frame_mux) { j = 0; ++f; }
    }
    float *out = dx + (size_t)xn * xs + xf;
    if (vec && xf + 3 < x_frames) {
        *reinterpret_cast<float4 *>(out) = make_float4(g[0], g[1], g[2], g[3]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (xf + i < x_frames) out[i] = g[i];
    }
}

}   // namespace bb200

using namespace bb200;

extern "C" int bbcu_bit_fp32_RealToBinary_Forward(const float *x, int *y, const float *dev_thresholds, int threshold_frame_stride,
                                                  unsigned depth_modulation_size, unsigned frame_modulation_size, float input_range_lo,
                                                  float input_range_hi, unsigned point_size, unsigned x_depth_size, unsigned x_frame_size,
                                                  unsigned x_frame_stride, unsigned y_frame_stride, bbcu_stream_t stream)
{
    BB200_REQUIRE_PTR(x); BB200_REQUIRE_PTR(y);
    BB200_REQUIRE(depth_modulation_size > 0 && frame_modulation_size > 0 && point_size > 0 && input_range_hi != input_range_lo, BBCU_ERR_BAD_SIZE);
    const unsigned long long out_frames = (unsigned long long)x_frame_size * frame_modulation_size;
    const unsigned long long out_nodes = (unsigned long long)x_depth_size * depth_modulation_size * point_size;
    BB200_REQUIRE(out_frames < (1ull << 31) && out_nodes <= 65535ull * 64, BBCU_ERR_TOO_LARGE);
    BB200_REQUIRE(x_frame_stride >= x_frame_size && (unsigned long long)y_frame_stride * 32 >= out_frames, BBCU_ERR_BAD_STRIDE);
    BB200_REQUIRE(dev_thresholds == nullptr || (unsigned long long)threshold_frame_stride >= out_frames, BBCU_ERR_BAD_STRIDE);
    if (out_frames == 0 || out_nodes == 0) return BBCU_OK;
    BB200_REQUIRE(out_nodes <= 65535, BBCU_ERR_TOO_LARGE);
    auto kern = dev_thresholds != nullptr && depth_modulation_size == 1 ? k_real_to_binary_bit<true> : k_real_to_binary_bit<false>;
    launch(kern, dim3((unsigned)((out_frames + kR2bFrames - 1) / kR2bFrames), (unsigned)out_nodes), 256, 0, as_stream(stream),
        x, reinterpret_cast<uint32_t *>(y), dev_thresholds, depth_modulation_size, frame_modulation_size, input_range_lo, input_range_hi, point_size,
        x_frame_size, x_frame_stride, y_frame_stride, threshold_frame_stride);
    return launch_status();
}

static int b2r_check(const void *x, const void *y, int node_mux, int frame_mux, int y_nodes, int x_stride, int y_frames, int y_stride, bool xbit)
{
    BB200_REQUIRE_PTR(x); BB200_REQUIRE_PTR(y);
    BB200_REQUIRE(node_mux > 0 && frame_mux > 0 && y_nodes > 0 && y_nodes <= 65535 && y_frames >= 0, BBCU_ERR_BAD_SIZE);
    BB200_REQUIRE((long long)y_nodes * node_mux <= 65535, BBCU_ERR_TOO_LARGE);
    BB200_REQUIRE(y_stride >= y_frames && (long long)x_stride * (xbit ? 32 : 1) >= (long long)y_frames * frame_mux, BBCU_ERR_BAD_STRIDE);
    return BBCU_OK;
}

static int b2r_threads(int node_mux) { return 32 * (node_mux < 8 ? 8 : node_mux > 32 ? 32 : node_mux); }

extern "C" int bbcu_bit_fp32_BinaryToReal_Forward(const int *x, float *y, int node_mux_size, int frame_mux_size, int y_node_size,
                                                  int x_frame_stride, int y_frame_size, int y_frame_stride, bbcu_stream_t stream)
{
    int rc = b2r_check(x, y, node_mux_size, frame_mux_size, y_node_size, x_frame_stride, y_frame_size, y_frame_stride, true);
    if (rc || y_frame_size == 0) return rc;
    launch(k_binary_to_real_forward<true>, dim3((y_frame_size + 31) / 32, y_node_size), b2r_threads(node_mux_size), 0, as_stream(stream),
        x, y, node_mux_size, frame_mux_size, y_node_size, x_frame_stride, y_frame_size, y_frame_stride);
    return launch_status();
}

extern "C" int bbcu_fp32_BinaryToReal_Forward(const float *x, float *y, int node_mux_size, int frame_mux_size, int y_node_size,
                                              int x_frame_stride, int y_frame_size, int y_frame_stride, bbcu_stream_t stream)
{
    int rc = b2r_check(x, y, node_mux_size, frame_mux_size, y_node_size, x_frame_stride, y_frame_size, y_frame_stride, false);
    if (rc || y_frame_size == 0) return rc;
    launch(k_binary_to_real_forward<false>, dim3((y_frame_size + 31) / 32, y_node_size), b2r_threads(node_mux_size), 0, as_stream(stream),
        x, y, node_mux_size, frame_mux_size, y_node_size, x_frame_stride, y_frame_size, y_frame_stride);
    return launch_status();
}

extern "C" int bbcu_fp32_BinaryToReal_Backward(const float *dy, float *dx, int node_mux_size, int frame_mux_size, int y_node_size,
                                               int x_frame_stride, int y_frame_size, int y_frame_stride, bbcu_stream_t stream)
{
    int rc = b2r_check(dy, dx, node_mux_size, frame_mux_size, y_node_size, x_frame_stride, y_frame_size, y_frame_stride, false);
    if (rc || y_frame_size == 0) return rc;
    const long long xf = (long long)y_frame_size * frame_mux_size;
    const int vec = (reinterpret_cast<uintptr_t>(dx) & 15) == 0 && x_frame_stride % 4 == 0;
    launch(k_binary_to_real_backward, dim3((unsigned)((xf + 1023) / 1024), y_node_size * node_mux_size), 256, 0, as_stream(stream),
        dy, dx, node_mux_size, frame_mux_size, y_node_size, x_frame_stride, y_frame_size, y_frame_stride, vec);
    return launch_status();
}
