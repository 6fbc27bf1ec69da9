// Host-side helpers shared by the operator launchers: argument checks, launch-error capture,
// per-stream scratch memory and the frame-tile heuristic.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include "../../include/bbcu_b200.h"

namespace bb200 {

#define BB200_REQUIRE_PTR(p)   do { if ((p) == nullptr) return BBCU_ERR_NULL_POINTER; } while (0)
#define BB200_REQUIRE(cond, e) do { if (!(cond)) return (e); } while (0)
#define BB200_CUDA(call)       do { cudaError_t e_ = (call); if (e_ != cudaSuccess) { cudaGetLastError(); return (int)e_; } } while (0)

constexpr int kFramesPerIterHost = 128;   // frames one warp covers per iteration (32 lanes x 4)

// Status of the launches just made: a launch error is reported once and cleared, so it cannot resurface in a later call.
inline int launch_status() { return (int)cudaGetLastError(); }

// Device properties read once per device.
struct DeviceInfo {
    int sm_count;
    size_t l2_bytes;
    size_t total_bytes;          // device memory
};
const DeviceInfo &device_info();

// Scratch memory private to (device, stream): grows on demand through the device heap, is reused by
// later calls on the same stream and is released by bbcu_LocalHeap_GarbageCollect().  Stream order
// makes back-to-back calls on one stream safe; different streams get different blocks.  A stream has
// kScratchSlots independent blocks, for callers whose scratch is alive at the same time (slot 0: batch-norm
// sums, slot 1: per-node coefficient / pattern tables of the LUT operators, slot 2: the piece table of the bit Im2Col,
// slot 3: fp32 rows packed to bits).
constexpr int kScratchSlots = 5;
void *stream_scratch(cudaStream_t stream, size_t bytes, int slot = 0);

// A number that is another one after every request for the stream's block (0: it has none).  A caller that leaves something in the block for
// a later call of its own compares it: equal means that nobody has been handed the block since.
unsigned long long stream_scratch_ticket(cudaStream_t stream, int slot);

// 64 counters of the stream (slot 4), zeroed when they are made; a kernel that uses them leaves them zero.  nullptr when they cannot be had,
// for the per-thread default stream, whose one handle stands for a stream of every thread, and for a stream that is being captured: the
// graph may be launched on any stream, beside kernels of this one, and the zeroing would only be a node of the graph.
unsigned *stream_counters(cudaStream_t stream);

// Pass 1 of the DifferentiableLut6 training forward (raw LUT values into y, fp64 sums per node); with may_allocate = false
// it takes nothing from the heap or the stream scratch.
int dl6_forward_stats(const float *x, float *y, const int *idx, const float *W, double *dev_sums, float unbinarize_bias, int node_size,
                      int frame_size, int frame_stride, int lut_binarize, int binary_mode, bool may_allocate, cudaStream_t st);

// Frames handled by one CTA pass.  The gathered input rows of a frame tile (and, in the backward
// pass, the dx rows it reduces into) have to stay resident in L2 while every output node of the
// layer consumes them, so the tile narrows as the layer widens; it widens again, up to max_tile,
// while that still leaves enough CTAs to fill the machine.
int frame_tile(long long rows_touched, int bits_per_row_frame, int node_groups, int frame_size, int max_tile);

// Bit-in / bit-out LUT layers evaluated through a per-node pattern table and the BinaryLut6 kernel (binary_mode.cu).  Both return
// BBCU_ERR_NO_MEMORY when their scratch cannot be had, in which case the caller runs the per-frame kernels instead.
int bit_forward_by_table(bool with_bn, const int *x, int *y, const int *idx, const float *W, const float *rmean, const float *rvar, float gamma,
                         float beta, float bias, int O, int F, int stride, int lut_binarize, cudaStream_t st);
int dl6_bit_forward_training_by_table(const int *x, int *y, const int *idx, const float *W, float *mean, float *rstd, float *rmean, float *rvar,
                                      float gamma, float beta, float momentum, float bias, int O, int F, int stride, int lut_binarize,
                                      cudaStream_t st);

int bit_fp32_forward_by_table(const int *x, float *y, const int *idx, const float *W, float bias, int O, int F, long long xs, long long ys,
                              int lut_binarize, cudaStream_t st);

int bit_backward_by_table(bool bn, bool x_is_fp32, const void *x, const float *dy, float *dx, const int *idx, const float *W, float *dW,
                          const float *mean, const float *rstd, float *dmean_out, float *dvar_out, float gamma, float beta, float bias, int I, int O,
                          int F, long long xs, long long fs, int lut_binarize, cudaStream_t st);

// The batch-norm backward of a binary-mode layer on fp32 frames in two halves for frame-sharded callers (the caller adds `sums` over the
// ranks in between); both decline with BBCU_ERR_NO_MEMORY like the calls above.
int bit_backward_stats_by_table(const float *x, const float *dy, const int *idx, const float *W, const float *mean, const float *rstd, double *sums,
                                float gamma, float beta, float bias, int O, int F, long long fs, int lut_binarize, cudaStream_t st);
int bit_backward_apply_by_table(const float *x, const float *dy, float *dx, const int *idx, const float *W, float *dW, const float *mean,
                                const float *rstd, const double *sums, float *dmean_out, float *dvar_out, float gamma, float beta, float bias, int I,
                                int O, int F, long long fs, long long total_frames, int lut_binarize, cudaStream_t st);

// The training forward of a binary-mode layer on I fp32 rows through packed rows; declines (layers where it does not pay, no scratch) like the others.
int f32_binary_forward_packed(const float *x, float *y, const int *idx, const float *W, float *mean, float *rstd, float *rmean, float *rvar,
                              float gamma, float beta, float momentum, float bias, int I, int O, int F, long long fs, int lut_binarize,
                              cudaStream_t st);
int f32_binary_forward_by_table(int mode, const float *x, float *y, const int *idx, const float *W, float *mean, float *rstd, float *rmean,
                                float *rvar, float gamma, float beta, float momentum, float bias, int O, int F, long long fs, int lut_binarize,
                                cudaStream_t st);

// Small layers in probability mode, one launch per direction (lut6_small.cu).  All rows share the frame stride fs; vec: x, y, dy and dx rows
// start on 16-byte boundaries.  small_forward(): mode 0 y = clip(LUT), 1 training with batch norm, 2 inference (mean_in, and the running
// variance in rstd_in); small_backward() clears dx and adds to dW.
struct SmallLayerArgs {
    const float *x, *dy, *W, *mean_in, *rstd_in;
    const int *idx;
    float *y, *dx, *dW, *mean, *rstd, *running_mean, *running_var, *dmean, *dvar;
    float gamma, beta, momentum;
    int F, lut_binarize, vec;
    long long fs;
};
constexpr long long kSmallProbability = BBCU_B200_SMALL_NODE_FRAMES;       // see small_probability_layer()
bool small_probability_layer(int O, int F);

// Threads of the one-launch kernels, whose CTA is a node with all of its frames (four a lane and round): a warp for every 128 frames, up to
// eight, or fewer that take several rounds, so that more nodes share an SM and the layer takes fewer waves of CTAs.  A wave costs `fixed` and each of its
// rounds `per_round`; `sm_warps`: warps of the kernel that an SM holds (at least eight).
unsigned small_layer_threads(int O, int F, int sm_warps, int fixed, int per_round);
int small_forward(int mode, const SmallLayerArgs &a, int O, cudaStream_t st);
int small_backward(bool bn, const SmallLayerArgs &a, int I, int O, cudaStream_t st);

// Per-device int in the library's device image (zero until a kernel records a fault); nothing is allocated for it.
int *fault_word();

// Opt-in to more than 48 KB of dynamic shared memory, once per kernel and device (the attribute stays set, the call costs about as much
// as a small launch).  False when it is refused.
bool allow_big_smem_once(const void *kernel, int bytes);
template <typename K> inline bool allow_big_smem(K *kernel, int bytes) { return allow_big_smem_once(reinterpret_cast<const void *>(kernel), bytes); }

// Every kernel starts with grid_dependency() and every launch goes through launch(): the next kernel of the stream is then set up while
// the last blocks of this one still run, and waits here until all that came before it is finished and visible.  A pass is a chain of
// kernels of some microseconds, and the gaps between them were a tenth to a fifth of it (frozen LUT-CNN, 28 launches: 279 -> 222 us;
// modulated network, 19: 190 -> 154 us; training step of the LUT-CNN, 126: 4778 -> 4609 us).  Without an early trigger on purpose: blocks
// that wait take the places of others unevenly (252, 160 and 4664 us with one at the start of every kernel).
__device__ __forceinline__ void grid_dependency()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

inline cudaStream_t as_stream(bbcu_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

}   // namespace bb200
