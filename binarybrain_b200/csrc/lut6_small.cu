// Small LUT layers on fp32 frames in probability mode: one launch per direction.
//
// The persistent kernels of lut6_layers.cu need a table conversion in front, cleared sums, a finalise and a normalise pass behind: five to
// eight launches of 2-3 us each, which is all there is to a layer of a few hundred nodes on a few hundred frames.  Here one CTA is
// one node with all of its frames (1 to 8 warps, four consecutive frames per lane and round): table conversion, LUT values, batch
// statistics and output -- or batch sums, gradients and the table gradient -- without leaving the SM.  Bound by latency (wiring, then
// rows, then the reductions), not by throughput, so larger layers do not come here (small_probability_layer()).
//
// The LUT evaluation and its reverse pass are those of the persistent kernels (lut6_core.cuh), so a layer gives the same LUT values whichever
// way it runs; the batch-norm gradient is rounded differently (three products and two sums here, two fused multiply-adds there), and the sums
// over frames are taken in another order.  Semantics: include/bb/DifferentiableLutN.h:747-905 (forward), :1157-1266 (backward),
// include/bb/StochasticLutN.h:512-559, :668-752.
#include "common.cuh"
#include "async_copy.cuh"
#include "lut6_core.cuh"
#include "grid_clear.cuh"

namespace bb200 {

namespace {

enum { kSmallPlain = 0, kSmallTrain = 1, kSmallInfer = 2 };

// four consecutive frames of a row; frames from F on read as 0
__device__ __forceinline__ float4 load4(const float *row, int f, int F, int vec)
{
    if (vec && f + 3 < F) return __ldg(reinterpret_cast<const float4 *>(row + f));
    return make_float4(f < F ? __ldg(row + f) : 0.0f, f + 1 < F ? __ldg(row + f + 1) : 0.0f, f + 2 < F ? __ldg(row + f + 2) : 0.0f,
                       f + 3 < F ? __ldg(row + f + 3) : 0.0f);
}

__device__ __forceinline__ float centred(float v) { return __saturatef(v) - 0.5f; }           // condition_u() in probability mode

template <int MODE>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
k_lut6_small_forward(const SmallLayerArgs a)
{
    grid_dependency();
    extern __shared__ __align__(16) float s_raw[];                                             // kSmallTrain: the node's raw values
    __shared__ float4 s_tab[32];
    __shared__ double s_sum[kWarpsPerCta][2];
    __shared__ float s_stat[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, node = blockIdx.x;
    const float *rows[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) rows[j] = a.x + (size_t)__ldg(a.idx + (size_t)node * 6 + j) * a.fs;
    int f = 4 * (int)threadIdx.x;
    float4 xq[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) xq[j] = load4(rows[j], f, a.F, a.vec);                          // under way while the table is converted
    if (warp == 0) stage_table_x2(s_tab, a.W, node, lane, a.lut_binarize);
    float mean = 0.0f, rstd = 0.0f;
    if (MODE == kSmallInfer) {
        mean = a.mean_in[node];
        rstd = 1.0f / sqrtf(a.rstd_in[node]);                                                  // the running variance, DifferentiableLutN.h:866-868
    }
    __syncthreads();
    double s1 = 0.0, s2 = 0.0;
    float *yrow = a.y + (size_t)node * a.fs;
    auto store = [&](int at, const float (&v)[4]) {
        if (a.vec && at + 3 < a.F) {
            *reinterpret_cast<float4 *>(yrow + at) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (at + i < a.F) yrow[at + i] = v[i];
        }
    };
    const int step = 4 * (int)blockDim.x;
    for (; f < a.F; f += step) {
        f32x2 up[6][2], yp[2];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            up[j][0] = pack2(centred(xq[j].x), centred(xq[j].y));
            up[j][1] = pack2(centred(xq[j].z), centred(xq[j].w));
        }
        if (f + step < a.F) {
#pragma unroll
            for (int j = 0; j < 6; ++j) xq[j] = load4(rows[j], f + step, a.F, a.vec);
        }
        lut6_forward_x2<2>(s_tab, up, yp);
        float v[4];
        unpack2(yp[0], v[0], v[1]);
        unpack2(yp[1], v[2], v[3]);
        if (MODE == kSmallTrain) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (f + i < a.F) { s1 += (double)v[i]; s2 += (double)v[i] * (double)v[i]; }
            *reinterpret_cast<float4 *>(s_raw + f) = make_float4(v[0], v[1], v[2], v[3]);       // (padded to whole rounds)
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (MODE == kSmallInfer) { v[i] = (v[i] - mean) * rstd; v[i] = v[i] * a.gamma + a.beta; }
                v[i] = __saturatef(v[i]);
            }
            store(f, v);
        }
    }
    if (MODE == kSmallTrain) {
        s1 = warp_sum(s1);
        s2 = warp_sum(s2);
        if (lane == 0) { s_sum[warp][0] = s1; s_sum[warp][1] = s2; }
        __syncthreads();
        if (threadIdx.x == 0) {                                                                // as k_bn_finalize
            double t1 = 0.0, t2 = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { t1 += s_sum[w][0]; t2 += s_sum[w][1]; }
            const float rF  = 1.0f / (float)a.F;
            const float m   = (float)t1 * rF;
            const float var = fmaxf(1.0e-5f, fmaf((float)t2, rF, -(m * m)));
            const float r   = 1.0f / sqrtf(var);
            a.running_mean[node] = a.running_mean[node] * a.momentum + m * (1.0f - a.momentum);
            a.running_var[node]  = a.running_var[node]  * a.momentum + var * (1.0f - a.momentum);
            a.mean[node] = m;
            a.rstd[node] = r;
            s_stat[0] = m;
            s_stat[1] = r;
        }
        __syncthreads();
        mean = s_stat[0];
        rstd = s_stat[1];
        for (f = 4 * (int)threadIdx.x; f < a.F; f += step) {                                   // a thread reads back what it wrote
            const float4 q = *reinterpret_cast<const float4 *>(s_raw + f);
            float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float t = (v[i] - mean) * rstd;
                t = t * a.gamma + a.beta;
                v[i] = fmaxf(0.0f, fminf(1.0f, t));
            }
            store(f, v);
        }
    }
}

// dx is cleared on the way (`clear`), or by the launcher; dW is accumulated into.
template <bool BN>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 1)
k_lut6_small_backward(const SmallLayerArgs a, const GridClear clear)
{
    grid_dependency();
    __shared__ float4 s_tab[16];
    __shared__ double s_sum[kWarpsPerCta][2];
    __shared__ float s_stat[2];
    __shared__ float s_dc[kWarpsPerCta][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, node = blockIdx.x, warps = blockDim.x >> 5;
    const float *rows[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) rows[j] = a.x + (size_t)__ldg(a.idx + (size_t)node * 6 + j) * a.fs;
    const float *dyrow = a.dy + (size_t)node * a.fs;
    const int step = 4 * (int)blockDim.x;
    int f = 4 * (int)threadIdx.x;
    float4 xq[6], gq;
    auto fetch = [&](int at) {
#pragma unroll
        for (int j = 0; j < 6; ++j) xq[j] = load4(rows[j], at, a.F, a.vec);
        gq = load4(dyrow, at, a.F, a.vec);
    };
    auto input = [&](float (&u)[6], int i) {
#pragma unroll
        for (int j = 0; j < 6; ++j) u[j] = centred(i == 0 ? xq[j].x : i == 1 ? xq[j].y : i == 2 ? xq[j].z : xq[j].w);
    };
    fetch(f);
    if (warp == 0) stage_table_halves(s_tab, a.W, node, lane, a.lut_binarize);
    grid_clear_slices(clear);
    float mean = 0.0f, rstd = 0.0f, dmean = 0.0f, dvar = 0.0f;
    const float rF = 1.0f / (float)a.F;
    if (BN) { mean = a.mean_in[node]; rstd = a.rstd_in[node]; }
    __syncthreads();
    if (BN) {                                                                                  // the two batch sums, as k_lut6_backward_stats
        const float rstd2 = rstd * rstd;
        double s1 = 0.0, s2 = 0.0;
        for (int at = f; at < a.F; at += step) {
            if (at != f) fetch(at);
            const float gv[4] = {gq.x, gq.y, gq.z, gq.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float u[6];
                input(u, i);
                const float v = lut6_forward_halves(s_tab, u);
                const float tanh_x = ((v - mean) * rstd) * a.gamma + a.beta;
                float g = gv[i];                                                               // 0 from frame F on
                if (tanh_x <= 0.0f || tanh_x >= 1.0f) g = 0.0f;
                const float dxn = a.gamma * g;
                s1 -= (double)(dxn * (v - mean) * rstd2);
                s2 -= (double)(dxn * rstd);
            }
        }
        s1 = warp_sum(s1);
        s2 = warp_sum(s2);
        if (lane == 0) { s_sum[warp][0] = s1; s_sum[warp][1] = s2; }
        __syncthreads();
        if (threadIdx.x == 0) {
            double t1 = 0.0, t2 = 0.0;
            for (int w = 0; w < warps; ++w) { t1 += s_sum[w][0]; t2 += s_sum[w][1]; }
            const float dv = (float)t1 * rstd;
            const float dm = ((float)t2 - (mean * dv)) * rF;
            a.dvar[node] = dv;
            a.dmean[node] = dm;
            s_stat[0] = dm;
            s_stat[1] = dv;
            grid_clear_wait(clear, a.dW + (size_t)node * 64, &s_tab[0].x, 64);
        }
        __syncthreads();
        dmean = s_stat[0];
        dvar = s_stat[1];
        if (a.F > step) fetch(f);                                                              // more than one round: start over
    }
    if (!BN) {
        if (threadIdx.x == 0) grid_clear_wait(clear, a.dW + (size_t)node * 64, &s_tab[0].x, 64);
        __syncthreads();
    }
    size_t out[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) out[j] = (size_t)(rows[j] - a.x);                              // dx rows have the stride of x
    f32x2 acc2[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc2[i] = 0ull;
    for (int at = f; at < a.F; at += step) {
        if (at != f) fetch(at);
        const float gv[4] = {gq.x, gq.y, gq.z, gq.w};
        float dxv[4][6];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float u[6];
            input(u, i);
            KeptHalves D;
            const float v = lut6_forward_keep_halves(s_tab, u, D);
            float g = gv[i];
            if (BN) {
                const float tanh_x = ((v - mean) * rstd) * a.gamma + a.beta;
                if (tanh_x <= 0.0f || tanh_x >= 1.0f) g = 0.0f;
                const float dxc = (g * a.gamma) * rstd;
                g = dxc + dmean + (v * dvar * rF);
            }
            if (at + i >= a.F) g = 0.0f;
            lut6_reverse_halves(s_tab, u, D, g, acc2, dxv[i]);
        }
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            float *dst = a.dx + out[j] + at;
            if (a.vec) {
                red_add_v4(dst, dxv[0][j], dxv[1][j], dxv[2][j], dxv[3][j]);                   // rows are padded to whole quads; frames from F on add 0
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (at + i < a.F) atomicAdd(dst + i, dxv[i][j]);
            }
        }
    }
    float acc[64];
#pragma unroll
    for (int i = 0; i < 32; ++i) unpack2(acc2[i], acc[i], acc[i + 32]);
    warp_reduce_scatter64(acc, lane);
    s_dc[warp][2 * lane] = acc[0];
    s_dc[warp][2 * lane + 1] = acc[1];
    __syncthreads();
    if (warp == 0) {
        float2 c = make_float2(0.0f, 0.0f);
        for (int w = 0; w < warps; ++w) { c.x += s_dc[w][2 * lane]; c.y += s_dc[w][2 * lane + 1]; }
        const float2 gw = coeff_grads_to_table(c, lane);
        float *dst = a.dW + (size_t)node * 64 + 2 * lane;
        dst[0] += gw.x;
        dst[1] += gw.y;
    }
}

// Registers leave an SM 20 warps of the forward kernels and 8 of the backward ones.  In units of 0.1 us a wave of the forward costs about 20 and 6 a
// round, of the backward 23 and 18 (a sweep of 58 layers with 1, 2, 4 and 8 warps; forward / backward in us, as many warps as rounds -> this rule:
// 1024 nodes x 512 frames 7.8 / 17.8 -> 6.2 / 14.1, 4096 x 512 21.6 / 57 -> 16.8 / 43.7, 3015 x 260 14.7 / 43 -> 12.3 / 29, 982 x 1670 19.6 / 54 ->
// 14.1 / 37.8, 420 x 512 4.0 / 10.4 -> 3.9 / 9.3; on the worst layer 10 % from the best count).
unsigned forward_threads(int O, int F)  { return small_layer_threads(O, F, 20, 20, 6); }
unsigned backward_threads(int O, int F) { return small_layer_threads(O, F, 8, 23, 18); }

}   // namespace

// On the way of calls of 3 us: the device is asked for once, and not at all where one warp does (eight look-ups and 64-bit divisions took 0.35 us).
unsigned small_layer_threads(int O, int F, int sm_warps, int fixed, int per_round)
{
    const unsigned all = F > 128 * kWarpsPerCta ? kWarpsPerCta : (unsigned)(F + 127) / 128;      // warps that one round of frames keeps busy
    if (all == 1) return 32u;
    const unsigned sms = (unsigned)device_info().sm_count;
    if ((unsigned)O <= sms * ((unsigned)sm_warps / all)) return 32u * all;                       // one wave as it is
    unsigned best = all, best_cost = ~0u;
    for (unsigned w = all; w >= 1; --w) {
        const unsigned slots = sms * ((unsigned)sm_warps / w), rounds = ((unsigned)F + 128 * w - 1) / (128 * w);
        const unsigned cost = ((unsigned)O + slots - 1) / slots * ((unsigned)fixed + (unsigned)per_round * rounds);
        if (cost < best_cost) { best = w; best_cost = cost; }
    }
    return 32u * best;
}

// Measured on B200 against the persistent kernels, training forward / batch-normalised backward of a layer: 360 nodes x 100 frames 6 / 9 us
// (18 / 33), 1024 x 512 10 / 21 (20 / 46), 4096 x 512 24 / 60 (34 / 80), 2048 x 1000 27 / 72 (33 / 81; 64 from the saved output): even at
// 2^21 node-frames.  A CTA works through its node's frames alone, hence the limit on those (64 x 11000: 16 / 39 against 21 / 49).
bool small_probability_layer(int O, int F) { return O > 0 && F > 0 && (long long)O * F <= kSmallProbability && F <= BBCU_B200_SMALL_FRAMES; }

int small_forward(int mode, const SmallLayerArgs &a, int O, cudaStream_t st)
{
    const unsigned threads = forward_threads(O, a.F);
    if (mode == kSmallTrain) {
        const int round = 4 * (int)threads;
        launch(k_lut6_small_forward<kSmallTrain>, O, threads, (a.F + round - 1) / round * round * (int)sizeof(float), st, a);
    } else if (mode == kSmallInfer) {
        launch(k_lut6_small_forward<kSmallInfer>, O, threads, 0, st, a);
    } else {
        launch(k_lut6_small_forward<kSmallPlain>, O, threads, 0, st, a);
    }
    return launch_status();
}

int small_backward(bool bn, const SmallLayerArgs &a, int I, int O, cudaStream_t st)
{
    GridClear clear;
    const int rc = grid_clear_setup(clear, a.dx, (size_t)I * (size_t)a.fs, st);
    if (rc) return rc;
    if (bn) launch(k_lut6_small_backward<true>, O, backward_threads(O, a.F), 0, st, a, clear);
    else    launch(k_lut6_small_backward<false>, O, backward_threads(O, a.F), 0, st, a, clear);
    return launch_status();
}

}   // namespace bb200
