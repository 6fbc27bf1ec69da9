// Bit-input LUT layers by pattern table.
//
// With bit-packed inputs every input of a node is one of two values (0.5 - bias, 0.5 + bias), so a node's LUT value over a
// frame depends only on the frame's 6-bit input pattern p: y = Y[p], 64 values per node.  Everything a bit-in / bit-out
// layer produces then follows from Y and from how often each pattern occurs:
//
//   * bit output (y > 0.5 after the optional batch-norm affine map) is a 64-bit truth table B[p] per node, and the layer's
//     forward IS a BinaryLut6 forward with that table: 63 word-wide integer operations per 32 frames instead of a 63-node
//     fp32 tree per frame;
//   * the batch statistics of the training forward are  sum_p H[p] Y[p]  and  sum_p H[p] Y[p]^2  with H the per-node
//     histogram of the patterns over the frames (minterm masks and population counts on whole words).
//
// Y[p] is evaluated by the same tree walk, on the same conditioned inputs (+-bias), as the per-frame kernels, so the
// values -- and every threshold decision taken on them -- are bit-identical to evaluating the tree frame by frame.
//
// Reference semantics: the bit-input branches of include/bb/StochasticLutN.h:432-560 and include/bb/DifferentiableLutN.h:
// 747-905 (CPU), operators bbcu_bit_bit_fp32_StochasticLut_Forward, bbcu_bit_fp32_DifferentiableLutN_ForwardTraining /
// _ForwardInference (include/bbcu/bbcu.h:540-560, 600-618, 712-727).
#include <map>
#include <mutex>

#include "common.cuh"
#include "async_copy.cuh"
#include "bit_transpose.cuh"
#include "grid_clear.cuh"
#include "lut6_core.cuh"

namespace bb200 {

namespace {

enum { kTableRaw = 0, kTableNorm = 1, kTableNone = 2 };

constexpr long long kSmallLayer = 1LL << 21;         // node-frames, see small_layer()

// One warp per node: lane l evaluates patterns l and l + 32 as one packed pair (they differ in input 5 only).
// MODE kTableRaw : B[p] = Y[p] > 0.5                                   (StochasticLut6, bit -> bit)
//      kTableNorm: B[p] = ((Y[p] - mean) * scale) * gamma + beta > 0.5 (DifferentiableLut6 inference; scale = 1/sqrt(var))
//      kTableNone: Y only (training: the statistics come first)
template <int MODE>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
k_pattern_values(const float *__restrict__ W, float *__restrict__ Y, int *__restrict__ table, const float *__restrict__ mean_buf,
                 const float *__restrict__ var_buf, float gamma, float beta, float bias, int O, int lut_binarize)
{
    grid_dependency();
    __shared__ float4 s_tab[kWarpsPerCta][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int node = blockIdx.x * kWarpsPerCta + warp;
    if (node >= O) return;
    float4 *tab = s_tab[warp];
    stage_table_x2(tab, W, node, lane, lut_binarize);
    f32x2 up[6][1], yp[1];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        const float u = ((lane >> j) & 1) ? bias : -bias;
        up[j][0] = pack2(u, u);
    }
    up[5][0] = pack2(-bias, bias);
    lut6_forward_x2<1>(tab, up, yp);
    float lo, hi;
    unpack2(yp[0], lo, hi);
    if (Y != nullptr) {
        Y[(size_t)node * 64 + lane] = lo;
        Y[(size_t)node * 64 + 32 + lane] = hi;
    }
    if (MODE != kTableNone) {
        if (MODE == kTableNorm) {
            const float mean = mean_buf[node], scale = 1.0f / sqrtf(var_buf[node]);       // DifferentiableLutN.h:866-868
            lo = (lo - mean) * scale; lo = lo * gamma + beta;
            hi = (hi - mean) * scale; hi = hi * gamma + beta;
        }
        const unsigned w_lo = __ballot_sync(kFull, lo > 0.5f), w_hi = __ballot_sync(kFull, hi > 0.5f);
        if (lane == 0) { table[2 * (size_t)node] = (int)w_lo; table[2 * (size_t)node + 1] = (int)w_hi; }
    }
}

// Minterm masks of two sets of 6 input words, depth first.  At the leaves a full adder per bit takes both masks and what the pairs before
// left over (`ones`): its carries count two, and only they go through the population count.
template <int L>
struct Minterms {
    static __device__ __forceinline__ void count(uint32_t ma, uint32_t mb, const uint32_t (&xa)[6], const uint32_t (&xb)[6], uint32_t (&ones)[64],
                                                 uint32_t (&twos)[64], int base)
    {
        Minterms<L - 1>::count(ma & ~xa[L - 1], mb & ~xb[L - 1], xa, xb, ones, twos, base);
        Minterms<L - 1>::count(ma & xa[L - 1], mb & xb[L - 1], xa, xb, ones, twos, base + (1 << (L - 1)));
    }
};
template <>
struct Minterms<0> {
    static __device__ __forceinline__ void count(uint32_t ma, uint32_t mb, const uint32_t (&)[6], const uint32_t (&)[6], uint32_t (&ones)[64],
                                                 uint32_t (&twos)[64], int base)
    {
        const uint32_t o = ones[base];
        twos[base] += __popc((ma & mb) | (o & (ma ^ mb)));
        ones[base] = o ^ ma ^ mb;
    }
};

template <int N, int MASK>
__device__ __forceinline__ void butterfly_step_u32(uint32_t (&a)[64], int lane)
{
    const bool upper = (lane & MASK) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        const uint32_t send = upper ? a[i] : a[i + N / 2];
        const uint32_t keep = upper ? a[i + N / 2] : a[i];
        a[i] = keep + __shfl_xor_sync(kFull, send, MASK);
    }
}

// Per-node histogram of the input patterns.  Warp = one node for a tile of words; each lane takes whole words (32 frames), two at a time.
// Population counts issue at a quarter of the rate of logic, and with one per pattern and word they bound the kernel; the pairs halve them
// (8192 nodes x 16384 frames 78 -> 63 us).
constexpr int kHistWarps = 4;

__global__ void __launch_bounds__(kHistWarps * 32, 3)
k_pattern_histogram(const uint32_t *__restrict__ x, const int *__restrict__ idx, uint32_t *__restrict__ hist, int O, int F, long long xs, int groups,
                    int tile_words)
{
    grid_dependency();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x / groups;
    const int node = (blockIdx.x % groups) * kHistWarps + warp;
    if (node >= O) return;
    const uint32_t *rows[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) rows[j] = x + (size_t)__ldg(idx + (size_t)node * 6 + j) * xs;
    uint32_t cnt[64], ones[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) cnt[i] = ones[i] = 0;
    const int words = (F + 31) >> 5;
    const int w_end = min(words, (tile + 1) * tile_words);
    auto live = [&](int w) {                                            // the frames of a word that exist
        const int valid = F - w * 32;
        return w >= w_end ? 0u : valid >= 32 ? 0xffffffffu : (1u << valid) - 1u;
    };
    for (int w = tile * tile_words + lane; w < w_end; w += 64) {
        uint32_t xa[6], xb[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            xa[j] = __ldg(rows[j] + w);
            xb[j] = w + 32 < w_end ? __ldg(rows[j] + w + 32) : 0u;
        }
        Minterms<6>::count(live(w), live(w + 32), xa, xb, ones, cnt, 0);
    }
#pragma unroll
    for (int i = 0; i < 64; ++i) cnt[i] = 2 * cnt[i] + __popc(ones[i]);
    butterfly_step_u32<64, 16>(cnt, lane);
    butterfly_step_u32<32, 8>(cnt, lane);
    butterfly_step_u32<16, 4>(cnt, lane);
    butterfly_step_u32<8, 2>(cnt, lane);
    butterfly_step_u32<4, 1>(cnt, lane);
    atomicAdd(hist + (size_t)node * 64 + 2 * lane, cnt[0]);
    atomicAdd(hist + (size_t)node * 64 + 2 * lane + 1, cnt[1]);
}

// Training statistics and the truth table from Y and the histogram (include/bb/DifferentiableLutN.h:804-812 for the statistics).
__global__ void __launch_bounds__(kWarpsPerCta * 32)
k_dl6_bit_train_finalize(const float *__restrict__ Y, const uint32_t *__restrict__ hist, int *__restrict__ table, float *mean_out, float *rstd_out,
                         float *running_mean, float *running_var, float gamma, float beta, float momentum, int O, int F)
{
    grid_dependency();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int node = blockIdx.x * kWarpsPerCta + warp;
    if (node >= O) return;
    const float y0 = Y[(size_t)node * 64 + lane], y1 = Y[(size_t)node * 64 + 32 + lane];
    const double h0 = (double)hist[(size_t)node * 64 + lane], h1 = (double)hist[(size_t)node * 64 + 32 + lane];
    double s1 = h0 * (double)y0 + h1 * (double)y1;
    double s2 = h0 * ((double)y0 * (double)y0) + h1 * ((double)y1 * (double)y1);
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    const float rF   = 1.0f / (float)F;
    const float mean = (float)s1 * rF;
    const float var  = fmaxf(1.0e-5f, fmaf((float)s2, rF, -(mean * mean)));
    const float rstd = 1.0f / sqrtf(var);
    float lo = (y0 - mean) * rstd, hi = (y1 - mean) * rstd;
    lo = lo * gamma + beta;
    hi = hi * gamma + beta;
    const unsigned w_lo = __ballot_sync(kFull, lo > 0.5f), w_hi = __ballot_sync(kFull, hi > 0.5f);
    if (lane == 0) {
        table[2 * (size_t)node] = (int)w_lo;
        table[2 * (size_t)node + 1] = (int)w_hi;
        running_mean[node] = running_mean[node] * momentum + mean * (1.0f - momentum);
        running_var[node]  = running_var[node]  * momentum + var  * (1.0f - momentum);
        mean_out[node] = mean;
        rstd_out[node] = rstd;
    }
}

// BinaryLut6 leaves the bits past the last frame as its inputs make them; these layers clear them.
__global__ void k_clear_tail_bits(uint32_t *y, int O, int F, long long ys)
{
    grid_dependency();
    const int node = blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= O) return;
    y[(size_t)node * ys + (F >> 5)] &= (1u << (F & 31)) - 1u;
}

// StochasticLut6 bit -> fp32: y[f] = clip(Y[p(f)], 0, 1).  Warp = one node for a tile of words.  Each lane loads one word of each of
// the six rows (32 words per row and step, coalesced); a 32 x 32 bit transpose per row then gives lane l the bits of frame l of
// all 32 words.  The patterns of four consecutive words are assembled at once, one per byte (a four-bit field of every row is
// spread over the bytes by one multiplication), and for each of the 32 words the warp looks its 32 patterns up in the node's 64
// clipped values (shared memory) and stores 32 consecutive frames.
__global__ void __launch_bounds__(kWarpsPerCta * 32)
k_bit_gather_forward(const uint32_t *__restrict__ x, float *__restrict__ y, const int *__restrict__ idx, const float *__restrict__ Y, int O, int F,
                     long long xs, long long ys, int groups, int tile_words)
{
    grid_dependency();
    __shared__ float s_val[kWarpsPerCta][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x / groups;
    const int node = (blockIdx.x % groups) * kWarpsPerCta + warp;
    if (node >= O) return;
    float *val = s_val[warp];
    val[lane] = __saturatef(Y[(size_t)node * 64 + lane]);
    val[lane + 32] = __saturatef(Y[(size_t)node * 64 + 32 + lane]);
    __syncwarp();
    const uint32_t *rows[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) rows[j] = x + (size_t)__ldg(idx + (size_t)node * 6 + j) * xs;
    const int words = (F + 31) >> 5;
    const int w_end = min(words, (tile + 1) * tile_words);
    float *yrow = y + (size_t)node * ys;
    const BitTranspose transpose(lane);
    for (int w0 = tile * tile_words; w0 < w_end; w0 += 32) {
        uint32_t t[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) t[j] = transpose((w0 + lane < w_end) ? __ldg(rows[j] + w0 + lane) : 0u);      // bit k: frame `lane` of word w0 + k
        const int kn = min(32, w_end - w0);
        float *yw = yrow + (size_t)w0 * 32 + lane;
        const bool whole = kn == 32 && (long long)(w0 + 32) * 32 <= F;         // 32 full words: no guards
#pragma unroll
        for (int k0 = 0; k0 < 32; k0 += 4) {
            if (!whole && k0 >= kn) break;
            uint32_t p4 = 0u;                                                   // the patterns of words k0 .. k0 + 3, one per byte
#pragma unroll
            for (int j = 0; j < 6; ++j) p4 |= ((((t[j] >> k0) & 0xfu) * 0x00204081u) & 0x01010101u) << j;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float v = val[(p4 >> (8 * i)) & 63u];
                if (whole || (k0 + i < kn && (long long)(w0 + k0 + i) * 32 + lane < F)) yw[(k0 + i) * 32] = v;
            }
        }
    }
}

// --------------------------------------------------------------------------------------------- backward of bit-input layers
// With bit inputs the backward pass also factors through the pattern p of a frame:
//   dx_j(f) = g(f) * D_j[p(f)]          D_j[p] = dy/du_j at pattern p; y is linear in u_j, so D_j does not depend on bit j of p
//   dW      = K^T Hg                    Hg[p] = sum of g over the frames with pattern p; K[i][p] = prod_j k(bit_j(i), bit_j(p)),
//                                        k = 0.5 + bias where the bits agree, 0.5 - bias where they differ (one butterfly per input)
// and for the batch-norm form g(f) = mask[p] dy(f) gamma rstd + dmean + Y[p] dvar / F, so Hg and the two batch sums
// (include/bb/DifferentiableLutN.h:1190-1258) follow from Hdy[p] = sum of dy per pattern and the pattern counts H[p].
// Kernels: the sums per pattern and the pattern of every frame (k_pattern_sums); everything per node (k_bit_backward_finalize:
// batch sums, dW, the look-up tables of the last pass); dx (k_pattern_gather).
//
// dx is gathered by input row, not scattered by node: reductions into L2 run at 6 TB/s on B200 whatever their width (measured, 512
// bytes in 24 clocks per SM), so six of them per node-frame cost 0.54 ms for 8192 nodes x 16384 frames, while loads that hit L2 run
// at 18 TB/s.  An input row therefore sums over its consumers (a list made once per launch), reading their dy and pattern
// bytes, and is written once: no clear, no read-modify-write, 5 bytes per node-frame and consumer.
//
// In all of them lane l owns the frames 4l .. 4l+3 of every 128, so that dy is read and dx is written 16 bytes at a time.

struct BitBwdArgs {
    const uint32_t *x;                  // bit-packed rows, or (k_pattern_sums<true>) fp32 rows reinterpreted: an input is "set" where x > 0.5
    const float *dy;
    float *dx;
    const int *idx;
    float *hdy;                         // [O][64] sums of dy per pattern
    uint32_t *hist;                     // [O][64] pattern counts
    uint2 *mask;                        // [O] hard-tanh masks of the 64 patterns (batch norm only)
    uint8_t *pat;                       // [O][ps] patterns, bit 7: the mask passes
    float *etab;                        // [6 O][64] look-up tables, see k_bit_backward_finalize
    float2 *ntab;                       // [O] gamma rstd, dvar bias / F
    const int *edge_end, *edge_count, *edges;      // consumers of every input row (8 node + input number); count: negative for heavy rows
    const int2 *heavy;                  // chunks of the rows with more than heavy_from consumers: row, first consumer; heavy_count[0] of them
    const int *heavy_count;
    int heavy_from, heavy_chunk, heavy_ctas;
    int I, O, F, groups, tile_frames, tiles, nc, split;
    int vec;                            // dy and dx (and fp32 x) rows start on 16-byte boundaries
    long long xs, fs, ps;               // word stride of x, float stride of dy / dx, stride of pat
};

// bits of four frames (4l .. 4l+3 of the chunk, words of the 32 frames they are in) -> four patterns, one per byte
__device__ __forceinline__ uint32_t pattern_bytes(const uint32_t (&w)[6], int lane)
{
    const int sh = 4 * (lane & 7);
    uint32_t p4 = 0u;
#pragma unroll
    for (int j = 0; j < 6; ++j) p4 |= (((w[j] >> sh) & 0xfu) * (0x00204081u << j)) & (0x01010101u << j);
    return p4;
}

// four consecutive floats of a row; frames from F on read as 0
__device__ __forceinline__ float4 load_frames(const float *row, long long f, int F, int vec)
{
    if (vec && f + 3 < F) return __ldg(reinterpret_cast<const float4 *>(row + f));
    return make_float4(f < F ? __ldg(row + f) : 0.0f, f + 1 < F ? __ldg(row + f + 1) : 0.0f, f + 2 < F ? __ldg(row + f + 2) : 0.0f,
                       f + 3 < F ? __ldg(row + f + 3) : 0.0f);
}

// bits[i][w]: frames 32 w .. 32 w + 31 of row i, set where x > 0.5.  A warp packs 32 words (1024 frames); bound by reading x.
__global__ void __launch_bounds__(kWarpsPerCta * 32)
k_pack_bits(const float *__restrict__ x, uint32_t *__restrict__ bits, int I, int F, long long xs, long long ws, int runs)
{
    grid_dependency();
    const int lane = threadIdx.x & 31;
    const long long unit = (long long)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
    const int row = (int)(unit / runs), run = (int)(unit - (long long)row * runs);
    if (row >= I) return;
    const float *src = x + (size_t)row * xs + run * 1024 + lane;
    const int left = F - run * 1024 - lane;
    uint32_t mine = 0u;
#pragma unroll
    for (int h = 0; h < 32; h += 16) {
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = 32 * (h + k) < left ? __ldg(src + 32 * (h + k)) : 0.0f;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const uint32_t word = __ballot_sync(kFull, v[k] > 0.5f);
            if (lane == h + k) mine = word;
        }
    }
    if (run * 32 + lane < ws) bits[(size_t)row * ws + run * 32 + lane] = mine;
}

// Sums of dy per pattern, with BN the pattern counts, and the patterns as bytes.  Every lane keeps a histogram of its own in shared memory
// -- column `lane` of [64 patterns][32 lanes], free of bank conflicts and of atomics -- and the columns are added up once per tile.
// (Float atomics on one shared histogram per warp, compare-and-swap loops in hardware, took 0.68 ms for 8192 nodes x 16384 frames.)
// Shared memory takes four clocks per warp and 32 frames (a 64-bit load and store per frame), about as long as reading dy takes; with
// only 12 warps per SM (16 KiB of columns each) the loads have to be far ahead: 512 frames of dy are in flight per warp, and the lines of the 512 after
// them on their way to L2 (186 -> 166 us under ncu for 8192 x 8192 nodes x 16384 frames; reading dy and writing the patterns takes 105 at HBM
// speed.  One or two warps a CTA: 172 to 179).  Rows of x that do not start on 16-byte boundaries take the same loop with four loads of a word: a backward
// of 316 rows, 617 nodes and 49185 frames without batch norm 137 us, 134 with aligned rows (191 through the loop of 128 frames).
constexpr int kPsWarps = 4;
template <bool BN> struct PatternSlot { float s; uint32_t n; };      // n: count, bit 31: the pattern's mask bit
template <> struct PatternSlot<false> { float s; };

// Adds four frames (patterns one per byte, frames from `live` on do not count) to a lane's column; returns the patterns with their mask
// bits, which come with the slots.
template <bool BN>
__device__ __forceinline__ uint32_t pattern_columns_add(PatternSlot<BN> *mine, uint32_t p4, const float4 &g, int live)
{
    const float gv[4] = {g.x, g.y, g.z, g.w};
    uint32_t q4 = p4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        PatternSlot<BN> *slot = mine + 32 * __byte_perm(p4, 0u, 0x4440 + i);
        PatternSlot<BN> v = *slot;
        v.s += gv[i];
        if constexpr (BN) {
            q4 |= (v.n >> (24 - 8 * i)) & (0x80u << (8 * i));
            v.n += i < live ? 1u : 0u;
        }
        *slot = v;
    }
    return q4;
}

// adds the 32 columns of every pattern: lane l returns patterns l and l + 32
template <bool BN>
__device__ __forceinline__ void pattern_columns_reduce(const PatternSlot<BN> *slots, int lane, float (&s)[2], uint32_t (&n)[2])
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        s[h] = 0.0f;
        n[h] = 0u;
#pragma unroll 8
        for (int k = 0; k < 32; ++k) {
            const PatternSlot<BN> v = slots[(lane + 32 * h) * 32 + ((k + lane) & 31)];      // rotated: 32 different banks
            s[h] += v.s;
            if constexpr (BN) n[h] += v.n & 0x7fffffffu;
        }
    }
}

// XF32 (the statistics half of a sharded backward, always batch-normalised): the patterns come from fp32 rows.  XVEC: bit rows start on 16-byte
// boundaries (as a question to the arguments it cost those rows 2 %).
template <bool XF32, bool BN, bool XVEC>
__global__ void __launch_bounds__(kPsWarps * 32)
k_pattern_sums(const BitBwdArgs a)
{
    grid_dependency();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x / a.groups;
    const int node = (blockIdx.x % a.groups) * kPsWarps + warp;
    if (node >= a.O) return;
    PatternSlot<BN> *slots = reinterpret_cast<PatternSlot<BN> *>(smem_raw) + warp * 64 * 32, *mine = slots + lane;
    if constexpr (BN) {
        const uint2 mask = a.mask[node];
#pragma unroll 8
        for (int p = 0; p < 64; ++p) mine[p * 32] = PatternSlot<true>{0.0f, ((p < 32 ? mask.x : mask.y) << (31 - (p & 31))) & 0x80000000u};
    } else {
#pragma unroll 8
        for (int p = 0; p < 64; ++p) mine[p * 32] = PatternSlot<false>{0.0f};
    }
    const uint32_t *rows[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) rows[j] = a.x + (size_t)__ldg(a.idx + (size_t)node * 6 + j) * a.xs;
    const float *dyrow = a.dy + (size_t)node * a.fs;
    uint8_t *prow = a.pat + (size_t)node * a.ps;
    const int f_begin = tile * a.tile_frames, f_end = min(a.F, f_begin + a.tile_frames);

    int f = f_begin + 4 * lane;
    if constexpr (!XF32) {
        // 512 frames per step while whole steps are left; the loads of the next step are issued before this one is used, into the
        // other of two sets of registers.  Here a lane's frames are those of four neighbouring words of x, four of each, so that a row's words
        // come with one 128-bit load (and dy and the patterns still in whole 128 and 32 bytes), or four loads where rows of x start elsewhere.
        constexpr int NC = 4, kStep = 128 * NC;
        struct Set { uint4 w[6]; float4 dy[NC]; };
        const int steps = a.vec ? (f_end - f_begin) / kStep : 0;
        const int fl = f_begin + 128 * (lane >> 3) + 4 * (lane & 7);
        auto fetch = [&](Set &b, int k) {
            if (k < steps) {
                if (lane < 16 && k + 2 < steps) asm volatile("prefetch.global.L2 [%0];" ::"l"(dyrow + f_begin + (k + 2) * kStep + 32 * lane));
#pragma unroll
                for (int j = 0; j < 6; ++j) {
                    const uint32_t *x = rows[j] + ((fl + k * kStep) >> 5);
                    b.w[j] = XVEC ? __ldg(reinterpret_cast<const uint4 *>(x)) : make_uint4(__ldg(x), __ldg(x + 1), __ldg(x + 2), __ldg(x + 3));
                }
#pragma unroll
                for (int c = 0; c < NC; ++c) b.dy[c] = __ldg(reinterpret_cast<const float4 *>(dyrow + fl + k * kStep + 32 * c));
            }
        };
        auto use = [&](const Set &b, int k) {
            if (k < steps) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    uint32_t w[6];
#pragma unroll
                    for (int j = 0; j < 6; ++j) w[j] = c == 0 ? b.w[j].x : c == 1 ? b.w[j].y : c == 2 ? b.w[j].z : b.w[j].w;
                    *reinterpret_cast<uint32_t *>(prow + fl + k * kStep + 32 * c) = pattern_columns_add<BN>(mine, pattern_bytes(w, lane), b.dy[c], 4);
                }
            }
        };
        Set s0, s1;
        fetch(s0, 0);
        for (int k = 0; k < steps; k += 2) {
            fetch(s1, k + 1);
            use(s0, k);
            fetch(s0, k + 2);
            use(s1, k + 1);
        }
        f += steps * kStep;
    }
    for (; f < f_end; f += 128) {                          // what is left, unaligned rows, and fp32 rows
        uint32_t p4;
        if constexpr (XF32) {
            p4 = 0u;
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                const float4 v = load_frames(reinterpret_cast<const float *>(rows[j]), f, a.F, a.vec);
                p4 |= ((v.x > 0.5f ? 1u : 0u) | (v.y > 0.5f ? 0x100u : 0u) | (v.z > 0.5f ? 0x10000u : 0u) | (v.w > 0.5f ? 0x1000000u : 0u)) << j;
            }
        } else {
            uint32_t w[6];
#pragma unroll
            for (int j = 0; j < 6; ++j) w[j] = __ldg(rows[j] + (f >> 5));
            p4 = pattern_bytes(w, lane);
        }
        *reinterpret_cast<uint32_t *>(prow + f) = pattern_columns_add<BN>(mine, p4, load_frames(dyrow, f, a.F, a.vec), a.F - f);      // rows of pat are padded
    }
    __syncwarp();
    float s[2];
    uint32_t n[2];
    pattern_columns_reduce<BN>(slots, lane, s, n);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const size_t at = (size_t)node * 64 + 32 * h + lane;
        if (a.tiles == 1) {
            a.hdy[at] = s[h];
            if (BN) a.hist[at] = n[h];
        } else {                                              // several tiles: the launcher has cleared the sums
            atomicAdd(a.hdy + at, s[h]);
            if (BN) atomicAdd(a.hist + at, n[h]);
        }
    }
}

// ---- the consumers of every input row, as lists of 8 node + input number
__global__ void k_edge_count(const int *__restrict__ idx, int *count, int edges)
{
    grid_dependency();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < edges) atomicAdd(count + idx[e], 1);
}

// room for every row's list, in no particular order: `total` is a bump pointer, advanced once per warp; and the chunks of heavy rows,
// whose count is negated
__global__ void k_edge_room(int *count, int *cursor, int *total, int I, int2 *heavy, int *heavy_count, int heavy_from, int heavy_chunk)
{
    grid_dependency();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const int n = i < I ? count[i] : 0;
    int at = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(kFull, at, d);
        if (lane >= d) at += t;
    }
    int base = 0;
    if (lane == 31) base = atomicAdd(total, at);
    base = __shfl_sync(kFull, base, 31);
    if (i < I) cursor[i] = base + at - n;
    if (n > heavy_from) {
        const int chunks = (n + heavy_chunk - 1) / heavy_chunk, first = atomicAdd(heavy_count, chunks);
        for (int k = 0; k < chunks; ++k) heavy[first + k] = make_int2(i, k * heavy_chunk);
        count[i] = -n;
    }
}

// afterwards cursor[i] is the end of row i's list; dx of the heavy rows, which several CTAs add to, is cleared
__global__ void k_edge_fill(const int *__restrict__ idx, int *cursor, int *list, int edges, const int2 *__restrict__ heavy,
                            const int *__restrict__ heavy_count, float *dx, long long fs)
{
    grid_dependency();
    const int e = blockIdx.x * blockDim.x + threadIdx.x, chunks = heavy_count[0];
    if (e < edges) list[atomicAdd(cursor + idx[e], 1)] = e + 2 * (e / 6);
    for (int k = 0; k < chunks; ++k) {
        const int2 h = heavy[k];
        if (h.y == 0)
            for (long long f = e; f < fs; f += (long long)gridDim.x * blockDim.x) dx[(size_t)h.x * fs + f] = 0.0f;
    }
}

template <unsigned SEL>
__device__ __forceinline__ uint32_t prmt(uint32_t v)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(v), "n"(SEL));
    return r;
}

// dx_i(f) = sum over the consumers (node o, input j) of row i of g_o(f) D_j[p_o(f)], frames from F on 0.  A CTA is one row and NC
// chunks of 128 frames; `split` warps share the consumers (rows with many of them, or few rows).  One warp per CTA otherwise, because
// the number of consumers varies from row to row and a CTA of several rows waits for the longest.  Rows with far more consumers than the
// average (more than heavy_from) would hold up the whole pass as one CTA's loop: the first heavy_ctas CTAs take them, in chunks of
// consumers, and add the chunks' sums to the row, which k_edge_fill has cleared.
// The tables of a consumer live in registers, one entry per lane, and a look-up is a shuffle whose source lane is the pattern rotated by
// j + 1 (the rotation serves the patterns of four frames at once): bits 0 .. 4 are the other five inputs, bit 5 is input j.  No single
// resource is exhausted (8192 x 8192 nodes x 8192 frames under ncu: issue 69 %, L1 68 %, logic pipe 59 %, a third of the stalls on L2
// loads, 27 warps per SM): two shuffles, 5 bytes and 16 instructions per consumer and frame.  With batch norm g is put together here;
// writing g out once and reading it back would spare a shuffle and six instructions, but costs 10 bytes per node-frame of HBM traffic.
// Several rows one after the other in a CTA keep more tiles in flight than L2 holds (8 rows: 509 -> 617 us for 16384 frames).
// SHORT: a row's last tile, of which the last chunks have no frames and are left out.
template <bool BN, int NC, bool WHOLE, bool SHORT>
__device__ __forceinline__ void pattern_gather(const BitBwdArgs &a, const int *list, int n, int part, int f0, int lane, float (&acc)[NC][4])
{
    int e_n = part < n ? __ldg(list + part) : 0;
    for (int k = part; k < n; k += a.split) {
        const int node = e_n >> 3, j = e_n & 7;
        if (k + a.split < n) e_n = __ldg(list + k + a.split);
        const float *t = a.etab + (size_t)(6 * node + j) * 64 + lane;
        const float D = __ldg(t);
        const float base = BN ? __ldg(t + 32) : 0.0f;
        const float2 gs = BN ? __ldg(a.ntab + node) : make_float2(1.0f, 0.0f);
        const uint32_t minus_slope = __float_as_uint(-gs.y);
        const float *dyrow = a.dy + (size_t)node * a.fs;
        const uint8_t *prow = a.pat + (size_t)node * a.ps;
        const uint32_t low = ((1u << (5 - j)) - 1u) * 0x01010101u;        // bits that the rotation takes from the left of their byte
        float4 dyq[NC];
        uint32_t q4[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int f = f0 + 128 * c;
            if (WHOLE) {
                dyq[c] = __ldg(reinterpret_cast<const float4 *>(dyrow + f));
                q4[c] = __ldg(reinterpret_cast<const uint32_t *>(prow + f));
            } else {
                dyq[c] = load_frames(dyrow, f, a.F, a.vec);
                q4[c] = f < a.F ? __ldg(reinterpret_cast<const uint32_t *>(prow + f)) : 0u;
            }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if (SHORT && f0 - 4 * lane + 128 * c >= a.F) break;
            const float dyv[4] = {dyq[c].x, dyq[c].y, dyq[c].z, dyq[c].w};
            const uint32_t rot = ((q4[c] >> (j + 1)) & low) | ((q4[c] << (5 - j)) & ~low);        // (bits 6 and 7 of the bytes: anything)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t r = rot >> (8 * i);
                const float d = __shfl_sync(kFull, D, r);
                float g = dyv[i];
                if (BN) {
                    const float slope = __uint_as_float(((rot << (26 - 8 * i)) & 0x80000000u) ^ minus_slope);      // +slope where input j is set
                    const uint32_t pass = i == 0 ? prmt<0x8888>(q4[c]) : i == 1 ? prmt<0x9999>(q4[c])               // bit 7 of the frame's byte, replicated
                                        : i == 2 ? prmt<0xaaaa>(q4[c]) : prmt<0xbbbb>(q4[c]);
                    g = fmaf(__uint_as_float(__float_as_uint(g) & pass), gs.x, fmaf(slope, d, __shfl_sync(kFull, base, r)));
                }
                acc[c][i] = fmaf(g, d, acc[c][i]);
            }
        }
    }
}

// The sum over `n` consumers for one tile of a row, written (ADD: added) to dx by the CTA's first warp; nothing where n is negative (a heavy
// row.  Asking that first, instead of before the store, costs every CTA a wait for n: 811 -> 816 us for 8192 x 8192 nodes x 16384 frames.)
template <bool BN, int NC, bool ADD>
__device__ __forceinline__ void gather_tile(const BitBwdArgs &a, int row, const int *list, int n, int tile, float4 *s_part)
{
    const int part = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int f_begin = tile * (128 * NC), f0 = f_begin + 4 * lane;
    float acc[NC][4];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[c][i] = 0.0f;
    // A last tile most of whose chunks have frames has a form of its own without batch norm, where asking for each costs more than it saves (500 rows, 20000
    // nodes, 1000 frames 212.5 -> 210.3 us for the operator; 92 frames in the last tile, 3000 rows and nodes: 91.9 without asking, 90.4 with).  With batch norm
    // that form costs the others 1 % (8192 rows and nodes, 16384 frames 793 -> 801): SHORT = BN, so that none is built there.
    if (a.vec && f_begin + 128 * NC <= a.F)       pattern_gather<BN, NC, true, false>(a, list, n, part, f0, lane, acc);
    else if (!BN && f_begin + 64 * NC < a.F)      pattern_gather<BN, NC, false, BN>(a, list, n, part, f0, lane, acc);
    else if (f_begin < a.F)                       pattern_gather<BN, NC, false, true>(a, list, n, part, f0, lane, acc);
    if (a.split > 1) {
        if (ADD) __syncthreads();                                       // (the tile before has been read)
#pragma unroll
        for (int c = 0; c < NC; ++c) s_part[(part * NC + c) * 32 + lane] = make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
        __syncthreads();
        if (part != 0) return;
        for (int k = 1; k < a.split; ++k)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float4 v = s_part[(k * NC + c) * 32 + lane];
                acc[c][0] += v.x; acc[c][1] += v.y; acc[c][2] += v.z; acc[c][3] += v.w;
            }
    }
    if (!ADD && n < 0) return;
    float *out = a.dx + (size_t)row * a.fs;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int f = f0 + 128 * c;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (f + i >= a.F) acc[c][i] = 0.0f;
        if (a.vec && f + 3 < a.fs) {
            if (ADD) red_add_v4(out + f, acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
            else     *reinterpret_cast<float4 *>(out + f) = make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (f + i < a.fs) {
                    if (ADD) atomicAdd(out + f + i, acc[c][i]);
                    else     out[f + i] = acc[c][i];
                }
        }
    }
}

// The chunks of the heavy rows, one (tile, chunk) after another; tiles of 256 frames at most, for which the registers of the ordinary path do.
template <bool BN, int NC>
__device__ __forceinline__ void gather_heavy(const BitBwdArgs &a, float4 *s_part)
{
    constexpr int HC = NC > 2 ? 2 : NC;
    const int chunks = __ldg(a.heavy_count), items = chunks * ((a.F + 128 * HC - 1) / (128 * HC));
    for (int item = blockIdx.x; item < items; item += a.heavy_ctas) {
        const int tile = item / chunks;
        const int2 h = __ldg(a.heavy + (item - tile * chunks));
        const int n = -__ldg(a.edge_count + h.x);
        gather_tile<BN, HC, true>(a, h.x, a.edges + (__ldg(a.edge_end + h.x) - n + h.y), min(n - h.y, a.heavy_chunk), tile, s_part);
    }
}

template <bool BN, int NC>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4)
k_pattern_gather(const BitBwdArgs a)
{
    grid_dependency();
    extern __shared__ __align__(16) unsigned char smem_raw[];           // split > 1: float4 [split][NC][32]
    float4 *s_part = reinterpret_cast<float4 *>(smem_raw);
    const int block = (int)blockIdx.x - a.heavy_ctas;
    if (block < 0) {
        gather_heavy<BN, NC>(a, s_part);
        return;
    }
    const int tile = block / a.I, row = block - tile * a.I;
    const int n = __ldg(a.edge_count + row);
    gather_tile<BN, NC, false>(a, row, a.edges + (__ldg(a.edge_end + row) - n), n, tile, s_part);
}

// Per-pattern gradient sums -> table-entry gradients: for every input, (a, b) -> (a hi + b lo, a lo + b hi) with hi = 0.5 + bias,
// lo = 0.5 - bias.  Lane l holds patterns 2l and 2l + 1 on entry and table entries 2l and 2l + 1 on return.
__device__ __forceinline__ float2 pattern_sums_to_table_grads(float2 v, int lane, float bias)
{
    const float hi = 0.5f + bias, lo = 0.5f - bias;
    v = make_float2(v.x * hi + v.y * lo, v.x * lo + v.y * hi);
#pragma unroll
    for (int b = 0; b < 5; ++b) {
        const float tx = __shfl_xor_sync(kFull, v.x, 1 << b), ty = __shfl_xor_sync(kFull, v.y, 1 << b);
        v.x = v.x * hi + tx * lo;
        v.y = v.y * hi + ty * lo;
    }
    return v;
}

// LUT value and the six input derivatives at patterns `lane` and `lane + 32` of a node whose table is staged in `tab2`.
__device__ __forceinline__ void eval_pattern_pair(const float4 *tab2, int lane, float bias, float (&y)[2], float (&d)[2][6])
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float u[6];
#pragma unroll
        for (int j = 0; j < 5; ++j) u[j] = ((lane >> j) & 1) ? bias : -bias;
        u[5] = h ? bias : -bias;
        KeptHalves K;
        f32x2 unused[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) unused[i] = 0ull;
        y[h] = lut6_forward_keep_halves(tab2, u, K);
        lut6_reverse_halves(tab2, u, K, 1.0f, unused, d[h]);
    }
}

// The look-up tables of a node's six edges, 64 floats each: D_j for the 32 values of the other five bits -- entry m belongs to the
// patterns whose bits j+1 .. j+5 (mod 6) are m, the low bits of the pattern rotated by j + 1 -- and, with batch norm, the part of
// dmean + Y[p] dvar / F that does not depend on bit j (the rest is +-D_j times dvar bias / F).
template <bool BN>
__device__ __forceinline__ void store_edge_tables(float *etab, int lane, const float (&y)[2], const float (&d)[2][6], float dmean, float dvar_rF)
{
#pragma unroll
    for (int j = 0; j < 6; ++j) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const unsigned p = lane + 32 * h, q = p | (p << 6);
            const float other = j == 5 ? y[1 - h] : __shfl_xor_sync(kFull, y[h], 1 << (j & 31));
            if (!((p >> j) & 1u)) {                                                          // D_j is the same with bit j set
                float *t = etab + 64 * j + ((q >> (j + 1)) & 31u);
                t[0] = d[h][j];
                if (BN) t[32] = dmean + (0.5f * (y[h] + other)) * dvar_rF;
            }
        }
    }
}

__global__ void __launch_bounds__(kWarpsPerCta * 32)
k_pattern_derivatives(const float *__restrict__ W, float *__restrict__ etab, float bias, int O, int lut_binarize)
{
    grid_dependency();
    __shared__ float4 s_tab[kWarpsPerCta][16];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int node = blockIdx.x * kWarpsPerCta + warp;
    if (node >= O) return;
    stage_table_halves(s_tab[warp], W, node, lane, lut_binarize);
    float y[2], d[2][6];
    eval_pattern_pair(s_tab[warp], lane, bias, y, d);
    store_edge_tables<false>(etab + (size_t)node * 6 * 64, lane, y, d, 0.0f, 0.0f);
}

// Hard-tanh mask of every pattern of every node: the gradient passes where 0 < affine(Y[p]) < 1 (include/bb/DifferentiableLutN.h:1204-1206).
__global__ void __launch_bounds__(kWarpsPerCta * 32)
k_pattern_masks(const float *__restrict__ W, uint2 *__restrict__ mask, const float *__restrict__ mean_buf, const float *__restrict__ rstd_buf, float gamma,
                float beta, float bias, int O, int lut_binarize)
{
    grid_dependency();
    __shared__ float4 s_tab[kWarpsPerCta][16];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int node = blockIdx.x * kWarpsPerCta + warp;
    if (node >= O) return;
    stage_table_halves(s_tab[warp], W, node, lane, lut_binarize);
    const float mean = mean_buf[node], rstd = rstd_buf[node];
    unsigned m[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float u[6];
#pragma unroll
        for (int j = 0; j < 5; ++j) u[j] = ((lane >> j) & 1) ? bias : -bias;
        u[5] = h ? bias : -bias;
        const float t = ((lut6_forward_halves(s_tab[warp], u) - mean) * rstd) * gamma + beta;
        m[h] = __ballot_sync(kFull, !(t <= 0.0f || t >= 1.0f));
    }
    if (lane == 0) mask[node] = make_uint2(m[0], m[1]);
}

// One warp per node.  BN = false: dW += K^T Hdy.  BN = true: the batch sums, dmean / dvar, dW += K^T Hg with
// Hg[p] = mask[p] gamma rstd Hdy[p] + (dmean + Y[p] dvar / F) H[p], and the look-up tables of k_pattern_gather.
// `sums_out` (frame-sharded callers): the node's local (dstd, dmeanx) go out as fp64 and nothing else is done.
// `sums_in`: the sums over ALL ranks' frames come in instead of being formed from this rank's Hdy; rF = 1 / total frames.
template <bool BN>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
k_bit_backward_finalize(const float *__restrict__ hdy, const uint32_t *__restrict__ hist, const uint2 *__restrict__ mask, const float *__restrict__ W,
                        float *__restrict__ etab, float2 *__restrict__ ntab, float *dW, const float *__restrict__ mean_buf,
                        const float *__restrict__ rstd_buf, float *dmean_out, float *dvar_out, float gamma, float beta, float bias, int O, float rF,
                        int lut_binarize, double *sums_out, const double *__restrict__ sums_in)
{
    grid_dependency();
    __shared__ float4 s_tab[BN ? kWarpsPerCta : 1][16];
    __shared__ float s_hg[kWarpsPerCta][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int node = blockIdx.x * kWarpsPerCta + warp;
    if (node >= O) return;
    float hg[2] = {hdy[(size_t)node * 64 + lane], hdy[(size_t)node * 64 + 32 + lane]};                // patterns lane, lane + 32
    if (BN) {
        stage_table_halves(s_tab[warp], W, node, lane, lut_binarize);
        float y[2], d[2][6];
        eval_pattern_pair(s_tab[warp], lane, bias, y, d);
        const float mean = mean_buf[node], rstd = rstd_buf[node], rstd2 = rstd * rstd;
        const uint2 mw = mask[node];
        const bool m0 = (mw.x >> lane) & 1u, m1 = (mw.y >> lane) & 1u;
        const float dxn0 = m0 ? gamma * hg[0] : 0.0f, dxn1 = m1 ? gamma * hg[1] : 0.0f;       // sum over the pattern's frames of gamma * masked dy
        double dstd, dmeanx;
        if (sums_in != nullptr) {
            dstd = sums_in[2 * (size_t)node];
            dmeanx = sums_in[2 * (size_t)node + 1];
        } else {
            dstd = -((double)(dxn0 * (y[0] - mean) * rstd2) + (double)(dxn1 * (y[1] - mean) * rstd2));
            dmeanx = -((double)(dxn0 * rstd) + (double)(dxn1 * rstd));
            dstd = warp_sum(dstd);
            dmeanx = warp_sum(dmeanx);
        }
        if (sums_out != nullptr) {
            if (lane == 0) { sums_out[2 * (size_t)node] = dstd; sums_out[2 * (size_t)node + 1] = dmeanx; }
            return;
        }
        const float dvar = (float)dstd * rstd;
        const float dmean = ((float)dmeanx - (mean * dvar)) * rF;
        if (lane == 0) { dvar_out[node] = dvar; dmean_out[node] = dmean; }
        hg[0] = (dxn0 * rstd) + (dmean + (y[0] * dvar * rF)) * (float)hist[(size_t)node * 64 + lane];
        hg[1] = (dxn1 * rstd) + (dmean + (y[1] * dvar * rF)) * (float)hist[(size_t)node * 64 + 32 + lane];
        store_edge_tables<true>(etab + (size_t)node * 6 * 64, lane, y, d, dmean, dvar * rF);
        if (lane == 0) ntab[node] = make_float2(gamma * rstd, bias * dvar * rF);
    }
    s_hg[warp][lane] = hg[0];
    s_hg[warp][lane + 32] = hg[1];
    __syncwarp();
    const float2 gw = pattern_sums_to_table_grads(reinterpret_cast<const float2 *>(s_hg[warp])[lane], lane, bias);
    float *dst = dW + (size_t)node * 64 + 2 * lane;
    dst[0] += gw.x;
    dst[1] += gw.y;
}

// --------------------------------------------------------------------------------------------- binary mode on fp32 frames, forward
// Inputs are conditioned to 0.5 +- bias by x > 0.5 (include/bb/DifferentiableLutN.h:779-786), so the same per-pattern values apply;
// the pattern of a frame comes from six compares.  A lane owns four consecutive frames of every 128 (one 128-bit load per input row).
//   PASS_COUNT : pattern counts per node (shared-memory integer atomics, added to `hist` per tile) and the four patterns of the lane
//                as one 32-bit word into `pat` ([node][frame] bytes) for the output pass of the training forward;
//   PASS_OUTPUT: y[f] = val[p(f)], the patterns read back from `pat`;
//   PASS_DIRECT: both in one go, y[f] = val[p(f)] straight from x (StochasticLut6 forward, inference);
//   PASS_STATS : the first half of a frame-sharded training forward: pattern counts, and y[f] = Y[p(f)] unclipped (the raw LUT value the
//                normalise half works on).
// val[p]: clip(Y[p]) (StochasticLut6), or the truth-table bit as 0 / 1 (DifferentiableLut6 in binary mode).
enum { kPassCount = 0, kPassOutput = 1, kPassDirect = 2, kPassStats = 3 };

struct F32BinArgs {
    const float *x;
    float *y;
    const int *idx;
    const float *Y;          // [O][64] per-pattern values (kPassDirect without a table)
    const int *table;        // [O][2] truth tables, or nullptr: val = clip(Y)
    uint32_t *hist;          // [O][64]
    unsigned char *pat;      // [O][fs] pattern bytes
    int O, F, groups, tile_frames;
    long long fs;            // frame stride of x, y and pat (elements); a multiple of 4
};

template <int PASS>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
k_f32_binary_forward(const F32BinArgs a)
{
    grid_dependency();
    __shared__ float    s_val[kWarpsPerCta][64];
    __shared__ unsigned s_cnt[kWarpsPerCta][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x / a.groups;
    const int node = (blockIdx.x % a.groups) * kWarpsPerCta + warp;
    if (node >= a.O) return;
    constexpr bool kCounts = PASS == kPassCount || PASS == kPassStats;
    if (kCounts) {
        s_cnt[warp][lane] = 0u;
        s_cnt[warp][lane + 32] = 0u;
    }
    if (PASS == kPassStats) {
        s_val[warp][lane] = a.Y[(size_t)node * 64 + lane];
        s_val[warp][lane + 32] = a.Y[(size_t)node * 64 + 32 + lane];
    } else if (PASS == kPassCount) {
    } else if (a.table != nullptr) {
        const uint32_t lo = (uint32_t)a.table[2 * (size_t)node], hi = (uint32_t)a.table[2 * (size_t)node + 1];
        s_val[warp][lane] = ((lo >> lane) & 1u) ? 1.0f : 0.0f;
        s_val[warp][lane + 32] = ((hi >> lane) & 1u) ? 1.0f : 0.0f;
    } else {
        s_val[warp][lane] = __saturatef(a.Y[(size_t)node * 64 + lane]);
        s_val[warp][lane + 32] = __saturatef(a.Y[(size_t)node * 64 + 32 + lane]);
    }
    __syncwarp();
    long long off[6];
    if (PASS != kPassOutput) {
#pragma unroll
        for (int j = 0; j < 6; ++j) off[j] = (long long)__ldg(a.idx + (size_t)node * 6 + j) * a.fs;
    }
    const int f_begin = tile * a.tile_frames, f_end = min(a.F, f_begin + a.tile_frames);
    unsigned char *prow = a.pat ? a.pat + (size_t)node * a.fs : nullptr;
    float *yrow = a.y ? a.y + (size_t)node * a.fs : nullptr;
    // the loads of step i + 1 are issued before step i is processed (the loop body is short and would otherwise wait on every load)
    float4 xq[PASS == kPassOutput ? 1 : 6];
    uint32_t pq = 0;
    auto fetch = [&](int f) {
        if (PASS == kPassOutput) {
            pq = *reinterpret_cast<const uint32_t *>(prow + f);
        } else {
#pragma unroll
            for (int j = 0; j < 6; ++j) xq[j] = __ldg(reinterpret_cast<const float4 *>(a.x + off[j] + f));
        }
    };
    int f = f_begin + 4 * lane;
    if (f < f_end) fetch(f);
    for (; f < f_end; f += 128) {
        uint32_t p4 = pq;                                          // the patterns of frames f .. f+3, one per byte
        if (PASS != kPassOutput) {
            p4 = 0;
#pragma unroll
            for (int j = 0; j < 6; ++j)
                p4 |= ((xq[j].x > 0.5f ? 1u : 0u) | (xq[j].y > 0.5f ? 0x100u : 0u) | (xq[j].z > 0.5f ? 0x10000u : 0u) | (xq[j].w > 0.5f ? 0x1000000u : 0u)) << j;
        }
        if (f + 128 < f_end) fetch(f + 128);
        if (kCounts) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (f + i < a.F) atomicAdd(&s_cnt[warp][(p4 >> (8 * i)) & 63u], 1u);
            if (PASS == kPassCount) *reinterpret_cast<uint32_t *>(prow + f) = p4;
        }
        if (PASS != kPassCount) {
            const float4 o = make_float4(s_val[warp][p4 & 63u], s_val[warp][(p4 >> 8) & 63u], s_val[warp][(p4 >> 16) & 63u], s_val[warp][(p4 >> 24) & 63u]);
            if (f + 3 < a.F) {
                *reinterpret_cast<float4 *>(yrow + f) = o;
            } else {
                const float ov[4] = {o.x, o.y, o.z, o.w};
                for (int i = 0; i < 4 && f + i < a.F; ++i) yrow[f + i] = ov[i];
            }
        }
    }
    if (kCounts) {
        __syncwarp();
        atomicAdd(a.hist + (size_t)node * 64 + lane, s_cnt[warp][lane]);
        atomicAdd(a.hist + (size_t)node * 64 + 32 + lane, s_cnt[warp][lane + 32]);
    }
}

// Per-node (sum y, sum y^2) over this rank's frames from the pattern counts: sums[node] = (sum_p H[p] Y[p], sum_p H[p] Y[p]^2).
__global__ void __launch_bounds__(kWarpsPerCta * 32)
k_counts_to_sums(const float *__restrict__ Y, const uint32_t *__restrict__ hist, double *__restrict__ sums, int O)
{
    grid_dependency();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int node = blockIdx.x * kWarpsPerCta + warp;
    if (node >= O) return;
    const double y0 = (double)Y[(size_t)node * 64 + lane], y1 = (double)Y[(size_t)node * 64 + 32 + lane];
    const double h0 = (double)hist[(size_t)node * 64 + lane], h1 = (double)hist[(size_t)node * 64 + 32 + lane];
    const double s1 = warp_sum(h0 * y0 + h1 * y1), s2 = warp_sum(h0 * (y0 * y0) + h1 * (y1 * y1));
    if (lane == 0) { sums[2 * (size_t)node] = s1; sums[2 * (size_t)node + 1] = s2; }
}

// --------------------------------------------------------------------------------------------- small layers: one launch per direction
// Where a layer has up to a million or two node-frames, the kernels above take a few microseconds each and the launches between them take as
// long again.  Here one CTA is one node with all of its frames (1 to 8 warps): tables, counts, statistics and output without
// leaving the SM.  The rows are read twice (the second time from L1 or L2), counts and sums go through shared-memory atomics, and the
// backward scatters dx, which it clears first (grid_clear.cuh), with reductions in L2 (36 clocks per SM, warp and 32 frames) -- which is
// why larger layers do not come here: see small_layer().

struct SmallBinArgs {
    const void *x;                      // fp32 rows, or bit rows
    void *y;                            // forward: fp32 rows (0 / 1), or bit rows
    const float *dy;
    float *dx;
    const int *idx;
    const float *W;
    float *dW;
    const float *mean_in, *rstd_in;     // backward
    float *mean, *rstd, *running_mean, *running_var, *dmean, *dvar;
    float gamma, beta, momentum, bias;
    int F, lut_binarize, vec;           // vec: fp32 rows start on 16-byte boundaries
    long long xs, ys, fs;               // strides of x, y and dy / dx
};

// the patterns of frames f .. f+3 (one per byte) of a node with input rows `rows`
template <bool XBIT>
__device__ __forceinline__ uint32_t small_patterns(const SmallBinArgs &a, const size_t (&rows)[6], int f, int lane)
{
    if (XBIT) {
        uint32_t w[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) w[j] = f < a.F ? __ldg(static_cast<const uint32_t *>(a.x) + rows[j] + (f >> 5)) : 0u;
        return pattern_bytes(w, lane);
    }
    uint32_t p4 = 0u;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const float4 v = load_frames(static_cast<const float *>(a.x) + rows[j], f, a.F, a.vec);
        p4 |= ((v.x > 0.5f ? 1u : 0u) | (v.y > 0.5f ? 0x100u : 0u) | (v.z > 0.5f ? 0x10000u : 0u) | (v.w > 0.5f ? 0x1000000u : 0u)) << j;
    }
    return p4;
}

// Training forward of a batch-normalised layer on two-valued inputs: the arithmetic of k_pattern_values and k_dl6_bit_train_finalize.
// WARPS: how many an SM has to hold.  64 leave 32 registers, with which the rows are waited for sooner than need be.
template <bool XBIT, int WARPS>
__global__ void __launch_bounds__(kWarpsPerCta * 32, WARPS / kWarpsPerCta)
k_small_binary_forward(const SmallBinArgs a)
{
    grid_dependency();
    __shared__ float4 s_tab[32];
    __shared__ unsigned s_cnt[64];
    __shared__ unsigned s_table[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, node = blockIdx.x;
    const float2 *table = reinterpret_cast<const float2 *>(a.W + (size_t)node * 64) + lane;
    float2 w = make_float2(0.0f, 0.0f);
    if (!XBIT && warp == 0) w = *table;                                                     // (bit rows are here sooner: 2 % slower that way)
    size_t rows[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) rows[j] = (size_t)__ldg(a.idx + (size_t)node * 6 + j) * a.xs;
    const int f_first = 4 * (int)threadIdx.x;
    const uint32_t p_first = small_patterns<XBIT>(a, rows, f_first, lane);       // under way while the table is evaluated, and kept for the output
    float y0 = 0.0f, y1 = 0.0f;
    if (warp == 0) {
        s_cnt[lane] = 0u;
        s_cnt[lane + 32] = 0u;
        stage_table_x2(s_tab, XBIT ? *table : w, lane, a.lut_binarize);
        f32x2 up[6][1], yp[1];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            const float u = ((lane >> j) & 1) ? a.bias : -a.bias;
            up[j][0] = pack2(u, u);
        }
        up[5][0] = pack2(-a.bias, a.bias);
        lut6_forward_x2<1>(s_tab, up, yp);
        unpack2(yp[0], y0, y1);                                              // patterns lane, lane + 32
    }
    __syncthreads();
    const int step = 4 * (int)blockDim.x;
    for (int f = f_first; f < a.F; f += step) {
        const uint32_t p4 = f == f_first ? p_first : small_patterns<XBIT>(a, rows, f, lane);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (f + i < a.F) atomicAdd(&s_cnt[(p4 >> (8 * i)) & 63u], 1u);
    }
    __syncthreads();
    if (warp == 0) {
        const double h0 = (double)s_cnt[lane], h1 = (double)s_cnt[lane + 32];
        const double s1 = warp_sum(h0 * (double)y0 + h1 * (double)y1);
        const double s2 = warp_sum(h0 * ((double)y0 * (double)y0) + h1 * ((double)y1 * (double)y1));
        const float rF   = 1.0f / (float)a.F;
        const float mean = (float)s1 * rF;
        const float var  = fmaxf(1.0e-5f, fmaf((float)s2, rF, -(mean * mean)));
        const float rstd = 1.0f / sqrtf(var);
        float lo = (y0 - mean) * rstd, hi = (y1 - mean) * rstd;
        lo = lo * a.gamma + a.beta;
        hi = hi * a.gamma + a.beta;
        const unsigned w_lo = __ballot_sync(kFull, lo > 0.5f), w_hi = __ballot_sync(kFull, hi > 0.5f);
        if (lane == 0) {
            s_table[0] = w_lo;
            s_table[1] = w_hi;
            a.running_mean[node] = a.running_mean[node] * a.momentum + mean * (1.0f - a.momentum);
            a.running_var[node]  = a.running_var[node]  * a.momentum + var  * (1.0f - a.momentum);
            a.mean[node] = mean;
            a.rstd[node] = rstd;
        }
    }
    __syncthreads();
    const uint32_t lo = s_table[0], hi = s_table[1];
    for (int base = 4 * 32 * warp; base < a.F; base += step) {               // warp-uniform: bit outputs shuffle
        const int f = base + 4 * lane;
        const uint32_t p4 = f == f_first ? p_first : small_patterns<XBIT>(a, rows, f, lane);
        uint32_t bits = 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t p = p4 >> (8 * i);
            bits |= f + i < a.F ? (((p & 32u ? hi : lo) >> (p & 31u)) & 1u) << i : 0u;
        }
        if (XBIT) {
            bits <<= 4 * (lane & 7);
#pragma unroll
            for (int m = 1; m < 8; m <<= 1) bits |= __shfl_xor_sync(kFull, bits, m);
            if ((lane & 7) == 0 && f < a.F) static_cast<uint32_t *>(a.y)[(size_t)node * a.ys + (f >> 5)] = bits;
        } else {
            float *out = static_cast<float *>(a.y) + (size_t)node * a.ys + f;
            const float4 o = make_float4(bits & 1u ? 1.0f : 0.0f, bits & 2u ? 1.0f : 0.0f, bits & 4u ? 1.0f : 0.0f, bits & 8u ? 1.0f : 0.0f);
            if (a.vec && f + 3 < a.F) {
                *reinterpret_cast<float4 *>(out) = o;
            } else {
                if (f < a.F) out[0] = o.x;
                if (f + 1 < a.F) out[1] = o.y;
                if (f + 2 < a.F) out[2] = o.z;
                if (f + 3 < a.F) out[3] = o.w;
            }
        }
    }
}

// Backward (BN: batch-normalised layer): the arithmetic of k_bit_backward_finalize and k_pattern_gather.  WARPS as above: 24 leave 80 registers.
template <bool XBIT, bool BN, int WARPS>
__global__ void __launch_bounds__(kWarpsPerCta * 32, WARPS / kWarpsPerCta)
k_small_binary_backward(const SmallBinArgs a, const GridClear clear)
{
    grid_dependency();
    __shared__ float4 s_tab[16];
    __shared__ float s_hdy[64], s_hg[64];
    __shared__ unsigned s_cnt[64];
    __shared__ float s_edge[6 * 64];
    __shared__ float s_node[2];
    __shared__ unsigned s_mask[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, node = blockIdx.x;
    float2 w = make_float2(0.0f, 0.0f);
    if (warp == 0) w = reinterpret_cast<const float2 *>(a.W + (size_t)node * 64)[lane];          // on its way before the rows are waited for
    size_t rows[6], out[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const size_t r = (size_t)__ldg(a.idx + (size_t)node * 6 + j);
        rows[j] = r * a.xs;
        out[j] = XBIT ? r * a.fs : rows[j];                                     // fp32 x shares the stride of dx
    }
    const float *dyrow = a.dy + (size_t)node * a.fs;
    // under way while the patterns are evaluated, and kept for the second pass
    const int f_first = 4 * (int)threadIdx.x;
    const uint32_t p_first = small_patterns<XBIT>(a, rows, f_first, lane);
    const float4 g_first = load_frames(dyrow, f_first, a.F, a.vec);
    float y[2], d[2][6], mean = 0.0f, rstd = 0.0f;
    bool m[2] = {false, false};
    if (warp == 0) {
        s_hdy[lane] = 0.0f;
        s_hdy[lane + 32] = 0.0f;
        s_cnt[lane] = 0u;
        s_cnt[lane + 32] = 0u;
        stage_table_halves(s_tab, w, lane, a.lut_binarize);
        eval_pattern_pair(s_tab, lane, a.bias, y, d);
        if (BN) {
            mean = a.mean_in[node];
            rstd = a.rstd_in[node];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float t = ((y[h] - mean) * rstd) * a.gamma + a.beta;
                m[h] = !(t <= 0.0f || t >= 1.0f);
                const unsigned w = __ballot_sync(kFull, m[h]);
                if (lane == 0) s_mask[h] = w;
            }
        } else {
            store_edge_tables<false>(s_edge, lane, y, d, 0.0f, 0.0f);
        }
    }
    grid_clear_slices(clear);
    __syncthreads();
    const int step = 4 * (int)blockDim.x;
    for (int f = f_first; f < a.F; f += step) {
        const uint32_t p4 = f == f_first ? p_first : small_patterns<XBIT>(a, rows, f, lane);
        const float4 g = f == f_first ? g_first : load_frames(dyrow, f, a.F, a.vec);
        const float gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (f + i < a.F) {
                const uint32_t p = (p4 >> (8 * i)) & 63u;
                atomicAdd(&s_hdy[p], gv[i]);
                if (BN) atomicAdd(&s_cnt[p], 1u);
            }
    }
    __syncthreads();
    if (warp == 0) {
        float hg[2] = {s_hdy[lane], s_hdy[lane + 32]};
        if (BN) {
            const float rF = 1.0f / (float)a.F, rstd2 = rstd * rstd;
            const float dxn0 = m[0] ? a.gamma * hg[0] : 0.0f, dxn1 = m[1] ? a.gamma * hg[1] : 0.0f;
            const double dstd = warp_sum(-((double)(dxn0 * (y[0] - mean) * rstd2) + (double)(dxn1 * (y[1] - mean) * rstd2)));
            const double dmeanx = warp_sum(-((double)(dxn0 * rstd) + (double)(dxn1 * rstd)));
            const float dvar = (float)dstd * rstd;
            const float dmean = ((float)dmeanx - (mean * dvar)) * rF;
            hg[0] = (dxn0 * rstd) + (dmean + (y[0] * dvar * rF)) * (float)s_cnt[lane];
            hg[1] = (dxn1 * rstd) + (dmean + (y[1] * dvar * rF)) * (float)s_cnt[lane + 32];
            store_edge_tables<true>(s_edge, lane, y, d, dmean, dvar * rF);
            if (lane == 0) {
                a.dvar[node] = dvar;
                a.dmean[node] = dmean;
                s_node[0] = a.gamma * rstd;
                s_node[1] = a.bias * dvar * rF;
            }
        }
        s_hg[lane] = hg[0];
        s_hg[lane + 32] = hg[1];
        __syncwarp();
        const float2 gw = pattern_sums_to_table_grads(reinterpret_cast<const float2 *>(s_hg)[lane], lane, a.bias);
        float *dst = a.dW + (size_t)node * 64 + 2 * lane;
        dst[0] += gw.x;
        dst[1] += gw.y;
        __syncwarp();
        if (lane == 0) grid_clear_wait(clear, a.dW + (size_t)node * 64, s_edge, 6 * 64);
    }
    __syncthreads();
    float D[6], base[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        D[j] = s_edge[64 * j + lane];
        base[j] = BN && j == 5 ? s_edge[64 * j + 32 + lane] : 0.0f;          // input 5 is split off here, so one base table serves all six
    }
    const float gain = BN ? s_node[0] : 1.0f, slope = BN ? s_node[1] : 0.0f;
    const uint32_t mask_lo = BN ? s_mask[0] : 0u, mask_hi = BN ? s_mask[1] : 0u;
    for (int f_warp = 4 * 32 * warp; f_warp < a.F; f_warp += step) {
        const int f = f_warp + 4 * lane;
        const uint32_t p4 = f == f_first ? p_first : small_patterns<XBIT>(a, rows, f, lane);
        const float4 gq = f == f_first ? g_first : load_frames(dyrow, f, a.F, a.vec);
        float g[4] = {gq.x, gq.y, gq.z, gq.w};
        const uint32_t q2[2] = {__byte_perm(p4, 0u, 0x4140) * 65u, __byte_perm(p4, 0u, 0x4342) * 65u};
        if (BN) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t q = q2[i >> 1] >> (16 * (i & 1));
                const bool upper = (q & 32u) != 0u;
                const float add = fmaf(upper ? slope : -slope, __shfl_sync(kFull, D[5], q), __shfl_sync(kFull, base[5], q));
                const bool pass = ((upper ? mask_hi : mask_lo) >> (q & 31u)) & 1u;
                g[i] = f + i < a.F ? fmaf(pass ? g[i] : 0.0f, gain, add) : 0.0f;
            }
        }
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = g[i] * __shfl_sync(kFull, D[j], q2[i >> 1] >> (16 * (i & 1) + j + 1));
            float *dst = a.dx + out[j] + f;
            if (a.vec) {
                if (f < a.F) red_add_v4(dst, v[0], v[1], v[2], v[3]);        // rows are padded to whole quads; frames from F on add 0
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (f + i < a.F) atomicAdd(dst + i, v[i]);
            }
        }
    }
}

// Where the one-launch kernels pay.  Measured on B200, forward + backward of a layer on fp32 frames against the general kernels: 360
// nodes x 100 frames 17 / 55 us, 1024 x 1024 41 / 66, 2048 x 1000 (2^21 node-frames) 70 / 86, 8192 x 256 71 / 120, but 4096 x 1000
// 129 / 115; and however few the nodes, a CTA works through its frames alone: 64 x 16384 125 / 64.
bool small_layer(int O, int F) { return (long long)O * F <= kSmallLayer && F <= 4096; }

// Warps of a CTA: in the forward as many as there are rounds of frames.  In the backward, of which an SM holds 24, a wave costs about as much as a
// round, 2.7 us (sweep of 58 layers with 1, 2, 3, 4 and 8 warps; as many warps as rounds -> this rule, in us: 1024 nodes x 512 frames 14.6 -> 12.3,
// 982 x 1670 35.6 -> 28.9, 550 x 927 16.3 -> 13.8, 3428 x 415 28.4 -> 25.9, 2816 x 596 34.1 -> 28.6).
unsigned small_threads(int F) { return 32u * (unsigned)(F > 128 * kWarpsPerCta ? kWarpsPerCta : (F + 127) / 128); }
unsigned small_backward_threads(int O, int F) { return small_layer_threads(O, F, 24, 27, 27); }

// Whether O CTAs take no more waves on SMs that hold `few` warps (and 32 CTAs) than on SMs that hold `many`: then the kernel with more registers is the
// faster one.  In us with many / few: forward on fp32 rows 948 nodes x 1174 frames 10.8 / 14.5, 393 x 1032 8.8 / 8.4, 8635 x 78 14.5 / 14.0; backward on
// bit rows 948 x 1174 16.3 / 24.0, 393 x 1032 10.7 / 16.4, 1159 x 115 9.0 / 8.1, 1930 x 158 12.0 / 11.3.
bool waves_as_few(int O, unsigned threads, int few, int many)
{
    const int warps = (int)threads / 32, sms = device_info().sm_count;
    auto waves = [&](int hold) { const int slots = sms * (hold / warps < 32 ? hold / warps : 32); return (O + slots - 1) / slots; };
    return waves(few) <= waves(many);
}

struct Scratch {
    float    *Y;        // [O][64]
    uint32_t *hist;     // [O][64]
    int      *table;    // [O][2]
    unsigned char *pat; // extra bytes asked for by the caller (pattern bytes of the fp32 binary-mode training forward)
};

// What the statistics half of a frame-sharded backward left in a stream's scratch (pattern counts, per-pattern dy sums, pattern
// bytes and masks), so that the apply half that follows it on the same stream need not repeat that pass.  It holds while nobody has been
// handed the block (`ticket`), within one capture of the stream or outside of any (`capture`), and for the same call; the apply half
// redoes the pass when something differs.
struct PassOneRecord {
    const void *x, *dy, *idx, *W, *mean, *rstd;
    float gamma, beta, bias;
    int O, F, lut_binarize;
    long long fs;
    unsigned long long ticket, capture;
    bool operator==(const PassOneRecord &r) const
    {
        return x == r.x && dy == r.dy && idx == r.idx && W == r.W && mean == r.mean && rstd == r.rstd && gamma == r.gamma && beta == r.beta && bias == r.bias &&
               O == r.O && F == r.F && lut_binarize == r.lut_binarize && fs == r.fs && ticket == r.ticket && capture == r.capture;
    }
};
// what such a record reads at this moment; ticket 0 when the stream cannot be asked
PassOneRecord pass_one(const void *x, const void *dy, const void *idx, const void *W, const void *mean, const void *rstd, float gamma, float beta, float bias,
                       int O, int F, int lut_binarize, long long fs, cudaStream_t st)
{
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long capture = 0;
    const bool known = cudaStreamGetCaptureInfo(st, &status, &capture) == cudaSuccess;
    if (!known) cudaGetLastError();
    return PassOneRecord{x, dy, idx, W, mean, rstd, gamma, beta, bias, O, F, lut_binarize, fs, known ? stream_scratch_ticket(st, 1) : 0,
                         status == cudaStreamCaptureStatusActive ? capture : 0};
}
std::mutex g_record_mu;
std::map<std::pair<int, cudaStream_t>, PassOneRecord> g_records;

std::pair<int, cudaStream_t> record_key(cudaStream_t st)
{
    int dev = 0;
    cudaGetDevice(&dev);
    return std::make_pair(dev, st);
}

bool carve(Scratch &s, int O, cudaStream_t st, size_t extra = 0)
{
    const size_t per_node = 64 * 4 + 64 * 4 + 8 + 64 * 4;        // Y, pattern counts, truth table, per-pattern dy sums
    const size_t fixed = (per_node * (size_t)O + 255) & ~(size_t)255;
    unsigned char *base = static_cast<unsigned char *>(stream_scratch(st, fixed + extra, 1));
    if (base == nullptr) return false;
    s.pat = base + fixed;
    s.Y = reinterpret_cast<float *>(base);
    s.hist = reinterpret_cast<uint32_t *>(base + (size_t)O * 256);
    s.table = reinterpret_cast<int *>(base + (size_t)O * 768);
    return true;
}

int run_binary_lut(const int *x, int *y, const int *idx, const int *table, int O, int F, int stride, cudaStream_t st)
{
    int rc = bbcu_bit_BinaryLut6_Forward(x, y, idx, table, O, F, stride, reinterpret_cast<bbcu_stream_t>(st));
    if (rc) return rc;
    if (F & 31) {
        launch(k_clear_tail_bits, (O + 255) / 256, 256, 0, st, reinterpret_cast<uint32_t *>(y), O, F, stride);
        return launch_status();
    }
    return BBCU_OK;
}

}   // namespace

// StochasticLut6 bit -> bit (with_bn = false) and DifferentiableLut6 bit inference (with_bn = true).  Returns
// BBCU_ERR_NO_MEMORY when the scratch cannot be had; the caller then falls back to the per-frame kernel.
int bit_forward_by_table(bool with_bn, const int *x, int *y, const int *idx, const float *W, const float *rmean, const float *rvar, float gamma,
                         float beta, float bias, int O, int F, int stride, int lut_binarize, cudaStream_t st)
{
    if (O == 0 || F == 0) return BBCU_OK;
    Scratch s;
    if (!carve(s, O, st)) return BBCU_ERR_NO_MEMORY;
    const int blocks = (O + kWarpsPerCta - 1) / kWarpsPerCta;
    if (with_bn) launch(k_pattern_values<kTableNorm>, blocks, kWarpsPerCta * 32, 0, st, W, nullptr, s.table, rmean, rvar, gamma, beta, bias, O, lut_binarize);
    else         launch(k_pattern_values<kTableRaw>, blocks, kWarpsPerCta * 32, 0, st, W, nullptr, s.table, nullptr, nullptr, 0.0f, 0.0f, bias, O, lut_binarize);
    BB200_CUDA(cudaPeekAtLastError());
    return run_binary_lut(x, y, idx, s.table, O, F, stride, st);
}

int dl6_bit_forward_training_by_table(const int *x, int *y, const int *idx, const float *W, float *mean, float *rstd, float *rmean, float *rvar,
                                      float gamma, float beta, float momentum, float bias, int O, int F, int stride, int lut_binarize,
                                      cudaStream_t st)
{
    if (O == 0 || F == 0) return BBCU_OK;
    if (small_layer(O, F)) {
        SmallBinArgs a = {};
        a.x = x; a.y = y; a.idx = idx; a.W = W; a.mean = mean; a.rstd = rstd; a.running_mean = rmean; a.running_var = rvar;
        a.gamma = gamma; a.beta = beta; a.momentum = momentum; a.bias = bias; a.F = F; a.lut_binarize = lut_binarize; a.xs = stride; a.ys = stride;
        launch(k_small_binary_forward<true, 64>, O, small_threads(F), 0, st, a);
        return launch_status();
    }
    Scratch s;
    if (!carve(s, O, st)) return BBCU_ERR_NO_MEMORY;
    const int groups = (O + kWarpsPerCta - 1) / kWarpsPerCta;
    launch(k_pattern_values<kTableNone>, groups, kWarpsPerCta * 32, 0, st, W, s.Y, nullptr, nullptr, nullptr, 0.0f, 0.0f, bias, O, lut_binarize);
    BB200_CUDA(cudaPeekAtLastError());
    BB200_CUDA(cudaMemsetAsync(s.hist, 0, (size_t)O * 256, st));
    // word tiles: wide enough to amortise the 64-counter reduction (about 400 instructions per warp), narrow enough to fill the GPU
    const int words = (F + 31) / 32;
    int tile_words = 4096;
    const int hist_groups = (O + kHistWarps - 1) / kHistWarps;
    while (tile_words > 32 && (long long)hist_groups * ((words + tile_words - 1) / tile_words) < 4LL * device_info().sm_count) tile_words /= 2;
    const long long blocks = (long long)hist_groups * ((words + tile_words - 1) / tile_words);
    BB200_REQUIRE(blocks < (1LL << 31), BBCU_ERR_TOO_LARGE);
    launch(k_pattern_histogram, (unsigned)blocks, kHistWarps * 32, 0, st, reinterpret_cast<const uint32_t *>(x), idx, s.hist, O, F, stride, hist_groups,
                                                                     tile_words);
    BB200_CUDA(cudaPeekAtLastError());
    launch(k_dl6_bit_train_finalize, groups, kWarpsPerCta * 32, 0, st, s.Y, s.hist, s.table, mean, rstd, rmean, rvar, gamma, beta, momentum, O, F);
    BB200_CUDA(cudaPeekAtLastError());
    return run_binary_lut(x, y, idx, s.table, O, F, stride, st);
}

// StochasticLut6 bit -> fp32 forward.
int bit_fp32_forward_by_table(const int *x, float *y, const int *idx, const float *W, float bias, int O, int F, long long xs, long long ys,
                              int lut_binarize, cudaStream_t st)
{
    if (O == 0 || F == 0) return BBCU_OK;
    Scratch s;
    if (!carve(s, O, st)) return BBCU_ERR_NO_MEMORY;
    const int groups = (O + kWarpsPerCta - 1) / kWarpsPerCta;
    launch(k_pattern_values<kTableNone>, groups, kWarpsPerCta * 32, 0, st, W, s.Y, nullptr, nullptr, nullptr, 0.0f, 0.0f, bias, O, lut_binarize);
    BB200_CUDA(cudaPeekAtLastError());
    // frame tiles as in the other LUT kernels: the tile's input rows stay in L2 while all nodes consume them
    const int tf = frame_tile(3LL * O, 1, groups, F, 1 << 20);
    const int tile_words = ((tf + 1023) / 1024) * 32;
    const long long blocks = (long long)groups * (((F + 31) / 32 + tile_words - 1) / tile_words);
    BB200_REQUIRE(blocks < (1LL << 31), BBCU_ERR_TOO_LARGE);
    launch(k_bit_gather_forward, (unsigned)blocks, kWarpsPerCta * 32, 0, st, reinterpret_cast<const uint32_t *>(x), y, idx, s.Y, O, F, xs, ys, groups,
                                                                        tile_words);
    return launch_status();
}

// Binary mode on fp32 frames.  mode 0: StochasticLut6 forward (y = clip of the per-pattern value); 1: DifferentiableLut6 inference
// (running statistics); 2: DifferentiableLut6 training forward (batch statistics from the pattern counts); 3: the statistics half of a
// frame-sharded training forward (raw per-pattern values into y, this rank's fp64 sums [O][2] through the `mean` argument).  Declines (NO_MEMORY) when the
// rows are not 16-byte aligned or the pattern bytes of the training forward would not be a reasonable scratch.
int f32_binary_forward_by_table(int mode, const float *x, float *y, const int *idx, const float *W, float *mean, float *rstd, float *rmean,
                                float *rvar, float gamma, float beta, float momentum, float bias, int O, int F, long long fs, int lut_binarize,
                                cudaStream_t st)
{
    if (O == 0 || F == 0) return BBCU_OK;
    const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0 && fs % 4 == 0;
    if (mode == 2 && small_layer(O, F)) {
        SmallBinArgs a = {};
        a.x = x; a.y = y; a.idx = idx; a.W = W; a.mean = mean; a.rstd = rstd; a.running_mean = rmean; a.running_var = rvar;
        a.gamma = gamma; a.beta = beta; a.momentum = momentum; a.bias = bias; a.F = F; a.lut_binarize = lut_binarize; a.xs = fs; a.ys = fs; a.vec = aligned;
        const unsigned threads = small_threads(F);
        launch(waves_as_few(O, threads, 48, 64) ? k_small_binary_forward<false, 48> : k_small_binary_forward<false, 64>, O, threads, 0, st, a);
        return launch_status();
    }
    if (!aligned) return BBCU_ERR_NO_MEMORY;
    const size_t pat_bytes = mode == 2 ? (size_t)O * (size_t)fs : 0;
    if (pat_bytes > ((size_t)1 << 30)) return BBCU_ERR_NO_MEMORY;
    Scratch s;
    if (!carve(s, O, st, pat_bytes)) return BBCU_ERR_NO_MEMORY;
    F32BinArgs a = {};
    a.x = x; a.y = y; a.idx = idx; a.Y = s.Y; a.hist = s.hist; a.O = O; a.F = F; a.fs = fs;
    a.groups = (O + kWarpsPerCta - 1) / kWarpsPerCta;
    const unsigned threads = kWarpsPerCta * 32;
    // frame tiles narrow enough for the tile's input rows to stay in L2 while every node reads them
    const int tf = frame_tile(3LL * O, 32, a.groups, F, 1 << 20);
    a.tile_frames = ((tf + 127) / 128) * 128;
    if (a.tile_frames < 1024) a.tile_frames = 1024;               // at least eight steps per warp and tile: set-up and the 64 count atomics amortise
    const long long blocks = (long long)a.groups * ((F + a.tile_frames - 1) / a.tile_frames);
    BB200_REQUIRE(blocks < (1LL << 31), BBCU_ERR_TOO_LARGE);
    if (mode == 0) {
        launch(k_pattern_values<kTableNone>, a.groups, threads, 0, st, W, s.Y, nullptr, nullptr, nullptr, 0.0f, 0.0f, bias, O, lut_binarize);
        BB200_CUDA(cudaPeekAtLastError());
        launch(k_f32_binary_forward<kPassDirect>, (unsigned)blocks, threads, 0, st, a);
        return launch_status();
    }
    if (mode == 3) {          // first half of a sharded training forward: raw values into y, per-rank sums (mean doubles as the sums pointer)
        launch(k_pattern_values<kTableNone>, a.groups, threads, 0, st, W, s.Y, nullptr, nullptr, nullptr, 0.0f, 0.0f, bias, O, lut_binarize);
        BB200_CUDA(cudaPeekAtLastError());
        BB200_CUDA(cudaMemsetAsync(s.hist, 0, (size_t)O * 256, st));
        launch(k_f32_binary_forward<kPassStats>, (unsigned)blocks, threads, 0, st, a);
        BB200_CUDA(cudaPeekAtLastError());
        launch(k_counts_to_sums, a.groups, threads, 0, st, s.Y, s.hist, reinterpret_cast<double *>(mean), O);
        return launch_status();
    }
    if (mode == 1) {
        launch(k_pattern_values<kTableNorm>, a.groups, threads, 0, st, W, nullptr, s.table, rmean, rvar, gamma, beta, bias, O, lut_binarize);
        BB200_CUDA(cudaPeekAtLastError());
        a.table = s.table;
        launch(k_f32_binary_forward<kPassDirect>, (unsigned)blocks, threads, 0, st, a);
        return launch_status();
    }
    launch(k_pattern_values<kTableNone>, a.groups, threads, 0, st, W, s.Y, nullptr, nullptr, nullptr, 0.0f, 0.0f, bias, O, lut_binarize);
    BB200_CUDA(cudaPeekAtLastError());
    BB200_CUDA(cudaMemsetAsync(s.hist, 0, (size_t)O * 256, st));
    a.pat = s.pat;
    launch(k_f32_binary_forward<kPassCount>, (unsigned)blocks, threads, 0, st, a);
    BB200_CUDA(cudaPeekAtLastError());
    launch(k_dl6_bit_train_finalize, a.groups, threads, 0, st, s.Y, s.hist, s.table, mean, rstd, rmean, rvar, gamma, beta, momentum, O, F);
    BB200_CUDA(cudaPeekAtLastError());
    a.table = s.table;
    launch(k_f32_binary_forward<kPassOutput>, (unsigned)blocks, threads, 0, st, a);
    return launch_status();
}

// ---------------------------------------------------------------------------------------------- backward launchers
namespace {

// Scratch and arguments shared by all backward calls.  The block in slot 1 has the same size whatever the call (sums, counts, masks,
// look-up tables, pattern bytes), so that the apply half of a frame-sharded backward finds what its statistics half left there.
bool backward_setup(BitBwdArgs &a, const void *x, const float *dy, const int *idx, int O, int F, long long xs, long long fs, cudaStream_t st)
{
    const long long ps = ((long long)F + 127) / 128 * 128;
    const size_t tables = (size_t)O * (6 * 64 * sizeof(float) + sizeof(float2) + sizeof(uint2));
    if ((size_t)O * (size_t)ps > ((size_t)1 << 32)) return false;        // 4 GiB of patterns at most
    Scratch s;
    if (!carve(s, O, st, ((tables + 255) & ~(size_t)255) + (size_t)O * (size_t)ps)) return false;
    a = BitBwdArgs{};
    a.x = static_cast<const uint32_t *>(x); a.dy = dy; a.idx = idx;
    a.hist = s.hist;
    a.hdy = reinterpret_cast<float *>(s.hist) + (size_t)O * 64;          // the block between the pattern counts and the truth tables
    a.etab = reinterpret_cast<float *>(s.pat);
    a.ntab = reinterpret_cast<float2 *>(a.etab + (size_t)O * 6 * 64);
    a.mask = reinterpret_cast<uint2 *>(a.ntab + O);
    a.pat = s.pat + ((tables + 255) & ~(size_t)255);
    a.O = O; a.F = F; a.xs = xs; a.fs = fs; a.ps = ps;
    a.vec = (reinterpret_cast<uintptr_t>(dy) & 15) == 0 && fs % 4 == 0;
    return true;
}

bool pack_bits(const float *x, uint32_t *bits, int I, int F, long long xs, long long ws, cudaStream_t st)
{
    const int runs = (int)((ws + 31) / 32);
    const long long blocks = ((long long)I * runs + kWarpsPerCta - 1) / kWarpsPerCta;
    if (blocks >= (1LL << 31)) return false;
    launch(k_pack_bits, (unsigned)blocks, kWarpsPerCta * 32, 0, st, x, bits, I, F, xs, ws, runs);
    return true;
}

// How k_pattern_gather divides its work.  The tile is 512 frames (the tables of a consumer are loaded once per tile) unless the dy and
// pattern rows of such a tile, 5 bytes per node and frame, exceed two thirds of L2, or the GPU would run short of warps.  The warps of a
// CTA are chosen by the average number of consumers of a row; a row with more than eight times the average, and more than 64, is heavy.
// Backward of 8192 x 8192 nodes x 16384 frames: even wiring 811 us; one row feeding every node 7210 as the loop of one CTA per tile, 2765 / 990 /
// 886 with 1 / 4 / 8 CTAs per SM for the chunks (which cost nothing where there are none).  2048 x 2048 x 2048: 66; 1035, 95 / 72 / 72.
void gather_shape(BitBwdArgs &a)
{
    const DeviceInfo &di = device_info();
    const long long fan = (6LL * a.O + a.I - 1) / a.I;
    int nc = 4;
    while (nc > 1 && (5LL * a.O * 128 * nc > (long long)(di.l2_bytes / 3 * 2) || (long long)a.I * ((a.fs + 128 * nc - 1) / (128 * nc)) < 16LL * di.sm_count)) nc /= 2;
    a.nc = nc;
    a.tiles = (int)((a.fs + 128 * nc - 1) / (128 * nc));
    const long long blocks = (long long)a.I * a.tiles;
    a.split = 1;
    while (a.split < kWarpsPerCta && (fan >= 32LL * a.split || (fan >= 4LL * a.split && blocks * a.split < 8LL * di.sm_count))) a.split *= 2;
    const long long heavy_from = 8 * fan > 64 ? 8 * fan : 64;
    a.heavy_from = (int)(heavy_from < (1 << 30) ? heavy_from : 1 << 30);
    a.heavy_chunk = 32 * a.split <= a.heavy_from / 2 ? 32 * a.split : a.heavy_from / 2;
    a.heavy_ctas = 8 * di.sm_count;
}

// Words of a packed row: whole 16-byte pieces, which k_pattern_sums reads with one load, or no padding where only then the rows take no more than the
// limit.  (Beyond it a backward goes through the per-node kernels.)
constexpr long long kPackedBytes = 1LL << 30;
constexpr long long packed_row_words(long long rows, long long frames)
{
    const long long padded = (frames + 127) / 128 * 4;
    return rows * padded * 4 <= kPackedBytes ? padded : (frames + 31) / 32;
}
static_assert(packed_row_words(1LL << 26, 33) == 4 && packed_row_words((1LL << 26) + 1, 33) == 2 && packed_row_words(1LL << 27, 33) * (1LL << 27) * 4 == kPackedBytes,
              "whatever fits without padding is packed");

// Slot 3 of the stream's scratch: consumer lists, the chunks of heavy rows, and the bits of the I rows where x is fp32.  The block is the same
// size when they need not be packed, so that a call after which that is known does not have to grow it.
bool input_side(BitBwdArgs &a, int I, bool x_is_fp32, bool packed, cudaStream_t st)
{
    if (I == 0) return false;
    a.I = I;
    gather_shape(a);
    const int edges = 6 * a.O;
    const long long ws = packed_row_words(I, a.F);
    // a heavy row has more than heavy_from >= 2 heavy_chunk consumers, so its chunks number at most 3 / 2 of its consumers over heavy_chunk
    const size_t heavy_most = (size_t)edges / (size_t)a.heavy_chunk * 3 / 2 + 2;
    const size_t list_bytes = (heavy_most * sizeof(int2) + (2 * (size_t)I + 2 + (size_t)edges) * sizeof(int) + 255) & ~(size_t)255;
    size_t bit_bytes = x_is_fp32 ? (size_t)I * (size_t)ws * 4 : 0;
    if (bit_bytes > (size_t)kPackedBytes) {
        if (!packed) return false;
        bit_bytes = 0;
    }
    int2 *heavy = static_cast<int2 *>(stream_scratch(st, list_bytes + bit_bytes, 3));
    if (heavy == nullptr) return false;
    int *count = reinterpret_cast<int *>(heavy + heavy_most), *total = count + I, *heavy_count = total + 1, *cursor = heavy_count + 1, *list = cursor + I;
    a.edge_count = count; a.edge_end = cursor; a.edges = list; a.heavy = heavy; a.heavy_count = heavy_count;
    cudaMemsetAsync(count, 0, ((size_t)I + 2) * sizeof(int), st);
    launch(k_edge_count, (edges + 255) / 256, 256, 0, st, a.idx, count, edges);
    launch(k_edge_room, (I + 255) / 256, 256, 0, st, count, cursor, total, I, heavy, heavy_count, a.heavy_from, a.heavy_chunk);
    launch(k_edge_fill, (edges + 255) / 256, 256, 0, st, a.idx, cursor, list, edges, heavy, heavy_count, a.dx, a.fs);
    if (x_is_fp32 && !packed) {
        uint32_t *bits = reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned char *>(heavy) + list_bytes);
        if (!pack_bits(reinterpret_cast<const float *>(a.x), bits, I, a.F, a.xs, ws, st)) return false;
        a.x = bits;
        a.xs = ws;
    }
    return true;
}

// Pattern sums (and counts) and pattern bytes.  Tiles as wide as still give every SM two rounds of warps: the columns of a tile cost
// about as much to clear and add up as 500 frames.
template <bool XF32>
int launch_pattern_sums(BitBwdArgs a, bool bn, cudaStream_t st)
{
    a.groups = (a.O + kPsWarps - 1) / kPsWarps;
    const bool xvec = (reinterpret_cast<uintptr_t>(a.x) & 15) == 0 && a.xs % 4 == 0;
    if (XF32) a.vec = a.vec && xvec;
    long long tile = ((long long)a.F + 127) / 128 * 128;
    while (tile > 1024 && (long long)a.O * ((a.F + tile - 1) / tile) < 24LL * device_info().sm_count) tile = (tile / 2 + 127) / 128 * 128;
    a.tile_frames = (int)tile;
    a.tiles = (int)((a.F + tile - 1) / tile);
    const long long blocks = (long long)a.groups * a.tiles;
    BB200_REQUIRE(blocks < (1LL << 31), BBCU_ERR_TOO_LARGE);
    if (a.tiles > 1) {
        BB200_CUDA(cudaMemsetAsync(a.hdy, 0, (size_t)a.O * 256, st));
        if (bn) BB200_CUDA(cudaMemsetAsync(a.hist, 0, (size_t)a.O * 256, st));
    }
    const int smem = kPsWarps * 64 * 32 * (int)(bn ? sizeof(PatternSlot<true>) : sizeof(PatternSlot<false>));
    void (*kern)(BitBwdArgs) = k_pattern_sums<XF32, true, true>;
    if constexpr (!XF32) {
        if (!bn) kern = xvec ? k_pattern_sums<false, false, true> : k_pattern_sums<false, false, false>;
        else if (!xvec) kern = k_pattern_sums<false, true, false>;
    }
    BB200_REQUIRE(allow_big_smem(kern, smem), BBCU_ERR_NO_MEMORY);
    launch(kern, (unsigned)blocks, kPsWarps * 32, smem, st, a);
    return launch_status();
}

int launch_pattern_gather(BitBwdArgs a, bool bn, cudaStream_t st)
{
    a.vec = a.vec && (reinterpret_cast<uintptr_t>(a.dx) & 15) == 0;
    const int nc = a.nc;
    const long long blocks = (long long)a.I * a.tiles + a.heavy_ctas;
    BB200_REQUIRE(blocks < (1LL << 31), BBCU_ERR_TOO_LARGE);
    const int smem = a.split > 1 ? a.split * nc * 32 * (int)sizeof(float4) : 0;
    auto kern = bn ? (nc == 4 ? k_pattern_gather<true, 4> : nc == 2 ? k_pattern_gather<true, 2> : k_pattern_gather<true, 1>)
                   : (nc == 4 ? k_pattern_gather<false, 4> : nc == 2 ? k_pattern_gather<false, 2> : k_pattern_gather<false, 1>);
    launch(kern, (unsigned)blocks, a.split * 32, smem, st, a);
    return launch_status();
}

}   // namespace

// Training forward in binary mode by way of the bit operators: pack the rows, count patterns and evaluate truth tables on bits, expand the
// output.  Per node-frame that moves 4 bytes of y (and 4 per input row and frame) against the 24 + 1 that the per-node passes of
// f32_binary_forward_by_table() read through L2, for two launches more, a reduction of 64 counters per node that costs about as much as 1500
// frames, and packing that grows with the rows.  Measured on B200 (220 layers of 2^22 to 2^27 node-frames, 256 to 40000 frames and 0.25 to 3
// rows a node; packed / by node): 8192 nodes x 16384 frames 292 / 368 us with a row a node, 377 / 412 with two, 422 / 430 with two and a
// half; 8192 x 4096 125 / 121 with two; 4096 x 4096 63.2 / 62.4 with one and a half; 1024 x 4096 25.7 / 21.3 with one; 30000 x 300 107 / 58;
// 23000 x 780 105 / 85; 20676 x 1164 112 / 103.  With the rule below a layer takes 0.5 % longer than with the better of the two, on average
// (always by node 6 %, packed up to two rows a node whatever the size 14 %).
static bool packed_forward_pays(int I, int O, int F, long long fs, bool aligned)
{
    const long long node_frames = (long long)O * F;
    if (!aligned || (long long)O * fs > (1LL << 30)) return I <= 2LL * O;              // by node declines these
    if (node_frames >= 3LL << 24) return F >= 1024 && I <= 2LL * O;                    // rows of fp32 frames no longer stay in L2
    return node_frames >= 1LL << 23 && F >= 3072 && 2LL * I <= 3LL * O;
}

int f32_binary_forward_packed(const float *x, float *y, const int *idx, const float *W, float *mean, float *rstd, float *rmean, float *rvar,
                              float gamma, float beta, float momentum, float bias, int I, int O, int F, long long fs, int lut_binarize,
                              cudaStream_t st)
{
    const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0 && fs % 4 == 0;
    if (small_layer(O, F) || I < 1 || !packed_forward_pays(I, O, F, fs, aligned)) return BBCU_ERR_NO_MEMORY;
    const long long ws = ((long long)F + 127) / 128 * 4;                // whole 16-byte pieces
    const size_t x_bytes = (size_t)I * (size_t)ws * 4, y_bytes = (size_t)O * (size_t)ws * 4;
    if (x_bytes + y_bytes > ((size_t)1 << 30)) return BBCU_ERR_NO_MEMORY;
    uint32_t *xb = static_cast<uint32_t *>(stream_scratch(st, x_bytes + y_bytes, 3));
    if (xb == nullptr) return BBCU_ERR_NO_MEMORY;
    int *yb = reinterpret_cast<int *>(xb + (size_t)I * (size_t)ws);
    if (!pack_bits(x, xb, I, F, fs, ws, st)) return BBCU_ERR_NO_MEMORY;
    BB200_CUDA(cudaPeekAtLastError());
    const int rc = dl6_bit_forward_training_by_table(reinterpret_cast<const int *>(xb), yb, idx, W, mean, rstd, rmean, rvar, gamma, beta, momentum, bias,
                                                     O, F, (int)ws, lut_binarize, st);
    if (rc) return rc;
    return bbcu_fp32_ConvBitToReal(yb, y, 0.0f, 1.0f, O, F, (int)ws, (int)fs, reinterpret_cast<bbcu_stream_t>(st));
}

// Backward of the bit-input layers (StochasticLut6: bn = false; DifferentiableLut6: bn = true); writes all of dx's I rows.
int bit_backward_by_table(bool bn, bool x_is_fp32, const void *x, const float *dy, float *dx, const int *idx, const float *W, float *dW,
                          const float *mean, const float *rstd, float *dmean_out, float *dvar_out, float gamma, float beta, float bias, int I, int O,
                          int F, long long xs, long long fs, int lut_binarize, cudaStream_t st)
{
    if (x_is_fp32 && xs != fs) return BBCU_ERR_NO_MEMORY;          // fp32 x shares the stride of dy / dx in every caller; otherwise decline
    if (small_layer(O, F)) {
        SmallBinArgs a = {};
        a.x = x; a.dy = dy; a.dx = dx; a.idx = idx; a.W = W; a.dW = dW; a.mean_in = mean; a.rstd_in = rstd; a.dmean = dmean_out; a.dvar = dvar_out;
        a.gamma = gamma; a.beta = beta; a.bias = bias; a.F = F; a.lut_binarize = lut_binarize; a.xs = xs; a.fs = fs;
        a.vec = ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dx) | (x_is_fp32 ? reinterpret_cast<uintptr_t>(x) : 0)) & 15) == 0 && fs % 4 == 0;
        GridClear clear;
        const int rcc = grid_clear_setup(clear, dx, (size_t)I * (size_t)fs, st);
        if (rcc) return rcc;
        const unsigned threads = small_backward_threads(O, F);
        auto kern = x_is_fp32 ? (bn ? k_small_binary_backward<false, true, 24> : k_small_binary_backward<false, false, 24>)
                  : waves_as_few(O, threads, 16, 24) ? (bn ? k_small_binary_backward<true, true, 16> : k_small_binary_backward<true, false, 16>)
                                                     : (bn ? k_small_binary_backward<true, true, 24> : k_small_binary_backward<true, false, 24>);
        launch(kern, O, threads, 0, st, a, clear);
        return launch_status();
    }
    BitBwdArgs a;
    if (!backward_setup(a, x, dy, idx, O, F, xs, fs, st)) return BBCU_ERR_NO_MEMORY;
    a.dx = dx;
    if (!input_side(a, I, x_is_fp32, false, st)) return BBCU_ERR_NO_MEMORY;
    BB200_CUDA(cudaPeekAtLastError());
    const unsigned blocks = (unsigned)((O + kWarpsPerCta - 1) / kWarpsPerCta), threads = kWarpsPerCta * 32;
    if (bn) launch(k_pattern_masks, blocks, threads, 0, st, W, a.mask, mean, rstd, gamma, beta, bias, O, lut_binarize);
    else    launch(k_pattern_derivatives, blocks, threads, 0, st, W, a.etab, bias, O, lut_binarize);
    BB200_CUDA(cudaPeekAtLastError());
    const int rc = launch_pattern_sums<false>(a, bn, st);
    if (rc) return rc;
    if (bn) launch(k_bit_backward_finalize<true>, blocks, threads, 0, st, a.hdy, a.hist, a.mask, W, a.etab, a.ntab, dW, mean, rstd, dmean_out, dvar_out, gamma, beta,
                                                                     bias, O, 1.0f / (float)F, lut_binarize, nullptr, nullptr);
    else    launch(k_bit_backward_finalize<false>, blocks, threads, 0, st, a.hdy, nullptr, nullptr, nullptr, nullptr, nullptr, dW, nullptr, nullptr, nullptr, nullptr,
                                                                      0.0f, 0.0f, bias, O, 0.0f, lut_binarize, nullptr, nullptr);
    BB200_CUDA(cudaPeekAtLastError());
    return launch_pattern_gather(a, bn, st);
}

// ---- the two halves of the batch-norm backward for frame-sharded callers (binary mode on fp32 rows)
// Statistics half: this rank's (dstd, dmeanx) per node into `sums` ([O][2] fp64), to be added over the ranks by the caller.  (The number of
// input rows is not known here, so the patterns come straight from the fp32 rows.)
int bit_backward_stats_by_table(const float *x, const float *dy, const int *idx, const float *W, const float *mean, const float *rstd, double *sums,
                                float gamma, float beta, float bias, int O, int F, long long fs, int lut_binarize, cudaStream_t st)
{
    if (O == 0) return BBCU_OK;
    if (F == 0) { BB200_CUDA(cudaMemsetAsync(sums, 0, sizeof(double) * 2 * (size_t)O, st)); return BBCU_OK; }
    BitBwdArgs a;
    if (!backward_setup(a, x, dy, idx, O, F, fs, fs, st)) return BBCU_ERR_NO_MEMORY;
    const unsigned blocks = (unsigned)((O + kWarpsPerCta - 1) / kWarpsPerCta), threads = kWarpsPerCta * 32;
    launch(k_pattern_masks, blocks, threads, 0, st, W, a.mask, mean, rstd, gamma, beta, bias, O, lut_binarize);
    BB200_CUDA(cudaPeekAtLastError());
    int rc = launch_pattern_sums<true>(a, true, st);
    if (rc) return rc;
    launch(k_bit_backward_finalize<true>, blocks, threads, 0, st, a.hdy, a.hist, a.mask, W, nullptr, nullptr, nullptr, mean, rstd, nullptr, nullptr, gamma, beta, bias,
                                                             O, 0.0f, lut_binarize, sums, nullptr);
    rc = launch_status();
    if (rc == BBCU_OK) {
        const PassOneRecord r = pass_one(x, dy, idx, W, mean, rstd, gamma, beta, bias, O, F, lut_binarize, fs, st);
        std::lock_guard<std::mutex> g(g_record_mu);
        g_records[record_key(st)] = r;
    }
    return rc;
}

// Apply half: `sums` hold (dstd, dmeanx) over the frames of ALL ranks, total_frames is their number; writes all of dx's I rows,
// dW receives this rank's share.
int bit_backward_apply_by_table(const float *x, const float *dy, float *dx, const int *idx, const float *W, float *dW, const float *mean,
                                const float *rstd, const double *sums, float *dmean_out, float *dvar_out, float gamma, float beta, float bias, int I,
                                int O, int F, long long fs, long long total_frames, int lut_binarize, cudaStream_t st)
{
    const PassOneRecord now = pass_one(x, dy, idx, W, mean, rstd, gamma, beta, bias, O, F, lut_binarize, fs, st);
    bool have = false;
    {
        std::lock_guard<std::mutex> g(g_record_mu);
        auto it = g_records.find(record_key(st));
        have = it != g_records.end() && now.ticket != 0 && it->second == now;
        if (it != g_records.end()) g_records.erase(it);
    }
    BitBwdArgs a;
    if (!backward_setup(a, x, dy, idx, O, F, fs, fs, st)) return BBCU_ERR_NO_MEMORY;      // the same block as before
    a.dx = dx;
    if (!input_side(a, I, true, have, st)) return BBCU_ERR_NO_MEMORY;
    BB200_CUDA(cudaPeekAtLastError());
    const unsigned blocks = (unsigned)((O + kWarpsPerCta - 1) / kWarpsPerCta), threads = kWarpsPerCta * 32;
    if (!have) {
        launch(k_pattern_masks, blocks, threads, 0, st, W, a.mask, mean, rstd, gamma, beta, bias, O, lut_binarize);
        BB200_CUDA(cudaPeekAtLastError());
        const int rc = launch_pattern_sums<false>(a, true, st);
        if (rc) return rc;
    }
    launch(k_bit_backward_finalize<true>, blocks, threads, 0, st, a.hdy, a.hist, a.mask, W, a.etab, a.ntab, dW, mean, rstd, dmean_out, dvar_out, gamma, beta, bias,
                                                             O, 1.0f / (float)total_frames, lut_binarize, nullptr, sums);
    BB200_CUDA(cudaPeekAtLastError());
    return launch_pattern_gather(a, true, st);
}

}   // namespace bb200
