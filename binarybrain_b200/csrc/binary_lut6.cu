// BinaryLut6: bit-packed 6-input LUT inference forward.
//
// Semantics of BinaryBrain include/bb/BinaryLutN.h:436-463: for every frame the six input bits form an
// index (input k -> bit k) into the node's 64-entry truth table.  Frames are processed 32 per word, by logic on whole words, against the
// 448 operations a word of the reference kernel's 64 masked AND chains (cuda/BinaryLut6.cu:82-160).
//
// Four ways, chosen in bbcu_bit_BinaryLut6_Forward, where the rules and both sides of each stand:
//   k_binary_lut6_imm    15 operations a word with the table bytes as lop3 immediates: layers of several rounds of its grid
//   k_binary_lut6_pipe   a multiplexer tree, 63 operations a word, fed by bulk copies: the other layers with rows on 16-byte boundaries
//   k_binary_lut6_words  the tree, a word of a node per thread: the smallest calls
//   k_binary_lut6        the tree, rows that start anywhere (k_binary_lut6_2pipe: 16-byte boundaries where the others cannot be set up)
// All but the words keep the nodes of one tile of words in flight together, so that the tile's input rows stay in L2 for their readers.

#include <type_traits>

#include "common.cuh"
#include "async_copy.cuh"

namespace bb200 {

constexpr int kBlWarps = 8;

struct BlArgs {
    const uint32_t *x;
    uint32_t *y;
    const int *idx;
    const int *table;
    int O, nwords, Tw, groups;
    long long stride;
};

// level-1 select masks of a node: v_k = (x0 & A[k]) ^ B[k] equals table bit 2k (x0 = 0) / 2k+1 (x0 = 1)
__device__ __forceinline__ uint32_t lut6_word(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t x4, uint32_t x5,
                                              const uint32_t (&A)[32], const uint32_t (&B)[32])
{
    uint32_t v[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = (x0 & A[k]) ^ B[k];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = (v[2 * k] & ~x1) | (v[2 * k + 1] & x1);
#pragma unroll
    for (int k = 0; k < 8; ++k)  v[k] = (v[2 * k] & ~x2) | (v[2 * k + 1] & x2);
#pragma unroll
    for (int k = 0; k < 4; ++k)  v[k] = (v[2 * k] & ~x3) | (v[2 * k + 1] & x3);
#pragma unroll
    for (int k = 0; k < 2; ++k)  v[k] = (v[2 * k] & ~x4) | (v[2 * k + 1] & x4);
    return (v[0] & ~x5) | (v[1] & x5);
}

// Word-at-a-time kernel for rows that are not 16-byte aligned (any stride, any base address).
__global__ void __launch_bounds__(kBlWarps * 32)
k_binary_lut6(const BlArgs a)
{
    grid_dependency();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x / a.groups;
    const int node = (blockIdx.x % a.groups) * kBlWarps + warp;
    if (node >= a.O) return;

    const uint32_t t0 = (uint32_t)__ldg(a.table + 2 * (size_t)node);
    const uint32_t t1 = (uint32_t)__ldg(a.table + 2 * (size_t)node + 1);
    uint32_t A[32], B[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        const uint32_t t  = (k < 16) ? t0 : t1;
        const uint32_t lo = (t >> ((2 * k) & 31)) & 1u, hi = (t >> ((2 * k + 1) & 31)) & 1u;
        B[k] = 0u - lo;
        A[k] = 0u - (lo ^ hi);
    }
    const uint32_t *rows[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) rows[j] = a.x + (size_t)__ldg(a.idx + (size_t)node * 6 + j) * a.stride;
    uint32_t *yrow = a.y + (size_t)node * a.stride;

    const int w_begin = tile * a.Tw;
    const int w_end   = min(a.nwords, w_begin + a.Tw);
    for (int w = w_begin + lane; w < w_end; w += 32) {
        uint32_t xv[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) xv[j] = __ldg(rows[j] + w);
        yrow[w] = lut6_word(xv[0], xv[1], xv[2], xv[3], xv[4], xv[5], A, B);
    }
}

// ---------------------------------------------------------------------------------------------
// Two-pipe variant (aligned rows where the persistent kernels below cannot be set up; its tree is theirs).
//   * Level 1 of the tree only ever produces one of {0, x0, ~x0, ~0}.  In two's complement that is
//     x0 * a + b with (a, b) in {(0,0), (1,0), (-1,-1), (0,-1)}: an integer multiply-add, which issues to the
//     FMA pipe and leaves the 31 selects of levels 2..6 to the INT/logic pipe, so the two pipes split the
//     63 ops per 32 frames about evenly instead of the logic pipe taking all of them.
//   * The 32 (a, b) pairs of a node are derived by 32 lanes in parallel (lane k does pair k) and exchanged
//     through shared memory, instead of every lane deriving all 64 values.
//   * Each lane carries 8 words (two 128-bit loads per input row) per iteration.
// ---------------------------------------------------------------------------------------------
template <typename AB>     // AB: int2[32] in registers, or a pointer to the warp's 32 pairs in shared memory
__device__ __forceinline__ uint32_t lut6_word_imad(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t x4, uint32_t x5,
                                                   const AB &ab)
{
    uint32_t v[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = x0 * (uint32_t)ab[k].x + (uint32_t)ab[k].y;
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = (v[2 * k] & ~x1) | (v[2 * k + 1] & x1);
#pragma unroll
    for (int k = 0; k < 8; ++k)  v[k] = (v[2 * k] & ~x2) | (v[2 * k + 1] & x2);
#pragma unroll
    for (int k = 0; k < 4; ++k)  v[k] = (v[2 * k] & ~x3) | (v[2 * k + 1] & x3);
#pragma unroll
    for (int k = 0; k < 2; ++k)  v[k] = (v[2 * k] & ~x4) | (v[2 * k + 1] & x4);
    return (v[0] & ~x5) | (v[1] & x5);
}

__global__ void __launch_bounds__(kBlWarps * 32)
k_binary_lut6_2pipe(const BlArgs a)
{
    grid_dependency();
    __shared__ int2 s_ab[kBlWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x / a.groups;
    const int node = (blockIdx.x % a.groups) * kBlWarps + warp;
    if (node >= a.O) return;
    {
        // lane k: table bits 2k (x0 = 0) and 2k+1 (x0 = 1) -> (a, b)
        const uint32_t t  = (uint32_t)__ldg(a.table + 2 * (size_t)node + (lane >> 4));
        const uint32_t lo = (t >> ((2 * lane) & 31)) & 1u, hi = (t >> ((2 * lane + 1) & 31)) & 1u;
        s_ab[warp][lane] = make_int2((int)hi - (int)lo, -(int)lo);
        __syncwarp();
    }
    int2 ab[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) ab[k] = s_ab[warp][k];
    const uint32_t *rows[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) rows[j] = a.x + (size_t)__ldg(a.idx + (size_t)node * 6 + j) * a.stride;
    uint32_t *yrow = a.y + (size_t)node * a.stride;

    const int w_begin = tile * a.Tw;
    const int w_end   = min(a.nwords, w_begin + a.Tw);
    for (int w = w_begin + 4 * lane; w < w_end; w += 256) {
        const bool second = (w + 128) < w_end;
        uint4 lo[6], hi[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            lo[j] = __ldg(reinterpret_cast<const uint4 *>(rows[j] + w));
            hi[j] = second ? __ldg(reinterpret_cast<const uint4 *>(rows[j] + w + 128)) : make_uint4(0, 0, 0, 0);
        }
        uint4 o;
        o.x = lut6_word_imad(lo[0].x, lo[1].x, lo[2].x, lo[3].x, lo[4].x, lo[5].x, ab);
        o.y = lut6_word_imad(lo[0].y, lo[1].y, lo[2].y, lo[3].y, lo[4].y, lo[5].y, ab);
        o.z = lut6_word_imad(lo[0].z, lo[1].z, lo[2].z, lo[3].z, lo[4].z, lo[5].z, ab);
        o.w = lut6_word_imad(lo[0].w, lo[1].w, lo[2].w, lo[3].w, lo[4].w, lo[5].w, ab);
        *reinterpret_cast<uint4 *>(yrow + w) = o;
        if (second) {
            o.x = lut6_word_imad(hi[0].x, hi[1].x, hi[2].x, hi[3].x, hi[4].x, hi[5].x, ab);
            o.y = lut6_word_imad(hi[0].y, hi[1].y, hi[2].y, hi[3].y, hi[4].y, hi[5].y, ab);
            o.z = lut6_word_imad(hi[0].z, hi[1].z, hi[2].z, hi[3].z, hi[4].z, hi[5].z, ab);
            o.w = lut6_word_imad(hi[0].w, hi[1].w, hi[2].w, hi[3].w, hi[4].w, hi[5].w, ab);
            *reinterpret_cast<uint4 *>(yrow + w + 128) = o;
        }
    }
}

// Depth-first multiplexer tree over NW words at once.  A level-1 node costs one 64-bit shared-memory read of its
// (a, b) pair, shared by all NW words; walking depth first keeps about one live value per level and word, so eight
// words fit in registers and the pair reads amortise to four per word instead of thirty-two.
template <int L, int K, int NW>
struct MuxTree {
    static __device__ __forceinline__ void eval(const int2 *ab, const uint32_t (&x)[6][NW], uint32_t (&out)[NW])
    {
        uint32_t lo[NW], hi[NW];
        MuxTree<L - 1, 2 * K, NW>::eval(ab, x, lo);
        MuxTree<L - 1, 2 * K + 1, NW>::eval(ab, x, hi);
#pragma unroll
        for (int w = 0; w < NW; ++w) out[w] = (lo[w] & ~x[L - 1][w]) | (hi[w] & x[L - 1][w]);
    }
};

template <int K, int NW>
struct MuxTree<1, K, NW> {
    static __device__ __forceinline__ void eval(const int2 *ab, const uint32_t (&x)[6][NW], uint32_t (&out)[NW])
    {
        const int2 p = ab[K];
#pragma unroll
        for (int w = 0; w < NW; ++w) out[w] = x[0][w] * (uint32_t)p.x + (uint32_t)p.y;
    }
};

// ---------------------------------------------------------------------------------------------
// Persistent, bulk-copy-pipelined variant (aligned rows; layers of few rounds, or whose rows fill the tiles of k_binary_lut6_imm badly).
// Work item = (word tile of 256 words, node) of one warp; the warps of the grid take the items in order, so that those in
// flight sweep the nodes of one tile together and the tile's rows stay in L2.  (Items of a CTA and eight nodes left warps
// idle where the nodes are no multiple of 8: 36 nodes x 2^20 frames 8.9 -> 8.1 us.)  Each warp runs its own two-stage
// pipeline: its lanes start six 1 KiB bulk copies (one per gathered row) for item j+2 as soon as item j has been read out
// of shared memory into registers, then the warp computes item j while the copies of j+1 and j+2 are in flight.  No warp
// ever waits on a load it has only just issued, and no CTA-wide barrier exists after set-up.
// ---------------------------------------------------------------------------------------------
constexpr int kPipeCtas   = 2;                        // resident CTAs per SM
constexpr int kPipeNW     = 8;                        // words per lane and item
constexpr int kPipeWords  = 32 * kPipeNW;             // words per row segment and item (1 KiB)
constexpr int kPipeStages = 2;
// dynamic shared memory layout: [rows: warp x stage x 6 x 256 words][barriers: warp x stage, padded to 128 B][level-1 pairs: warp x 32 x int2]
constexpr int kPipeRowsBytes = kBlWarps * kPipeStages * 6 * kPipeWords * 4;
constexpr int kPipeBarBytes  = 128;
constexpr int kPipeAbBytes   = kBlWarps * 32 * 8;
constexpr int kPipeSmem      = kPipeRowsBytes + kPipeBarBytes + kPipeAbBytes;
static_assert(kBlWarps * kPipeStages * 8 <= kPipeBarBytes, "barrier block too small");

// Position of a work item, advanced incrementally (item index + gridDim) so that no division runs per item.
struct PipePos {
    int tile, node;
};

__device__ __forceinline__ PipePos pipe_advance(PipePos p, int dt, int dn, int nodes)
{
    p.node += dn;
    p.tile += dt;
    if (p.node >= nodes) { p.node -= nodes; ++p.tile; }
    return p;
}

// Lanes 0..5 each start the bulk copy of one gathered row segment (one instruction issue covers all six); lane 0 has
// armed the barrier with the byte count just before.
// `row` is the lane's input row of the item's node (pipe_row), fetched an item earlier so that the copy does not wait for it.
__device__ __forceinline__ void pipe_issue(const BlArgs &a, PipePos pos, int row, int lane, uint32_t *stage, uint64_t *bar)
{
    const int w0    = pos.tile * kPipeWords;
    const uint32_t bytes = (uint32_t)min(kPipeWords, a.nwords - w0) * 4u;
    if (lane == 0) mbar_arrive_expect_tx(bar, 6u * bytes);
    __syncwarp();
    if (lane < 6) bulk_copy_g2s(stage + lane * kPipeWords, a.x + (size_t)row * a.stride + w0, bytes, bar);
}

__device__ __forceinline__ int pipe_row(const BlArgs &a, int node, int lane)
{
    return lane < 6 ? __ldg(a.idx + (size_t)node * 6 + lane) : 0;
}

__global__ void __launch_bounds__(kBlWarps * 32, kPipeCtas)
k_binary_lut6_pipe(const BlArgs a, int n_tiles, int *fault)
{
    grid_dependency();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint32_t *s_rows = reinterpret_cast<uint32_t *>(smem_raw);                                   // [warp][stage][6][256]
    uint64_t *s_bar  = reinterpret_cast<uint64_t *>(smem_raw + kPipeRowsBytes);                   // [warp][stage]
    int2     *s_ab   = reinterpret_cast<int2 *>(smem_raw + kPipeRowsBytes + kPipeBarBytes);      // [warp][32]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *my_rows = s_rows + (size_t)warp * kPipeStages * 6 * kPipeWords;
    uint64_t *my_bar  = s_bar + warp * kPipeStages;
    int2     *my_ab   = s_ab + warp * 32;

    if (lane == 0) {
        for (int s = 0; s < kPipeStages; ++s) mbar_init(my_bar + s, 1);
        mbar_init_fence();
    }
    __syncwarp();

    // items first, first + all warps, ...: position of the current item and of the next two
    const int step = (int)gridDim.x * kBlWarps, first = (int)blockIdx.x * kBlWarps + warp;
    const int dt = step / a.O, dn = step - dt * a.O;
    PipePos p0;
    p0.tile = first / a.O;
    p0.node = first - p0.tile * a.O;
    PipePos p1 = pipe_advance(p0, dt, dn, a.O);
    PipePos p2 = pipe_advance(p1, dt, dn, a.O);

    if (p0.tile < n_tiles) pipe_issue(a, p0, pipe_row(a, p0.node, lane), lane, my_rows, my_bar);
    if (p1.tile < n_tiles) pipe_issue(a, p1, pipe_row(a, p1.node, lane), lane, my_rows + 6 * kPipeWords, my_bar + 1);
    int row2 = p2.tile < n_tiles ? pipe_row(a, p2.node, lane) : 0;          // input rows of item k+2, one item ahead of their use
    uint32_t tword = 0;
    if (p0.tile < n_tiles) tword = (uint32_t)__ldg(a.table + 2 * (size_t)p0.node + (lane >> 4));

    for (int k = 0; p0.tile < n_tiles; ++k) {
        const int s = k & 1;
        const uint32_t parity = (uint32_t)(k >> 1) & 1u;
        uint32_t *stage = my_rows + s * 6 * kPipeWords;
        const int w0 = p0.tile * kPipeWords;
        const int nw = min(kPipeWords, a.nwords - w0);

        // this node's level-1 (a, b) pairs; the table word of the NEXT item is fetched now and used next round
        {
            const uint32_t lo = (tword >> ((2 * lane) & 31)) & 1u, hi = (tword >> ((2 * lane + 1) & 31)) & 1u;
            __syncwarp();
            my_ab[lane] = make_int2((int)hi - (int)lo, -(int)lo);
            __syncwarp();
        }
        const bool have_next = p1.tile < n_tiles;
        if (have_next) tword = (uint32_t)__ldg(a.table + 2 * (size_t)p1.node + (lane >> 4));

        if (!mbar_wait(my_bar + s, parity)) {          // bounded: record the fault, let the other stage's copies land, leave
            if (lane == 0) atomicCAS(fault, 0, kFaultBarrierTimeout);
            if (have_next) mbar_wait(my_bar + (s ^ 1), (uint32_t)((k + 1) >> 1) & 1u);
            return;
        }
        const int w = 4 * lane;
        uint32_t xw[6][kPipeNW], o[kPipeNW];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
#pragma unroll
            for (int h = 0; h < kPipeNW / 4; ++h) {
                const uint4 v = *reinterpret_cast<const uint4 *>(stage + j * kPipeWords + w + 128 * h);
                xw[j][4 * h] = v.x; xw[j][4 * h + 1] = v.y; xw[j][4 * h + 2] = v.z; xw[j][4 * h + 3] = v.w;
            }
        }
        __syncwarp();                                   // every lane has read the stage out
        if (p2.tile < n_tiles) {
            proxy_fence_async();                        // reads above (generic proxy) before the refill (async proxy)
            pipe_issue(a, p2, row2, lane, stage, my_bar + s);
        }
        const PipePos p3 = pipe_advance(p2, dt, dn, a.O);
        if (p3.tile < n_tiles) row2 = pipe_row(a, p3.node, lane);
        MuxTree<6, 0, kPipeNW>::eval(my_ab, xw, o);
        uint32_t *yrow = a.y + (size_t)p0.node * a.stride + w0;
#pragma unroll
        for (int h = 0; h < kPipeNW / 4; ++h)
            if (w + 128 * h < nw) *reinterpret_cast<uint4 *>(yrow + w + 128 * h) = make_uint4(o[4 * h], o[4 * h + 1], o[4 * h + 2], o[4 * h + 3]);

        p0 = p1; p1 = p2; p2 = p3;
    }
}

// ---------------------------------------------------------------------------------------------
// One word of one node per thread: the smallest calls, where the pipeline's set-up and its eight words a lane are most of the time.
// Bound by latency: wiring, then the six words, then the tree with the table's bits spread to masks on the way (about 200 operations).
// ---------------------------------------------------------------------------------------------
template <int L, int K>
struct WordTree {
    static __device__ __forceinline__ uint32_t eval(uint32_t t0, uint32_t t1, const uint32_t (&x)[6])
    {
        const uint32_t lo = WordTree<L - 1, 2 * K>::eval(t0, t1, x), hi = WordTree<L - 1, 2 * K + 1>::eval(t0, t1, x);
        return (lo & ~x[L - 1]) | (hi & x[L - 1]);
    }
};

template <int K>
struct WordTree<0, K> {              // table bit K in all 32 positions
    static __device__ __forceinline__ uint32_t eval(uint32_t t0, uint32_t t1, const uint32_t (&)[6])
    {
        return (uint32_t)((int)((K < 32 ? t0 : t1) << (31 - (K & 31))) >> 31);
    }
};

constexpr int kWordThreads = 128;

__global__ void __launch_bounds__(kWordThreads)
k_binary_lut6_words(const BlArgs a)
{
    grid_dependency();
    const unsigned t = blockIdx.x * kWordThreads + threadIdx.x, words = (unsigned)a.nwords;
    const unsigned node = t / words, w = t - node * words;
    if (node >= (unsigned)a.O) return;
    const uint32_t t0 = (uint32_t)__ldg(a.table + 2 * (size_t)node), t1 = (uint32_t)__ldg(a.table + 2 * (size_t)node + 1);
    uint32_t x[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) x[j] = __ldg(a.x + (size_t)__ldg(a.idx + (size_t)node * 6 + j) * a.stride + w);
    a.y[(size_t)node * a.stride + w] = WordTree<6, 0>::eval(t0, t1, x);
}

// ---------------------------------------------------------------------------------------------
// Truth-table-immediate variant (aligned rows).
// lop3.b32 evaluates ANY three-input boolean function in one instruction, the function being an 8-bit immediate.  Byte b of a
// node's 64-bit table is exactly the function of (x0, x1, x2) that applies where x3 + 2 x4 + 4 x5 = b, so a word costs eight lop3
// with the table bytes as immediates and seven selects on x3, x4, x5: 15 logic operations instead of 63.  The immediates are
// instruction text, so each table byte is dispatched through an indexed branch (brx.idx) into 256 case bodies that hold the
// lop3 for all eight words of a lane; they return to one tail, which goes by the byte's position and folds the partial results as
// a binary counter does.  The byte is warp-uniform (one node per warp): the branches never diverge.  (Returning by a second indexed branch
// took 16 % longer.)
// What bounds it is the fetch of case bodies that are cold, and that is shared: four warps of a CTA -- one on every scheduler -- take
// neighbouring segments of the same node at the same time.  Registers only, clocks per word and scheduler, 28 warps per SM: every warp
// its own node 169, two sharing one 112, four 65, seven (all of a scheduler) 56, all 28 46, and four with two segments each 57; the
// multiplexer tree of k_binary_lut6_pipe takes 106 whatever is shared.
// The bodies write one set of registers, which costs four moves a word: with a second set of bodies for the odd bytes, 80 KiB of code in all,
// fetching them bounds the kernel again (1000 nodes x 2^20 frames 130 us instead of 92).  16384 x 2^20: 1951 -> 1483 us at the full clock, 5000 x 2^20
// 609 -> 414, 216 x 2^20 30.3 -> 22.7.  Under ncu (16384 nodes x 131072 frames, caches cold) 204 us against 272 of the tree: 46 instructions and 104
// clocks per word and scheduler, 45 % of the issue slots, no unit above 54 %: latency at 20 warps per SM, of shared memory and copies, of the branches
// and of the fetches (24 warps do not leave it the registers: 110 us instead of 92).
// %0-%7 x0 and the result, %8-%15 x1, %16-%23 x2, %24 / %25 the table words, %26 the lane's first piece of x3 in shared memory; x3, x4 and x5 are
// read there when they are needed (24 registers fewer).
// ---------------------------------------------------------------------------------------------
constexpr int kImmGroup  = 4;                          // warps that share a node
constexpr int kImmWarps  = 20;
constexpr int kImmTile   = kImmGroup * kPipeWords;     // words of a work item, 256 for each warp of the group
// dynamic shared memory, per warp: [x0..x2: 3 x 256 words][x3..x5: 2 x 3 x 256 words]
constexpr int kImmHalf   = 3 * kPipeWords;
constexpr int kImmSmem   = kImmWarps * 3 * kImmHalf * 4;
static_assert(kPipeWords == 256 && kImmSmem <= 227 * 1024, "the row distance is in the code below; one CTA per SM");

#define BB200_LOPS(imm) \
    "lop3.b32 p0, %16, %8, %0, " imm ";\n\tlop3.b32 p1, %17, %9, %1, " imm ";\n\tlop3.b32 p2, %18, %10, %2, " imm ";\n\tlop3.b32 p3, %19, %11, %3, " imm ";\n\t" \
    "lop3.b32 p4, %20, %12, %4, " imm ";\n\tlop3.b32 p5, %21, %13, %5, " imm ";\n\tlop3.b32 p6, %22, %14, %6, " imm ";\n\tlop3.b32 p7, %23, %15, %7, " imm ";\n\t"
#define BB200_CASE(h, l) "T" #h #l ":\n\t" BB200_LOPS("0x" #h #l) "bra.uni TAIL;\n\t"
#define BB200_ROW(h)                                                                                                                        \
    BB200_CASE(h, 0) BB200_CASE(h, 1) BB200_CASE(h, 2) BB200_CASE(h, 3) BB200_CASE(h, 4) BB200_CASE(h, 5) BB200_CASE(h, 6) BB200_CASE(h, 7) \
    BB200_CASE(h, 8) BB200_CASE(h, 9) BB200_CASE(h, A) BB200_CASE(h, B) BB200_CASE(h, C) BB200_CASE(h, D) BB200_CASE(h, E) BB200_CASE(h, F)
#define BB200_TGT(h)                                                                                                                        \
    "T" #h "0, T" #h "1, T" #h "2, T" #h "3, T" #h "4, T" #h "5, T" #h "6, T" #h "7, T" #h "8, T" #h "9, T" #h "A, T" #h "B, T" #h "C, T" #h "D, T" #h "E, T" #h "F"
// on to the case of the lowest byte of tw
#define BB200_DISPATCH "and.b32 byte, tw, 255;\n\tshr.u32 tw, tw, 8;\n\tbrx.idx byte, TBL;\n\t"
#define BB200_KEEP "mov.u32 a0, p0;\n\tmov.u32 a1, p1;\n\tmov.u32 a2, p2;\n\tmov.u32 a3, p3;\n\tmov.u32 a4, p4;\n\tmov.u32 a5, p5;\n\tmov.u32 a6, p6;\n\tmov.u32 a7, p7;\n\t"
// a row of the lane's words: u = row at `at` (second half at `at2`); d = u ? hi : lo
#define BB200_LOAD(at, at2) "ld.shared.v4.u32 {u0, u1, u2, u3}, [%26+" at "];\n\tld.shared.v4.u32 {u4, u5, u6, u7}, [%26+" at2 "];\n\t"
#define BB200_LOAD3 BB200_LOAD("0", "512")
#define BB200_LOAD4 BB200_LOAD("1024", "1536")
#define BB200_LOAD5 BB200_LOAD("2048", "2560")
#define BB200_SELECT(d, hi, lo)                                                                                                              \
    "lop3.b32 " d "0, u0, " hi "0, " lo "0, 0xCA;\n\tlop3.b32 " d "1, u1, " hi "1, " lo "1, 0xCA;\n\tlop3.b32 " d "2, u2, " hi "2, " lo "2, 0xCA;\n\t" \
    "lop3.b32 " d "3, u3, " hi "3, " lo "3, 0xCA;\n\tlop3.b32 " d "4, u4, " hi "4, " lo "4, 0xCA;\n\tlop3.b32 " d "5, u5, " hi "5, " lo "5, 0xCA;\n\t" \
    "lop3.b32 " d "6, u6, " hi "6, " lo "6, 0xCA;\n\tlop3.b32 " d "7, u7, " hi "7, " lo "7, 0xCA;\n\t"

// x[0][w] = table[x0[w] + 2 x1[w] + 4 x2[w] + 8 x3[w] + 16 x4[w] + 32 x5[w]] bitwise, for the 8 words of a lane
__device__ __forceinline__ void lut6_words_by_immediates(uint32_t (&x)[3][8], uint32_t table_lo, uint32_t table_hi, uint32_t upper)
{
    asm volatile(
        "{\n\t"
        ".reg .u32 p<8>, a<8>, b<8>, c<8>, u<8>;\n\t"
        ".reg .u32 byte, tw, i, t;\n\t"
        ".reg .pred q;\n\t"
        "TBL: .branchtargets " BB200_TGT(0) ", " BB200_TGT(1) ", " BB200_TGT(2) ", " BB200_TGT(3) ", " BB200_TGT(4) ", " BB200_TGT(5) ", "
        BB200_TGT(6) ", " BB200_TGT(7) ", " BB200_TGT(8) ", " BB200_TGT(9) ", " BB200_TGT(A) ", " BB200_TGT(B) ", " BB200_TGT(C) ", "
        BB200_TGT(D) ", " BB200_TGT(E) ", " BB200_TGT(F) ";\n\t"
        "mov.u32 i, 0;\n\t"
        "mov.u32 tw, %24;\n\t"
        BB200_DISPATCH
        BB200_ROW(0) BB200_ROW(1) BB200_ROW(2) BB200_ROW(3) BB200_ROW(4) BB200_ROW(5) BB200_ROW(6) BB200_ROW(7)
        BB200_ROW(8) BB200_ROW(9) BB200_ROW(A) BB200_ROW(B) BB200_ROW(C) BB200_ROW(D) BB200_ROW(E) BB200_ROW(F)
        "TAIL:\n\t"
        "and.b32 t, i, 1;\n\t"
        "setp.ne.u32 q, t, 0;\n\t"
        "@q bra.uni ODD;\n\t"
        BB200_KEEP
        BB200_LOAD3
        "add.u32 i, i, 1;\n\t"
        BB200_DISPATCH
        "ODD:\n\t"
        "and.b32 t, i, 2;\n\t"
        "setp.ne.u32 q, t, 0;\n\t"
        "@q bra.uni PAIR;\n\t"
        BB200_SELECT("b", "p", "a")
        "add.u32 i, i, 1;\n\t"
        BB200_DISPATCH
        "PAIR:\n\t"
        BB200_SELECT("p", "p", "a")
        BB200_LOAD4
        "setp.eq.u32 q, i, 7;\n\t"
        "@q bra.uni LAST;\n\t"
        BB200_SELECT("c", "p", "b")
        "mov.u32 tw, %25;\n\t"
        "mov.u32 i, 4;\n\t"
        BB200_DISPATCH
        "LAST:\n\t"
        BB200_SELECT("p", "p", "b")
        BB200_LOAD5
        BB200_SELECT("%", "p", "c")
        "}"
        : "+r"(x[0][0]), "+r"(x[0][1]), "+r"(x[0][2]), "+r"(x[0][3]), "+r"(x[0][4]), "+r"(x[0][5]), "+r"(x[0][6]), "+r"(x[0][7])
        : "r"(x[1][0]), "r"(x[1][1]), "r"(x[1][2]), "r"(x[1][3]), "r"(x[1][4]), "r"(x[1][5]), "r"(x[1][6]), "r"(x[1][7]),
          "r"(x[2][0]), "r"(x[2][1]), "r"(x[2][2]), "r"(x[2][3]), "r"(x[2][4]), "r"(x[2][5]), "r"(x[2][6]), "r"(x[2][7]),
          "r"(table_lo), "r"(table_hi), "r"(upper)
        : "memory");
}
#undef BB200_LOPS
#undef BB200_CASE
#undef BB200_ROW
#undef BB200_TGT
#undef BB200_DISPATCH
#undef BB200_KEEP
#undef BB200_SELECT
#undef BB200_LOAD
#undef BB200_LOAD3
#undef BB200_LOAD4
#undef BB200_LOAD5

// Whether a node's run is two tiles by the input rows, whose number is not among the operator's arguments: it is the range of the wiring's entries, of
// which every warp reads the same 64 while the rows of its first item are on their way (256 of them, before anything else, made 1000 nodes x 300000 frames
// 30.2 -> 30.6 us, and asking every call 216 x 262144, which is too short for two tiles, 9.0 -> 9.2; now 30.5 in a run where not asking takes 30.5,
// and 8.8).  Rows of two tiles that do not stay in L2 come from HBM once more for every
// reader.  Two to three rows a node are for two tiles where they do stay; up to two are either way within 5 %, sustained for two, cool for one; and
// beyond three few rows have a second reader.  In us by k_binary_lut6_pipe / with one tile / with two, cool: 8192 nodes x 2^20 frames reading 8192 rows
// 982 / 733 / 671, 16384 rows 984 / 759 / 791, 24576 983 / 775 / 944, 49152 1008 / 883 / 1126; 4000 x 2^20 reading 8000 rows 530 / 365 / 335, 12000
// 501 / 371 / 359, 24000 497 / 412 / 486; 2000 x 2^21 reading 12000 497 / 401 / 430; 13000 x 2^18 reading 3900 423 / 322 / 282, 39000 412 / 327 / 401.
__device__ __forceinline__ bool imm_two_tiles(const BlArgs &a, int run_rows, int lane)
{
    constexpr int kLook = 2;
    const long long entries = 6LL * a.O;
    unsigned lo = ~0u, hi = 0u;
#pragma unroll
    for (int k = 0; k < kLook; ++k) {
        const unsigned row = (unsigned)__ldg(a.idx + (entries * (32 * k + lane)) / (32 * kLook));
        lo = min(lo, row);
        hi = max(hi, row);
    }
    const long long rows = (long long)__reduce_max_sync(0xffffffffu, hi) - __reduce_min_sync(0xffffffffu, lo);
    return rows <= 2LL * a.O || (rows <= run_rows && rows <= 3LL * a.O);
}

// Persistent: a group of four warps takes (tile of 1024 words, node) items in tile-major order, each warp a segment of 256 words.  x0..x2 go to
// registers at the start of an item, and the copies of the next item's follow at once; x3..x5 are used from shared memory, in two buffers.
// Every lane copies, with cp.async, the 16-byte pieces that it will itself read: no barrier and no cross-lane dependence.
// TWO: a node's run may be two tiles, up to run_rows input rows (of which two tiles stay in L2).
template <bool TWO>
__global__ void __launch_bounds__(kImmWarps * 32, 1)
k_binary_lut6_imm(const BlArgs a, int run_rows)
{
    grid_dependency();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kGroups = kImmWarps / kImmGroup;
    const int segment = (warp % kImmGroup) * kPipeWords;
    const uint32_t lower = smem_addr(smem_raw) + (uint32_t)warp * 3 * kImmHalf * 4 + 16 * lane, upper = lower + kImmHalf * 4;
    const int tiles = a.nwords > segment ? (a.nwords - segment - 1) / kImmTile + 1 : 0;      // tiles that have words for this warp, and
    const int whole = (a.nwords + kImmTile - kPipeWords - segment) / kImmTile;               // those in which it has all 256
    const int step = (int)gridDim.x * kGroups, first = (int)blockIdx.x * kGroups + warp / kImmGroup;
    // A node's run is one or two tiles; the runs of a group are `first`, first + step, ...
    PipePos p0;
    p0.tile = first / a.O;
    p0.node = first - p0.tile * a.O;
    const int row0 = pipe_row(a, p0.node, lane);          // on its way while the wiring is looked at; a node's run does not move it
    const int run = TWO && imm_two_tiles(a, run_rows, lane) ? 2 : 1;
    const int dt = step / a.O, dn = step - dt * a.O, last = run - 1;
    auto advance = [&](PipePos p) {
        if ((p.tile & last) != last && p.tile + 1 < tiles) {
            ++p.tile;
            return p;
        }
        p.tile = (p.tile & ~last) + dt * run;
        p.node += dn;
        if (p.node >= a.O) { p.node -= a.O; p.tile += run; }
        return p;
    };
    p0.tile *= run;
    // three rows, from input `J` on, of item p to `dst`; lane j of `row` holds the item's input row j
    const uint32_t row_bytes = (uint32_t)a.stride * 4u;
    const uint64_t mine = (uint64_t)__cvta_generic_to_global(a.x) + (uint64_t)(segment + 4 * lane) * 4;
    auto issue = [&](const PipePos &p, int row, auto j_tag, uint32_t dst) {
        constexpr int J = decltype(j_tag)::value;
        if (p.tile < tiles) {
            const uint64_t base = mine + (uint64_t)(uint32_t)p.tile * (kImmTile * 4);
            const uint64_t s0 = base + (uint64_t)(uint32_t)__shfl_sync(0xffffffffu, row, J) * row_bytes,
                           s1 = base + (uint64_t)(uint32_t)__shfl_sync(0xffffffffu, row, J + 1) * row_bytes,
                           s2 = base + (uint64_t)(uint32_t)__shfl_sync(0xffffffffu, row, J + 2) * row_bytes;
            if (p.tile < whole) {
                cp_async16_at<0, 0>(dst, s0); cp_async16_at<512, 512>(dst, s0);
                cp_async16_at<1024, 0>(dst, s1); cp_async16_at<1536, 512>(dst, s1);
                cp_async16_at<2048, 0>(dst, s2); cp_async16_at<2560, 512>(dst, s2);
            } else {
                const int w0 = p.tile * kImmTile + segment + 4 * lane;
                if (w0 < a.nwords) { cp_async16_at<0, 0>(dst, s0); cp_async16_at<1024, 0>(dst, s1); cp_async16_at<2048, 0>(dst, s2); }
                if (w0 + 128 < a.nwords) { cp_async16_at<512, 512>(dst, s0); cp_async16_at<1536, 512>(dst, s1); cp_async16_at<2560, 512>(dst, s2); }
            }
        }
        cp_async_commit();
    };
    using Lo = std::integral_constant<int, 0>;
    using Hi = std::integral_constant<int, 3>;
    PipePos p1 = advance(p0);
    int row1 = 0, row2 = 0;                              // input rows of items k + 1 and k + 2 (lanes 0..5)
    uint2 table = make_uint2(0u, 0u);
    {
        if (p1.tile < tiles) row1 = pipe_row(a, p1.node, lane);
        issue(p0, row0, Hi{}, upper);
        issue(p0, row0, Lo{}, lower);
        issue(p1, row1, Hi{}, upper + kImmHalf * 4);
    }
    if (p0.tile < tiles) table = make_uint2((uint32_t)__ldg(a.table + 2 * (size_t)p0.node), (uint32_t)__ldg(a.table + 2 * (size_t)p0.node + 1));
    PipePos p2 = advance(p1);
    if (p2.tile < tiles) row2 = pipe_row(a, p2.node, lane);
    uint32_t buf = upper;
    while (p0.tile < tiles) {
        cp_async_wait<1>();                              // all but the newest copies, which are item k + 1's x3..x5
        uint32_t x[3][8];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x[j][4 * h]), "=r"(x[j][4 * h + 1]), "=r"(x[j][4 * h + 2]), "=r"(x[j][4 * h + 3])
                             : "r"(lower + 1024 * j + 512 * h) : "memory");
        }
        issue(p1, row1, Lo{}, lower);
        const uint2 tab = table;
        if (p1.tile < tiles) table = make_uint2((uint32_t)__ldg(a.table + 2 * (size_t)p1.node), (uint32_t)__ldg(a.table + 2 * (size_t)p1.node + 1));
        lut6_words_by_immediates(x, tab.x, tab.y, buf);
        issue(p2, row2, Hi{}, buf);
        buf = buf == upper ? upper + kImmHalf * 4 : upper;
        const int w = p0.tile * kImmTile + segment + 4 * lane;
        uint32_t *yrow = a.y + (size_t)p0.node * a.stride + w;
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (w + 128 * h < a.nwords) *reinterpret_cast<uint4 *>(yrow + 128 * h) = make_uint4(x[0][4 * h], x[0][4 * h + 1], x[0][4 * h + 2], x[0][4 * h + 3]);
        p0 = p1; p1 = p2; row1 = row2;
        p2 = advance(p2);
        if (p2.tile < tiles) row2 = pipe_row(a, p2.node, lane);
    }
    cp_async_wait<0>();
}

// Rounds of the persistent grid that the call takes (a round: every group of every SM one tile of a node).
long long imm_rounds(const BlArgs &a)
{
    const long long groups = (long long)(kImmWarps / kImmGroup) * device_info().sm_count;
    return ((a.nwords + kImmTile - 1) / kImmTile * (long long)a.O + groups - 1) / groups;
}

// Most tiles that a group takes of a node before the next node.  Two halve the case bodies to fetch, but the rows of both, 8 KiB an input, have to stay
// in L2 (of the inputs only the wiring tells: imm_two_tiles()), and they make the rounds coarser: 8192 nodes x 2^20 frames 982 us by
// k_binary_lut6_pipe, 727 with one tile, 668 with two, 796 with four; 20000 x 2^18 606, 467, 479, 618; 318 x 56770 (one round) 4.5, 4.6, 5.9, 5.9.
int imm_run_rows() { return (int)((long long)(device_info().l2_bytes / 10 * 9) / (2LL * kImmTile * 4)); }
int imm_run(const BlArgs &a) { return imm_rounds(a) >= 8 && a.O <= imm_run_rows() ? 2 : 1; }

// What the kernel's 32-bit arithmetic can take.
bool imm_fits(const BlArgs &a)
{
    return a.stride < (1 << 30) && ((long long)a.nwords / kImmTile + 2) * a.O < (1LL << 31) - 65536 && allow_big_smem(k_binary_lut6_imm<true>, kImmSmem) &&
           allow_big_smem(k_binary_lut6_imm<false>, kImmSmem);
}

int launch_immediate(BlArgs a, cudaStream_t st)
{
    a.Tw = imm_run(a);
    const long long tiles = (a.nwords + kImmTile - 1) / kImmTile, runs = (tiles + a.Tw - 1) / a.Tw * a.O, groups = kImmWarps / kImmGroup;
    const long long grid = (runs + groups - 1) / groups;
    launch(a.Tw == 2 ? k_binary_lut6_imm<true> : k_binary_lut6_imm<false>, (unsigned)(grid < device_info().sm_count ? grid : device_info().sm_count),
           kImmWarps * 32, kImmSmem, st, a, imm_run_rows());
    return launch_status();
}

}   // namespace bb200

using namespace bb200;

extern "C" int bbcu_bit_BinaryLut6_Forward(const int *x, int *y, const int *idx, const int *table, int node_size, int frame_size,
                                           int frame_stride, bbcu_stream_t stream)
{
    BB200_REQUIRE_PTR(x); BB200_REQUIRE_PTR(y); BB200_REQUIRE_PTR(idx); BB200_REQUIRE_PTR(table);
    BB200_REQUIRE(node_size >= 0 && frame_size >= 0, BBCU_ERR_BAD_SIZE);
    BB200_REQUIRE((long long)frame_stride * 32 >= frame_size, BBCU_ERR_BAD_STRIDE);
    if (node_size == 0 || frame_size == 0) return BBCU_OK;

    BlArgs a;
    a.x = reinterpret_cast<const uint32_t *>(x); a.y = reinterpret_cast<uint32_t *>(y); a.idx = idx; a.table = table;
    a.O = node_size; a.stride = frame_stride;
    a.nwords = (frame_size + 31) / 32;
    a.groups = (node_size + kBlWarps - 1) / kBlWarps;
    // 128-bit path: rows start 16-byte aligned and whole uint4 groups fit inside the row stride
    const bool vec = (frame_stride % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0) && ((reinterpret_cast<uintptr_t>(y) & 15) == 0);
    if (vec) a.nwords = (a.nwords + 3) & ~3;
    a.Tw = 0;
    // A word per thread while that is at most a quarter of what the pipeline's rounds of warps could take in 256-word tiles: a round costs
    // the same whether its tiles are full or not (1024 nodes x 200 frames 3.4 -> 2.0 us, 1024 x 4096 3.4 -> 2.9, 4096 x 2048 7.0 -> 4.4,
    // 10000 x 2048 13.2 -> 8.5; at 512 x 10000 both take 3.5, and 384 x 65536 is 10.1 against 6.0).
    const long long node_words = (long long)node_size * a.nwords, warps = (long long)kPipeCtas * kBlWarps * device_info().sm_count;
    const long long rounds = ((long long)node_size * ((a.nwords + kPipeWords - 1) / kPipeWords) + warps - 1) / warps;
    if (node_words <= 1024LL * device_info().sm_count * rounds && node_words < (1LL << 31) - kWordThreads) {
        launch(k_binary_lut6_words, (unsigned)((node_words + kWordThreads - 1) / kWordThreads), kWordThreads, 0, as_stream(stream), a);
        return launch_status();
    }
    // The table bytes as immediates where the rounds of its grid (four warps and 1024 words each) are hardly more than those of the pipeline (a warp and
    // 256 words), which take a little longer: at 1.05 times as many both sides are even (22916 nodes x 71132 frames 202 / 200 us, 4164 x 32966, at
    // 1.33, 23.9 / 26.5); below three rounds neither wins, and its cold case bodies cost up to 0.5 us.
    if (vec) {
        const long long rounds_pipe = ((long long)((a.nwords + kPipeWords - 1) / kPipeWords) * node_size + warps - 1) / warps;
        if (rounds_pipe >= 3 && 20 * imm_rounds(a) <= 21 * rounds_pipe && imm_fits(a)) return launch_immediate(a, as_stream(stream));
    }
    if (vec) {
        // persistent pipeline: two CTAs per SM, each warp of which walks (tile, node) items
        const bool attr_ok = allow_big_smem(k_binary_lut6_pipe, kPipeSmem);
        int *fault = fault_word();
        if (attr_ok && fault != nullptr) {
            const long long n_items = (long long)((a.nwords + kPipeWords - 1) / kPipeWords) * a.groups;
            BB200_REQUIRE(n_items < (1LL << 31) - 4096, BBCU_ERR_TOO_LARGE);      // 32-bit item arithmetic in the kernel
            long long grid = (long long)kPipeCtas * device_info().sm_count;
            if (grid > n_items) grid = n_items;
            launch(k_binary_lut6_pipe, (unsigned)grid, kBlWarps * 32, kPipeSmem, as_stream(stream), a, (a.nwords + kPipeWords - 1) / kPipeWords, fault);
            return launch_status();
        }
    }
    // word tile: frame_tile() counts in frames; a word is 32 of them
    const int tf = frame_tile(2LL * node_size, 1, a.groups, a.nwords * 32, 1024 * 32);
    a.Tw = ((tf / 32 + 127) / 128) * 128;
    const long long blocks = (long long)((a.nwords + a.Tw - 1) / a.Tw) * a.groups;
    BB200_REQUIRE(blocks < (1LL << 31), BBCU_ERR_TOO_LARGE);
    // aligned rows without the shared-memory opt-in (or without a fault word): the non-pipelined 128-bit kernel; otherwise word loads
    if (vec) launch(k_binary_lut6_2pipe, (unsigned)blocks, kBlWarps * 32, 0, as_stream(stream), a);
    else     launch(k_binary_lut6, (unsigned)blocks, kBlWarps * 32, 0, as_stream(stream), a);
    return launch_status();
}

// The same operator through the truth-table-immediate kernel wherever its 32-bit arithmetic reaches, through the kernels above beyond.  Rows must be
// 16-byte aligned (stride a multiple of 4 words, aligned base pointers).
extern "C" int bbcu_bit_BinaryLut6_Forward_Lop3Immediate(const int *x, int *y, const int *idx, const int *table, int node_size, int frame_size,
                                                         int frame_stride, bbcu_stream_t stream)
{
    BB200_REQUIRE_PTR(x); BB200_REQUIRE_PTR(y); BB200_REQUIRE_PTR(idx); BB200_REQUIRE_PTR(table);
    BB200_REQUIRE(node_size >= 0 && frame_size >= 0, BBCU_ERR_BAD_SIZE);
    BB200_REQUIRE((long long)frame_stride * 32 >= frame_size, BBCU_ERR_BAD_STRIDE);
    BB200_REQUIRE(frame_stride % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(table) & 7) == 0, BBCU_ERR_BAD_STRIDE);
    if (node_size == 0 || frame_size == 0) return BBCU_OK;
    BlArgs a;
    a.x = reinterpret_cast<const uint32_t *>(x); a.y = reinterpret_cast<uint32_t *>(y); a.idx = idx; a.table = table;
    a.O = node_size; a.stride = frame_stride;
    a.nwords = ((frame_size + 31) / 32 + 3) & ~3;
    a.groups = 0;
    a.Tw = 0;
    if (!imm_fits(a)) return bbcu_bit_BinaryLut6_Forward(x, y, idx, table, node_size, frame_size, frame_stride, stream);
    return launch_immediate(a, as_stream(stream));
}

extern "C" int bbcu_bit_BinatyLut6_Forward(const int *x, int *y, const int *idx, const int *table, int node_size, int frame_size,
                                           int frame_stride, bbcu_stream_t stream)
{
    return bbcu_bit_BinaryLut6_Forward(x, y, idx, table, node_size, frame_size, frame_stride, stream);
}
