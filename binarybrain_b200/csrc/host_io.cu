// BinaryLut6 forward on HOST frame buffers: the call a host-resident caller makes (x and y live in host memory, as
// BinaryBrain's FrameBuffer does before its first device lock, include/bb/Memory.h:524-662).  The frame axis is cut
// into chunks; a few stream-ordered slots each run  H2D copy -> kernel -> D2H copy  on their own stream, so the upload of
// a later chunk, the kernel of the next and the download of an earlier one overlap and the PCIe link is busy in both
// directions at once.  With pinned host memory the whole call costs about max(upload, download) instead of
// their sum plus the kernel.  Device chunk buffers come from the device heap and are cached between calls.
//
// What bounds it is the link: 55-57 GB/s one way, 45-49 GB/s each way when both run (2-D copies with rows of 1 KiB and more
// are within 10 % of that), plus the part that cannot overlap: the first upload and the last kernel and download.  Hence
// small chunks (chunk_words()).  5000 -> 5000 nodes x 100003 frames, 62.5 MB each way: 2.39 ms as one 4096-word chunk, 1.77 ms with
// 256-word chunks at the ends and 512 words between them; 1.97 at 128, 1.83 at 1024 words; 16384 nodes x 2^18 frames 15.7 -> 13.1 ms;
// 2000 x 20000 400 -> 250 us.  Three, four, six or eight slots are within 2 % of one another.
#include <mutex>

#include "common.cuh"

namespace {

constexpr int kSlots = 4;

// Words per row of the chunk that starts at word w0: `lo` at either end of the job (the first upload and the last download run
// alone), `mid` in between.  A chunk costs about 15 us of enqueueing, so it holds at least 1 MiB of the wider of x and y; rows
// shorter than 1 KiB slow the 2-D copies down, so the edge chunks have 256 words per row unless the job has fewer than three of those.
constexpr int kEdgeWords = 256;

int chunk_words(int w0, int words, int lo, int mid)
{
    const int left = words - w0;
    const int n = w0 == 0 || left < mid + lo ? lo : mid;
    return n < left ? n : left;
}

struct HostIo {
    cudaStream_t stream[kSlots] = {};
    void *x[kSlots] = {}, *y[kSlots] = {};
    size_t x_bytes = 0, y_bytes = 0;
    void *idx = nullptr, *table = nullptr;
    cudaEvent_t tables_up = nullptr;       // wiring and tables of the current call are on the device
    size_t idx_bytes = 0, table_bytes = 0;
    bool ready = false;
};

std::mutex g_mu;
HostIo g_io[64];

int ensure(HostIo &io, size_t xb, size_t yb, size_t ib, size_t tb)
{
    if (!io.ready) {
        for (int s = 0; s < kSlots; ++s) BB200_CUDA(cudaStreamCreateWithFlags(&io.stream[s], cudaStreamNonBlocking));
        BB200_CUDA(cudaEventCreateWithFlags(&io.tables_up, cudaEventDisableTiming));
        io.ready = true;
    }
    auto grow = [](void *&p, size_t &have, size_t want) -> int {
        if (have >= want) return 0;
        if (p) bbcu_LocalHeap_Free(p);
        p = bbcu_LocalHeap_Malloc(want);
        have = p ? want : 0;
        return p ? 0 : BBCU_ERR_NO_MEMORY;
    };
    if (io.x_bytes < xb) {
        for (int s = 0; s < kSlots; ++s) { size_t h = io.x_bytes; int rc = grow(io.x[s], h, xb); if (rc) return rc; }
        io.x_bytes = xb;
    }
    if (io.y_bytes < yb) {
        for (int s = 0; s < kSlots; ++s) { size_t h = io.y_bytes; int rc = grow(io.y[s], h, yb); if (rc) return rc; }
        io.y_bytes = yb;
    }
    int rc = grow(io.idx, io.idx_bytes, ib);
    if (rc) return rc;
    return grow(io.table, io.table_bytes, tb);
}

}   // namespace

extern "C" int bbcu_host_bit_BinaryLut6_Forward(const int *host_x_buf, int *host_y_buf, const int *host_input_index, const int *host_table,
                                                int input_node_size, int node_size, int frame_size, int frame_stride)
{
    BB200_REQUIRE_PTR(host_x_buf); BB200_REQUIRE_PTR(host_y_buf); BB200_REQUIRE_PTR(host_input_index); BB200_REQUIRE_PTR(host_table);
    BB200_REQUIRE(input_node_size > 0 && node_size >= 0 && frame_size >= 0, BBCU_ERR_BAD_SIZE);
    BB200_REQUIRE((long long)frame_stride * 32 >= frame_size, BBCU_ERR_BAD_STRIDE);
    if (node_size == 0 || frame_size == 0) return BBCU_OK;
    const int dev = bbcu_GetDevice();
    BB200_REQUIRE(dev >= 0 && dev < 64, BBCU_ERR_NO_DEVICE);

    std::lock_guard<std::mutex> lock(g_mu);          // one host-buffer call per process at a time: the slots are shared
    HostIo &io = g_io[dev];
    const int words = (frame_size + 31) / 32;
    const int wider = input_node_size > node_size ? input_node_size : node_size;
    int lo = ((words + 2) / 3 + 63) & ~63;
    if (lo > kEdgeWords) lo = kEdgeWords;
    const int mib = ((1 << 18) / wider + 63) & ~63;                          // words per row of a 1 MiB chunk
    if (lo < mib) lo = mib;
    const int mid = 2 * lo;
    const int widest = words < mid ? (words + 7) & ~7 : mid;                 // device row stride of the widest chunk (32-byte rows)
    int rc = ensure(io, sizeof(int) * (size_t)input_node_size * widest, sizeof(int) * (size_t)node_size * widest,
                    sizeof(int) * 6 * (size_t)node_size, sizeof(int) * 2 * (size_t)node_size);
    if (rc) return rc;

    // On any error the copies already enqueued into the caller's host_y_buf are drained before the status goes back: the caller
    // may free or reuse its buffers as soon as this function returns.
    auto drain = [&](int status) {
        for (int s = 0; s < kSlots; ++s)
            if (cudaStreamSynchronize(io.stream[s]) != cudaSuccess) cudaGetLastError();
        return status;
    };
    for (int k = 0, w0 = 0; w0 < words; ++k) {
        const int s = k % kSlots;
        cudaStream_t st = io.stream[s];
        const int nw = chunk_words(w0, words, lo, mid);
        const int cw = (nw + 7) & ~7;
        const int frames_k = w0 + nw == words ? frame_size - w0 * 32 : nw * 32;
        cudaError_t e = cudaMemcpy2DAsync(io.x[s], sizeof(int) * (size_t)cw, host_x_buf + w0, sizeof(int) * (size_t)frame_stride, sizeof(int) * (size_t)nw,
                                          (size_t)input_node_size, cudaMemcpyHostToDevice, st);
        // wiring and tables follow the first chunk on its stream; the other streams' kernels wait for them
        if (k == 0) {
            if (e == cudaSuccess) e = cudaMemcpyAsync(io.idx, host_input_index, sizeof(int) * 6 * (size_t)node_size, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaMemcpyAsync(io.table, host_table, sizeof(int) * 2 * (size_t)node_size, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(io.tables_up, st);
        } else if (k < kSlots && e == cudaSuccess) {
            e = cudaStreamWaitEvent(st, io.tables_up, 0);
        }
        if (e != cudaSuccess) { cudaGetLastError(); return drain((int)e); }
        rc = bbcu_bit_BinaryLut6_Forward(static_cast<const int *>(io.x[s]), static_cast<int *>(io.y[s]), static_cast<const int *>(io.idx),
                                         static_cast<const int *>(io.table), node_size, frames_k, cw, st);
        if (rc) return drain(rc);
        e = cudaMemcpy2DAsync(host_y_buf + w0, sizeof(int) * (size_t)frame_stride, io.y[s], sizeof(int) * (size_t)cw, sizeof(int) * (size_t)nw,
                              (size_t)node_size, cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) { cudaGetLastError(); return drain((int)e); }
        w0 += nw;
    }
    for (int s = 0; s < kSlots; ++s) {
        const cudaError_t e = cudaStreamSynchronize(io.stream[s]);
        if (e != cudaSuccess) { cudaGetLastError(); return drain((int)e); }
    }
    return BBCU_OK;
}

// Page-locked host memory for the buffers handed to the call above (pageable memory works too, but its copies are
// staged by the driver and do not overlap).
extern "C" void *bbcu_b200_host_alloc(size_t bytes)
{
    void *p = nullptr;
    if (cudaMallocHost(&p, bytes) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return p;
}

extern "C" void bbcu_b200_host_free(void *p)
{
    if (p && cudaFreeHost(p) != cudaSuccess) cudaGetLastError();
}
