// bb::OptimizerAdam and a parameter that is resized in place, without a device: the few symbols of the library and of the CUDA runtime
// that it uses are stood in for here.  The device heap of this file gives every tensor one address for good, whatever its size, as the
// caching heap does within a block's 512 bytes.  Built and run by tests/test_host_headers_compile.py; prints "ok".
#include <cstdio>
#include <map>
#include <vector>

#include "bb/LutModels.h"

static std::vector<void *> g_free;
static std::vector<int> g_sizes;                 // the sizes that the operator was given

extern "C" {
int   bbcu_IsDeviceAvailable(void) { return 1; }
void *bbcu_LocalHeap_Malloc(size_t)
{
    if (g_free.empty()) return std::malloc(4096);
    void *p = g_free.back();
    g_free.pop_back();
    return p;
}
void  bbcu_LocalHeap_Free(void *p) { if (p) g_free.push_back(p); }
void *bbcu_b200_host_alloc(size_t) { return nullptr; }
void  bbcu_b200_host_free(void *) {}
char const *bbcu_b200_error_string(int) { return "refused"; }
int   bbcu_fp32_Vector_set(float *, float, int, bbcu_stream_t) { return 0; }
int   bbcu_fp32_OptimizerAdam(int n, const int *sizes, float *const *, float *const *, float *const *, float *const *, float, float, float, bbcu_stream_t)
{
    g_sizes.assign(sizes, sizes + n);
    return 0;
}
int   bbcu_fp32_OptimizerAdamUpdate(int n, const int *sizes, float *const *p, float *const *g, float *const *m, float *const *v, float lr, float b1, float b2,
                                    bbcu_stream_t s)
{
    return bbcu_fp32_OptimizerAdam(n, sizes, p, g, m, v, lr, b1, b2, s);
}
}
cudaError_t CUDARTAPI cudaMemcpyAsync(void *dst, void const *src, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(dst, src, n); return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemsetAsync(void *dst, int v, size_t n, cudaStream_t) { std::memset(dst, v, n); return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
char const *CUDARTAPI cudaGetErrorString(cudaError_t) { return ""; }

#define EXPECT(c) do { if (!(c)) { std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c); return 1; } } while (0)

int main()
{
    auto p = std::make_shared<bb::Tensor>(bb::indices_t{64}), g = std::make_shared<bb::Tensor>(bb::indices_t{64});
    auto q = std::make_shared<bb::Tensor>(bb::indices_t{8}), h = std::make_shared<bb::Tensor>(bb::indices_t{8});
    auto opt = bb::OptimizerAdam<float>::Create();
    opt->AddVariables(p, g);
    opt->AddVariables(q, h);
    opt->Step();
    EXPECT((g_sizes == std::vector<int>{64, 8}));
    float *address = p->Dev();
    p->Resize(40);
    EXPECT(p->Dev() == address);                 // the case in question: another size, the same memory
    g->Resize(40);
    g->Dev();
    for (int update = 0; update < 2; ++update) {
        if (update) opt->Update(); else opt->Step();
        EXPECT((g_sizes == std::vector<int>{40, 8}));
    }
    p->Resize(100);                              // larger than its moments: refused, nothing is launched
    g->Resize(100);
    g_sizes.clear();
    try { opt->Step(); EXPECT(false); } catch (std::runtime_error const &) {}
    EXPECT(g_sizes.empty());
    std::printf("ok\n");
    return 0;
}
