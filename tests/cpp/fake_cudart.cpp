// A CUDA runtime that runs nothing, for tests of the host code on a machine without a
// GPU: device memory is host memory, kernels are counted instead of run, and a
// host-to-device copy or a memset on the legacy stream stays outstanding until that
// stream (or the device) is waited for, the latest that the runtime's documentation
// allows. Linked with the library's own objects in place of the runtime.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <utility>
#include <vector>

namespace
{
struct Write
{
    void *dst;
    std::vector<unsigned char> bytes;
};
std::vector<Write> outstanding;
int early_launches = 0, launches = 0, attribute_queries = 0;
std::map<std::pair<int, const void *>, size_t> smem_limit; // by device and kernel
int device             = 0;
cudaError_t last_error = cudaSuccess;
long next_handle = 0x1000, allocated = 0;

bool Legacy(cudaStream_t s)
{
    return s == nullptr || s == cudaStreamLegacy || s == cudaStreamPerThread;
}
void Land()
{
    for (const Write &w : outstanding)
        std::memcpy(w.dst, w.bytes.data(), w.bytes.size());
    outstanding.clear();
}
template <typename H> cudaError_t Handle(H *h)
{
    *h = reinterpret_cast<H>(next_handle += 16);
    return cudaSuccess;
}
cudaError_t Put(void *dst, const void *src, size_t n, bool to_host)
{
    if (to_host)
    {
        Land();
        std::memcpy(dst, src, n);
    }
    else if (n)
    {
        const unsigned char *p = static_cast<const unsigned char *>(src);
        outstanding.push_back({dst, std::vector<unsigned char>(p, p + n)});
    }
    return cudaSuccess;
}
} // namespace

extern "C" {
int fake_outstanding() { return int(outstanding.size()); }
int fake_early_launches() { return early_launches; }
int fake_launches() { return launches; }
long fake_allocated() { return allocated; }
int fake_attribute_queries() { return attribute_queries; }

void **__cudaRegisterFatBinary(void *) { return reinterpret_cast<void **>(&next_handle); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *,
                            void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

struct Call
{
    dim3 grid, block;
    size_t smem;
    void *stream;
} call;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, void *s)
{
    call = {g, b, m, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s)
{
    *g = call.grid, *b = call.block, *m = call.smem;
    *static_cast<void **>(s) = call.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *kernel, dim3 grid, dim3 block, void **, size_t smem,
                             cudaStream_t s)
{
    if (!grid.x || !grid.y || !grid.z || !block.x)
        return last_error = cudaErrorInvalidConfiguration;
    const auto limit = smem_limit.find({device, kernel});
    if (smem > (limit == smem_limit.end() ? 48 * 1024 : limit->second))
        return last_error = cudaErrorInvalidValue;
    ++launches;
    if (!Legacy(s) && !outstanding.empty())
        ++early_launches;
    return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int *n) { return *n = 2, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return device = d, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int)
{
    ++attribute_queries;
    return *v = 148, cudaSuccess;
}
cudaError_t cudaRuntimeGetVersion(int *v) { return *v = CUDART_VERSION, cudaSuccess; }
cudaError_t cudaGetLastError()
{
    const cudaError_t e = last_error;
    last_error          = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaFuncSetAttribute(const void *kernel, cudaFuncAttribute, int v)
{
    if (v > 227 * 1024)
        return cudaErrorInvalidValue;
    smem_limit[{device, kernel}] = size_t(v);
    return cudaSuccess;
}

cudaError_t cudaMalloc(void **p, size_t n)
{
    allocated += long(n);
    return *p = std::calloc(n + 1, 1), cudaSuccess;
}
cudaError_t cudaFree(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { return cudaMalloc(p, 1 << 16); }

cudaError_t cudaMemcpy(void *dst, const void *src, size_t n, cudaMemcpyKind k)
{
    return Put(dst, src, n, k == cudaMemcpyDeviceToHost);
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind k, cudaStream_t s)
{
    if (Legacy(s))
        return Put(dst, src, n, k == cudaMemcpyDeviceToHost);
    std::memcpy(dst, src, n); // in its stream's order
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *dst, size_t dp, const void *src, size_t sp, size_t w, size_t h,
                              cudaMemcpyKind, cudaStream_t)
{
    for (size_t r = 0; r < h; ++r)
        std::memcpy(static_cast<char *>(dst) + r * dp, static_cast<const char *>(src) + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *dst, int v, size_t n)
{
    outstanding.push_back({dst, std::vector<unsigned char>(n, static_cast<unsigned char>(v))});
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *dst, int v, size_t n, cudaStream_t s)
{
    return Legacy(s) ? cudaMemset(dst, v, n) : (std::memset(dst, v, n), cudaSuccess);
}
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    if (Legacy(s))
        Land();
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return Land(), cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return Handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return Handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return Handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t)
{
    return *ms = 1.0f, cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return Handle(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long)
{
    return Handle(e);
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
} // extern "C"
