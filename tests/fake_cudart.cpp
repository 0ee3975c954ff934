// fake_cudart.cpp -- see fake_cudart.h.  Memory is the host's, copies and fills
// happen at once, launches are recorded; inside a stream capture all three are
// kept and happen when the graph is launched.
#include "fake_cudart.h"

#include <cuda_runtime_api.h>

#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>

namespace {

std::recursive_mutex mu;
std::map<const void *, std::string> kernels;         // host stub -> device name
std::map<const void *, std::vector<char>> variables;  // host symbol -> its device memory
std::vector<fake::Launch> launched;
std::vector<fake::Fill> filled;
long n_calls = 0, fail_at = -1;
std::string fail_name;
bool hit = false;
int n_captures = 0;
cudaError_t last = cudaSuccess;

struct Graph {
    std::vector<std::function<void()>> ops;
};
Graph *capturing = nullptr;

struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
thread_local std::vector<Config> configs;

std::mutex meet_mu;
std::condition_variable meet_cv;
int meet_want = 0, meet_ms = 0, meet_in = 0;

// whether this call is the one to fail
bool fails()
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (n_calls++ != fail_at) return false;
    hit = true;
    return true;
}
cudaError_t err(cudaError_t e)
{
    last = e;
    return e;
}
cudaError_t act(std::function<void()> op)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (capturing) capturing->ops.push_back(op);
    else op();
    return cudaSuccess;
}

}  // namespace

namespace fake {

void reset()
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    launched.clear();
    filled.clear();
    n_calls = 0;
    fail_at = -1;
    fail_name.clear();
    hit = false;
    n_captures = 0;
    last = cudaSuccess;
}
long calls() { return n_calls; }
void fail_call(long k) { fail_at = k; }
void fail_launch(const char *kernel) { fail_name = kernel; }
bool failed() { return hit; }
const std::vector<Launch> &launches() { return launched; }
const std::vector<Fill> &fills() { return filled; }
int captures() { return n_captures; }
void meet(int threads, int ms)
{
    std::lock_guard<std::mutex> lk(meet_mu);
    meet_want = threads;
    meet_ms = ms;
    meet_in = 0;
}

}  // namespace fake

extern "C" {

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *)
{
    kernels[host] = name;
}
void __cudaRegisterVar(void **, char *host, char *, const char *, int, size_t size, int, int) { variables[host].resize(size); }
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *host)
{
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void *>(host));
    return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, CUstream_st *st)
{
    configs.push_back({g, b, smem, st});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st)
{
    const Config c = configs.back();
    configs.pop_back();
    *g = c.grid;
    *b = c.block;
    *smem = c.smem;
    *static_cast<cudaStream_t *>(st) = c.stream;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **args, size_t, cudaStream_t)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    const std::string name = kernels[reinterpret_cast<const void *>(k)];
    bool bad = fails();
    if (!fail_name.empty() && name.find(fail_name) != std::string::npos) {
        fail_name.clear();
        bad = hit = true;
    }
    if (bad) return err(cudaErrorLaunchOutOfResources);
    return act([=] { launched.push_back({name, g.x, b.x, {}}); });
}
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "a failure the test made"; }

cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return fails() ? err(cudaErrorInvalidValue) : cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = 8;
    return fails() ? err(cudaErrorInvalidValue) : cudaSuccess;
}

cudaError_t cudaMalloc(void **p, size_t bytes)
{
    *p = nullptr;
    if (fails()) return err(cudaErrorMemoryAllocation);
    *p = std::calloc(1, bytes ? bytes : 1);   // (pages that nobody touches cost nothing)
    return *p ? cudaSuccess : err(cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) { return cudaMalloc(p, bytes); }
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaGetSymbolAddress(void **p, const void *symbol)
{
    if (fails()) return err(cudaErrorInvalidSymbol);
    *p = variables[symbol].data();
    return cudaSuccess;
}

cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t bytes, cudaMemcpyKind, cudaStream_t)
{
    if (fails() || (bytes && (!to || !from))) return err(cudaErrorInvalidValue);
    return act([=] { std::memcpy(to, from, bytes); });
}
cudaError_t cudaMemcpy(void *to, const void *from, size_t bytes, cudaMemcpyKind k) { return cudaMemcpyAsync(to, from, bytes, k, nullptr); }
cudaError_t cudaMemcpy2DAsync(void *to, size_t tp, const void *from, size_t fp, size_t width, size_t height, cudaMemcpyKind, cudaStream_t)
{
    if (fails() || !to || !from || width > tp || width > fp) return err(cudaErrorInvalidValue);
    return act([=] {
        for (size_t r = 0; r < height; ++r) std::memcpy((char *)to + r * tp, (const char *)from + r * fp, width);
    });
}
cudaError_t cudaMemsetAsync(void *p, int value, size_t bytes, cudaStream_t)
{
    if (fails() || (bytes && !p)) return err(cudaErrorInvalidValue);
    return act([=] {
        if (bytes) std::memset(p, value, bytes);
        filled.push_back({p, bytes});
    });
}
cudaError_t cudaMemset(void *p, int value, size_t bytes) { return cudaMemsetAsync(p, value, bytes, nullptr); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    *s = fails() ? nullptr : reinterpret_cast<cudaStream_t>(std::malloc(1));
    return *s ? cudaSuccess : err(cudaErrorMemoryAllocation);
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    {
        std::unique_lock<std::mutex> lk(meet_mu);
        if (meet_want > 0) {
            ++meet_in;
            meet_cv.notify_all();
            meet_cv.wait_for(lk, std::chrono::milliseconds(meet_ms), [] { return meet_in >= meet_want; });
        }
    }
    return fails() ? err(cudaErrorUnknown) : cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    if (fails()) return err(cudaErrorUnknown);
    std::lock_guard<std::recursive_mutex> lk(mu);
    capturing = new Graph;
    ++n_captures;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    *g = reinterpret_cast<cudaGraph_t>(capturing);
    capturing = nullptr;
    return fails() ? err(cudaErrorUnknown) : cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long)
{
    if (fails()) return err(cudaErrorUnknown);
    *x = reinterpret_cast<cudaGraphExec_t>(new Graph(*reinterpret_cast<Graph *>(g)));
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<Graph *>(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete reinterpret_cast<Graph *>(x); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t)
{
    if (fails()) return err(cudaErrorUnknown);
    for (auto &op : reinterpret_cast<Graph *>(x)->ops) op();
    return cudaSuccess;
}

cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = reinterpret_cast<cudaEvent_t>(std::malloc(1)); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }

}  // extern "C"
