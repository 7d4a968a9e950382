// A CUDA runtime without a device, for LD_PRELOAD in front of libcudart: memory is host memory set to
// zero, copies are memmove, launches and graphs do nothing.  It lets the library's host side run on a CPU
// and its allocations fail one at a time.
//
//   fake_fail_at(n)   the n-th device allocation from now fails (1: the next one; 0: none)
//   fake_allocs()     device allocations asked for since fake_fail_at
//   fake_live(n, v)   device allocations alive: their number, the sizes of the first n in v, ascending
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

namespace {
std::mutex mu;
std::map<void*, size_t> live;
long long asked = 0, fail_at = 0;
thread_local int last_error = 0;
constexpr int kOutOfMemory = 2;
char symbol[1 << 21];
int dummy;

int device_alloc(void** p, size_t n) {
    std::lock_guard<std::mutex> lock(mu);
    if (++asked == fail_at) return last_error = kOutOfMemory;
    *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
    std::memset(*p, 0, n);
    live[*p] = n;
    return 0;
}
int device_free(void* p) {
    std::lock_guard<std::mutex> lock(mu);
    live.erase(p);
    std::free(p);
    return 0;
}
}  // namespace

extern "C" {
void fake_fail_at(long long n) { std::lock_guard<std::mutex> lock(mu); asked = 0; fail_at = n; }
long long fake_allocs() { std::lock_guard<std::mutex> lock(mu); return asked; }
long long fake_live(long long n, long long* v) {
    std::lock_guard<std::mutex> lock(mu);
    std::vector<long long> s;
    for (auto& b : live) s.push_back((long long)b.second);
    std::sort(s.begin(), s.end());
    for (size_t i = 0; i < s.size() && (long long)i < n; ++i) v[i] = s[i];
    return (long long)s.size();
}

int cudaMalloc(void** p, size_t n) { return device_alloc(p, n); }
int cudaMallocAsync(void** p, size_t n, void*) { return device_alloc(p, n); }
int cudaFree(void* p) { return device_free(p); }
int cudaFreeAsync(void* p, void*) { return device_free(p); }
int cudaMallocHost(void** p, size_t n) { *p = std::calloc(1, n); return 0; }
int cudaFreeHost(void* p) { std::free(p); return 0; }
int cudaMemcpy(void* d, const void* s, size_t n, int) { std::memmove(d, s, n); return 0; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int, void*) { std::memmove(d, s, n); return 0; }
int cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return 0; }
int cudaMemsetAsync(void* d, int v, size_t n, void*) { std::memset(d, v, n); return 0; }

int cudaGetLastError() { const int e = last_error; last_error = 0; return e; }
const char* cudaGetErrorString(int e) { return e == kOutOfMemory ? "out of memory" : "an error"; }

int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaSetDevice(int) { return 0; }
int cudaGetDeviceCount(int* n) { *n = 1; return 0; }
int cudaDeviceGetAttribute(int* v, int, int) { *v = 152; return 0; }
int cudaDeviceGetDefaultMemPool(void** p, int) { *p = &dummy; return 0; }
int cudaMemPoolSetAttribute(void*, int, void*) { return 0; }
int cudaDeviceSynchronize() { return 0; }
int cudaGetSymbolAddress(void** p, const void*) { *p = symbol; return 0; }

int cudaStreamCreateWithFlags(void** s, unsigned) { *s = std::malloc(1); return 0; }
int cudaStreamDestroy(void* s) { std::free(s); return 0; }
int cudaStreamSynchronize(void*) { return 0; }
int cudaStreamWaitEvent(void*, void*, unsigned) { return 0; }
int cudaStreamBeginCapture(void*, int) { return 0; }
int cudaStreamBeginCaptureToGraph(void*, void*, const void*, const void*, size_t, int) { return 0; }
int cudaStreamEndCapture(void*, void** g) { *g = &dummy; return 0; }
int cudaEventCreate(void** e) { *e = &dummy; return 0; }
int cudaEventCreateWithFlags(void** e, unsigned) { *e = &dummy; return 0; }
int cudaEventDestroy(void*) { return 0; }
int cudaEventRecord(void*, void*) { return 0; }
int cudaEventSynchronize(void*) { return 0; }
int cudaEventElapsedTime(float* t, void*, void*) { *t = 0.0f; return 0; }

int cudaGraphCreate(void** g, unsigned) { *g = &dummy; return 0; }
int cudaGraphDestroy(void*) { return 0; }
int cudaGraphAddNode(void** n, void*, const void*, const void*, size_t, void* params) {
    // the conditional node's body: phGraph_out, after the handle, the type and the size
    *n = &dummy;
    static void* body[1] = {&dummy};
    struct Conditional { unsigned long long handle; int type; unsigned size; void** graphs; };
    reinterpret_cast<Conditional*>(static_cast<char*>(params) + 16)->graphs = body;
    return 0;
}
int cudaGraphConditionalHandleCreate(unsigned long long* h, void*, unsigned, unsigned) { *h = 1; return 0; }
int cudaGraphInstantiate(void** e, void*, unsigned long long) { *e = &dummy; return 0; }
int cudaGraphLaunch(void*, void*) { return 0; }
int cudaGraphExecDestroy(void*) { return 0; }

int cudaFuncGetAttributes(void* a, const void*) { std::memset(a, 0, 64); return 0; }
int cudaFuncSetAttribute(const void*, int, int) { return 0; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}

struct Dim3 { unsigned x, y, z; };
extern "C" {
unsigned __cudaPushCallConfiguration(Dim3, Dim3, size_t, void*) { return 0; }
int __cudaPopCallConfiguration(Dim3* g, Dim3* b, size_t* sm, void* s) {
    *g = *b = Dim3{1, 1, 1};
    *sm = 0;
    *static_cast<void**>(s) = nullptr;
    return 0;
}
int __cudaGetKernel(void** k, const void*) { *k = &dummy; return 0; }
int __cudaLaunchKernel(void*, Dim3, Dim3, void**, size_t, void*) { return 0; }
int cudaLaunchKernel(const void*, Dim3, Dim3, void**, size_t, void*) { return 0; }
}
