// A CUDA runtime for host-side tests: device memory is host memory, kernels do
// nothing, and every call that the library makes is written to a log.  Preloaded
// into a child process, it takes the place of libcudart's entry points, so the
// library's host code (workspaces, streams, events, graphs, failures) runs
// without a GPU, and calls can be made to fail:
//   fake_limit(bytes)     device allocations beyond that total fail (0: none)
//   fake_fail(name, nth)  the nth call of that function from now on fails once
//   fake_pin(p, n)        a host range counts as page-locked
//   fake_hold(on)         cudaStreamSynchronize waits while set
//   fake_log(), fake_clear()
// One log line a call: the operation, its stream (a small number), its operands.
#include <cuda_runtime_api.h>
#include <cxxabi.h>

#include <condition_variable>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {

std::mutex mu;
std::condition_variable cv;
std::string text;
std::map<char*, size_t> dev_mem, host_mem;
std::map<const void*, std::string> kernels;
size_t limit = 0, used = 0;
std::string fail_name;
int fail_nth = 0;
bool hold = false;
long next_id = 1;
std::map<void*, bool> capturing;
thread_local struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t st;
} config;
thread_local cudaError_t last = cudaSuccess;

void line(const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    text += buf;
    text += '\n';
}

long id(const void* p) { return (long)(size_t)p; }

cudaError_t err(cudaError_t e)
{
    if (e != cudaSuccess) last = e;
    return e;
}

bool fails(const char* name)
{
    if (fail_nth == 0 || fail_name != name || --fail_nth != 0) return false;
    line("failed %s", name);
    return true;
}

#define ENTER                                        \
    std::unique_lock<std::mutex> lk(mu);             \
    if (fails(__func__)) return err(cudaErrorUnknown)

cudaError_t alloc(std::map<char*, size_t>& where, void** p, size_t n)
{
    *p = aligned_alloc(256, (n + 255) / 256 * 256);
    if (!*p) return err(cudaErrorMemoryAllocation);
    where[(char*)*p] = n;
    return cudaSuccess;
}

}  // namespace

extern "C" {

void fake_limit(size_t n) { std::lock_guard<std::mutex> lk(mu); limit = n; }
size_t fake_used() { std::lock_guard<std::mutex> lk(mu); return used; }
void fake_fail(const char* name, int nth) { std::lock_guard<std::mutex> lk(mu); fail_name = name; fail_nth = nth; }
void fake_pin(void* p, size_t n) { std::lock_guard<std::mutex> lk(mu); host_mem[(char*)p] = n; }
void fake_hold(int on)
{
    std::lock_guard<std::mutex> lk(mu);
    hold = on != 0;
    cv.notify_all();
}
const char* fake_log()
{
    static std::string copy;
    std::lock_guard<std::mutex> lk(mu);
    copy = text;
    return copy.c_str();
}
void fake_clear() { std::lock_guard<std::mutex> lk(mu); text.clear(); }

// ------------------------------------------------------------ modules and launches
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*)
{
    int status = 0;
    char* d = abi::__cxa_demangle(name, nullptr, nullptr, &status);
    std::string s = status == 0 ? d : name;
    free(d);
    const size_t at = s.find("k_"), paren = s.find('(', at == std::string::npos ? 0 : at);
    s = s.substr(at == std::string::npos ? 0 : at);
    if (paren != std::string::npos && at != std::string::npos) {       // without the parameters
        size_t depth = 0, i = 0;
        for (; i < s.size(); i++) {
            if (s[i] == '<') depth++;
            else if (s[i] == '>') depth--;
            else if (s[i] == '(' && depth == 0) break;
        }
        s = s.substr(0, i);
    }
    for (char& c : s)
        if (c == ' ') c = '_';
    std::lock_guard<std::mutex> lk(mu);
    kernels[host] = s;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* st)
{
    config = {g, b, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st)
{
    *g = config.grid;
    *b = config.block;
    *smem = config.smem;
    *(cudaStream_t*)st = config.st;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host)
{
    *k = (cudaKernel_t)host;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void**, size_t, cudaStream_t st)
{
    ENTER;
    line("launch %ld %s %u %u", id(st), kernels[(const void*)k].c_str(), g.x, b.x);
    return cudaSuccess;
}

// ------------------------------------------------------------ device
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp* p, int)
{
    memset((void*)p, 0, sizeof(*p));
    strcpy(p->name, "fake");
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest)
{
    *least = 0;
    *greatest = -5;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, enum cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static char scratch[1 << 23]; *p = scratch; return cudaSuccess; }
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}

// ------------------------------------------------------------ memory
cudaError_t cudaMalloc(void** p, size_t n)
{
    ENTER;
    *p = nullptr;
    if (limit && used + n > limit) {
        line("nomem %zu", n);
        return err(cudaErrorMemoryAllocation);
    }
    const cudaError_t e = alloc(dev_mem, p, n);
    if (e == cudaSuccess) used += n;
    line("malloc %ld %zu", id(*p), n);
    return e;
}
cudaError_t cudaFree(void* p)
{
    ENTER;
    if (!p) return cudaSuccess;
    line("free %ld", id(p));
    used -= dev_mem[(char*)p];
    dev_mem.erase((char*)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    ENTER;
    const cudaError_t e = alloc(host_mem, p, n);
    if (e == cudaSuccess) memset(*p, 0, n);
    return e;
}
cudaError_t cudaFreeHost(void* p)
{
    ENTER;
    host_mem.erase((char*)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void* p)
{
    ENTER;
    memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    for (auto& m : host_mem)
        if ((const char*)p >= m.first && (const char*)p < m.first + m.second) a->type = cudaMemoryTypeHost;
    for (auto& m : dev_mem)
        if ((const char*)p >= m.first && (const char*)p < m.first + m.second) a->type = cudaMemoryTypeDevice;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind kind, cudaStream_t st)
{
    ENTER;
    line("copy %ld %ld %ld %zu %d", id(st), id(d), id(s), n, (int)kind);
    if (!capturing[st]) memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind kind)
{
    ENTER;
    line("copy 0 %ld %ld %zu %d", id(d), id(s), n, (int)kind);
    memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st)
{
    ENTER;
    line("set %ld %ld %zu", id(st), id(d), n);
    if (!capturing[st]) memset(d, v, n);
    return cudaSuccess;
}

// ------------------------------------------------------------ streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned)
{
    ENTER;
    *st = (cudaStream_t)next_id++;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* st, unsigned, int)
{
    ENTER;
    *st = (cudaStream_t)next_id++;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamGetPriority(cudaStream_t, int* p) { *p = 0; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    ENTER;
    line("sync %ld", id(st));
    cv.wait(lk, [] { return !hold; });
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned)
{
    ENTER;
    line("wait %ld %ld", id(st), id(e));
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e)
{
    ENTER;
    *e = (cudaEvent_t)next_id++;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    ENTER;
    *e = (cudaEvent_t)next_id++;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st)
{
    ENTER;
    line("record %ld %ld", id(st), id(e));
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t st, enum cudaStreamCaptureMode)
{
    ENTER;
    line("begin %ld", id(st));
    if (capturing[st]) return err(cudaErrorIllegalState);
    capturing[st] = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t st, cudaGraph_t* g)
{
    std::unique_lock<std::mutex> lk(mu);
    line("end %ld", id(st));
    if (!capturing[st]) return err(cudaErrorIllegalState);
    capturing[st] = false;           // a capture that fails has ended too
    if (fails(__func__)) return err(cudaErrorUnknown);
    *g = (cudaGraph_t)next_id++;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long)
{
    ENTER;
    *x = (cudaGraphExec_t)next_id++;
    line("instantiate %ld", id(*x));
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t st)
{
    ENTER;
    line("replay %ld %ld", id(st), id(x));
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x)
{
    ENTER;
    line("destroy %ld", id(x));
    return cudaSuccess;
}

}  // extern "C"
