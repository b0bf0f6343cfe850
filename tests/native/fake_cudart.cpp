// A stand-in of the CUDA runtime (libcudart.so.12) for host tests of the
// drop-in: test infrastructure, no GPU.  Device memory is host memory with
// checked bounds; copies, fills and launches wait in their stream's queue
// until something waits for the stream, so that work which nothing orders runs
// as late as it may.  Kernels compute nothing: a launch is recorded, and checked
// against the attributes its function was given on the current device.  What
// breaks a rule of the runtime is counted (fake_violations, fake_message).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

// in fake_args.cu: sets a fault bit as a stage or residual launch, a launch of
// the face traces with these arguments would
void raise_stage(const void *stage_args);
void raise_trace(const void *trace_init);
size_t stage_args_bytes();
size_t trace_init_bytes();

namespace {

struct Alloc {
    size_t bytes;
    bool device;
};
std::map<char *, Alloc> mem;
size_t live = 0, peak = 0;  // device bytes
long fail_in = -1;          // device allocations until one fails (-1: none does)
int device = 0;
std::string faulty, failing;  // kernels whose launches set a fault flag, return an error
int violations = 0;
cudaError_t last = cudaSuccess;
std::string message;
std::map<std::string, long> launches;

void violation(const std::string &m)
{
    violations++;
    if (message.empty()) message = m;
}

using Work = std::function<void()>;
struct Stream {
    std::vector<Work> queue;
    std::vector<Work> *capture = nullptr;
};
struct Event {
    Stream *stream = nullptr;
};
Stream null_stream;
std::vector<Stream *> streams{&null_stream};
Stream &at(cudaStream_t s) { return s ? *reinterpret_cast<Stream *>(s) : null_stream; }
void put(Stream &s, Work w) { (s.capture ? *s.capture : s.queue).push_back(std::move(w)); }
void drain(Stream &s)
{
    std::vector<Work> q;
    q.swap(s.queue);
    for (auto &w : q) w();
}

// whether [p, p + n) lies in one allocation; host memory that was not
// allocated here is anything else
bool inside(const void *p, size_t n, bool is_device, const char *what)
{
    char *c = const_cast<char *>(static_cast<const char *>(p));
    auto it = mem.upper_bound(c);
    if (it != mem.begin()) {
        --it;
        if (c < it->first + it->second.bytes) {
            if (it->second.device != is_device && is_device) {
                violation(std::string(what) + ": host memory where device memory belongs");
                return false;
            }
            if (c + n > it->first + it->second.bytes) {
                violation(std::string(what) + " of " + std::to_string(n) + " bytes, " +
                          std::to_string(it->first + it->second.bytes - c) + " left");
                return false;
            }
            return true;
        }
    }
    if (is_device || !p) {
        violation(std::string(what) + ": not in an allocation");
        return false;
    }
    return true;
}
bool known(const void *p)
{
    char *c = const_cast<char *>(static_cast<const char *>(p));
    auto it = mem.upper_bound(c);
    return it != mem.begin() && c < (--it)->first + it->second.bytes;
}

struct Function {
    std::string name;
    std::map<int, int> smem;  // device -> dynamic shared memory it may ask for
};
std::map<const void *, Function> functions;
struct Var {
    size_t bytes;
    std::map<int, void *> at;
};
std::map<const void *, Var> vars;
struct Call {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
std::vector<Call> calls;

cudaError_t launch(const void *f, dim3 grid, size_t smem, cudaStream_t st, void **args)
{
    Function &fn = functions[f];
    launches[fn.name]++;
    if (!grid.x || smem > (size_t)std::max(48 * 1024, fn.smem.count(device) ? fn.smem[device] : 0)) {
        violation("launch of " + fn.name + " on device " + std::to_string(device) + " with " + std::to_string(smem) +
                  " bytes of shared memory");
        return cudaErrorInvalidValue;
    }
    if (!failing.empty() && fn.name.find(failing) != std::string::npos) return last = cudaErrorLaunchFailure;
    if (!faulty.empty() && fn.name.find(faulty) != std::string::npos) {
        const bool trace = faulty == "trace_kernel";
        const char *arg = static_cast<const char *>(args[trace ? 4 : 0]);
        const std::vector<char> v(arg, arg + (trace ? trace_init_bytes() : stage_args_bytes()));
        put(at(st), [trace, v] { trace ? raise_trace(v.data()) : raise_stage(v.data()); });
    }
    return cudaSuccess;
}

void *get(size_t bytes, bool dev)
{
    char *p = static_cast<char *>(std::calloc(1, bytes));
    mem[p] = {bytes, dev};
    if (dev) live += bytes, peak = std::max(peak, live);
    return p;
}
void release(void *p)
{
    auto it = mem.find(static_cast<char *>(p));
    if (!p) return;
    if (it == mem.end()) return violation("free of what was not allocated");
    if (it->second.device) live -= it->second.bytes;
    std::free(p);
    mem.erase(it);
}

}  // namespace

extern "C" {

// ---- the tests' side --------------------------------------------------------------
int fake_violations() { return violations; }
const char *fake_message() { return message.c_str(); }
void fake_fault(const char *kernel) { faulty = kernel; }
void fake_fail(const char *kernel) { failing = kernel; }
void fake_fail_alloc(long n) { fail_in = n; }
size_t fake_live() { return live; }
size_t fake_peak() { return peak; }
void fake_reset_peak() { peak = live; }
long fake_launches(const char *part)
{
    long n = 0;
    for (auto &l : launches)
        if (l.first.find(part) != std::string::npos) n += l.second;
    return n;
}

// ---- the runtime's ------------------------------------------------------------------
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError()
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { *lo = 0; *hi = -5; return cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t n)
{
    if (fail_in >= 0 && fail_in-- == 0) {
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    *p = get(n, true);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)  // waits for the device
{
    for (Stream *s : streams) drain(*s);
    release(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { *p = get(n, false); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaGetSymbolAddress(void **p, const void *sym)
{
    Var &v = vars[sym];
    if (!v.at[device]) v.at[device] = get(v.bytes, true);
    *p = v.at[device];
    return cudaSuccess;
}

cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st)
{
    const bool dd = k != cudaMemcpyDeviceToHost, sd = k != cudaMemcpyHostToDevice;
    if (!inside(d, n, dd, "copy to") || !inside(s, n, sd, "copy from")) return cudaErrorInvalidValue;
    if (!sd && !known(s)) {  // pageable: read before the call returns
        std::vector<char> v((const char *)s, (const char *)s + n);
        put(at(st), [d, v] { std::memcpy(d, v.data(), v.size()); });
    } else {
        put(at(st), [=] { std::memmove(d, s, n); });
        if (!dd && !known(d)) drain(at(st));  // pageable: written before the call returns
    }
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st)
{
    if (!inside(d, n, true, "fill")) return cudaErrorInvalidValue;
    put(at(st), [=] { std::memset(d, v, n); });
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { streams.push_back(new Stream); *s = reinterpret_cast<cudaStream_t>(streams.back()); return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { drain(at(s)); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { drain(at(s)); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t e, unsigned)
{
    Event *v = reinterpret_cast<Event *>(e);
    if (v->stream) drain(*v->stream);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = reinterpret_cast<cudaEvent_t>(new Event); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    reinterpret_cast<Event *>(e)->stream = &at(s);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return cudaStreamWaitEvent(nullptr, e, 0); }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) { at(s).capture = new std::vector<Work>; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g)
{
    *g = reinterpret_cast<cudaGraph_t>(at(s).capture);
    at(s).capture = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long)
{
    *x = reinterpret_cast<cudaGraphExec_t>(new std::vector<Work>(*reinterpret_cast<std::vector<Work> *>(g)));
    launches["graph instantiation"]++;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<std::vector<Work> *>(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete reinterpret_cast<std::vector<Work> *>(x); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s)
{
    for (auto &w : *reinterpret_cast<std::vector<Work> *>(x)) put(at(s), w);
    launches["graph launch"]++;
    return cudaSuccess;
}

cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v)
{
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) functions[f].smem[device] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3, void **args, size_t smem, cudaStream_t st) { return launch(f, g, smem, st, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args)
{
    return launch(f, c->gridDim, c->dynamicSmemBytes, c->stream, args);
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *st)
{
    calls.push_back({g, b, smem, st});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st)
{
    const Call c = calls.back();
    calls.pop_back();
    *g = c.grid;
    *b = c.block;
    *smem = c.smem;
    *static_cast<cudaStream_t *>(st) = c.stream;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *)
{
    functions[f].name = name;
}
void __cudaRegisterVar(void **, char *var, char *, const char *, int, size_t size, int, int) { vars[var].bytes = size; }
char __cudaInitModule(void **) { return 1; }

}  // extern "C"
