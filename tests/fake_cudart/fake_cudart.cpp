// A CUDA runtime without a GPU, for tests of the library's host code: built as
// libcudart.so.13 and put before the real one in a child process's library
// path.  Device memory is zeroed host memory and kernels do nothing, except
// those of the packet indexer and the header gather, so that streams open.
// Two devices.  What it watches is read back with fake_count:
//   launch:<text>   launches of kernels whose (mangled) name holds the text
//   pending         1 after a copy of pageable memory or a memset on the legacy
//                   stream that nothing waited for
//   unordered       launches on another stream while that is so
//   stale           copies queued on a stream whose pageable source had changed or
//                   gone by the time the stream was waited for
//   refused         launches with more dynamic shared memory than the kernel may
//                   have on the current device (they fail, as on a GPU)
//   capture, replay graphs captured and launched
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <utility>
#include <vector>

namespace {

struct Var {
    void* mem[2] = {nullptr, nullptr};
    size_t size = 0;
};
struct Config {
    dim3 grid, block;
    size_t smem = 0;
    cudaStream_t stream = nullptr;
};

std::recursive_mutex mu;
std::map<const void*, std::string> kernels;
std::map<const void*, Var> vars;
std::map<std::string, long long> counts, launches;
std::map<std::pair<const void*, int>, int> smem_limit;
std::set<void*> page_locked;
std::string last_unordered;
bool legacy_copy = false;
// queued copies from pageable memory: what the device may read as late as when
// the stream is waited for, and what it has to read
struct Queued {
    cudaStream_t stream;
    const void* src;
    std::string data;
};
std::vector<Queued> queued;
cudaStream_t capturing = nullptr;
thread_local Config config;
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;

using Lock = std::lock_guard<std::recursive_mutex>;

cudaError_t fail(cudaError_t e) {
    last = e;
    return e;
}
bool legacy(cudaStream_t s) { return s == nullptr || s == cudaStreamLegacy; }
bool pageable(const void* p) { return page_locked.empty() || !page_locked.count(const_cast<void*>(p)); }
void* handle() { return std::calloc(1, 16); }
void waited(cudaStream_t stream, bool all) {
    std::vector<Queued> rest;
    for (Queued& q : queued) {
        if (!all && q.stream != stream) rest.push_back(std::move(q));
        else if (std::memcmp(q.src, q.data.data(), q.data.size()) != 0) ++counts["stale"];
    }
    queued.swap(rest);
}

// parameter i of a launch
template <typename T>
T arg(void** a, int i) { return *static_cast<T*>(a[i]); }

long long next_packet(const uint8_t* s, long long p) { return p + 7 + ((long long)s[p + 4] << 8 | s[p + 5]); }

void emulate(const std::string& name, void** a) {
    if (name.find("k_index_fix") != std::string::npos) {
        const uint8_t* s = arg<const uint8_t*>(a, 0);
        const long long n = arg<long long>(a, 1);
        int total = 0;
        for (long long p = 0; p + 6 <= n; p = next_packet(s, p)) ++total;
        *arg<int*>(a, 8) = total;
    } else if (name.find("k_index_write") != std::string::npos) {
        const uint8_t* s = arg<const uint8_t*>(a, 0);
        const long long n = arg<long long>(a, 1);
        long long* out = arg<long long*>(a, 7);
        const int most = arg<int>(a, 8);
        int i = 0;
        for (long long p = 0; p + 6 <= n; p = next_packet(s, p))
            if (i < most) out[i++] = p;
    } else if (name.find("k_gather_headers") != std::string::npos) {
        const uint8_t* s = arg<const uint8_t*>(a, 0);
        const long long n = arg<long long>(a, 1);
        const long long* off = arg<const long long*>(a, 2);
        const int npk = arg<int>(a, 3);
        uint8_t* hdr = arg<uint8_t*>(a, 4);
        for (long long i = 0; i < (long long)npk * 68; ++i) {
            const long long at = off[i / 68] + i % 68;
            hdr[i] = at < n ? s[at] : 0;
        }
    }
}

void* var_memory(const void* symbol) {
    const auto it = vars.find(symbol);
    if (it == vars.end()) return nullptr;
    void*& m = it->second.mem[device];
    if (!m) m = std::calloc(1, it->second.size);
    return m;
}

}  // namespace

extern "C" {

long long fake_count(const char* what) {
    Lock lk(mu);
    const std::string w = what;
    if (w == "pending") return legacy_copy;
    if (w.rfind("launch:", 0) != 0) return counts[w];
    long long n = 0;
    for (const auto& kv : launches)
        if (kv.first.find(w.substr(7)) != std::string::npos) n += kv.second;
    return n;
}
const char* fake_last_unordered() { return last_unordered.c_str(); }

// ---- registration and launches
void** __cudaRegisterFatBinary(void*) { return static_cast<void**>(handle()); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    Lock lk(mu);
    kernels[host] = name;
}
void __cudaRegisterVar(void**, char* host, char*, const char*, int, size_t size, int, int) {
    Lock lk(mu);
    vars[host].size = size;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* stream) {
    config = Config{grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *static_cast<cudaStream_t*>(stream) = config.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* kernel, const void* entry) {
    *kernel = reinterpret_cast<cudaKernel_t>(const_cast<void*>(entry));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t kernel, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t stream) {
    Lock lk(mu);
    const void* entry = reinterpret_cast<const void*>(kernel);
    const std::string& name = kernels[entry];
    const auto lim = smem_limit.find({entry, device});
    if (smem > (size_t)(lim == smem_limit.end() ? 48 * 1024 : lim->second)) {
        ++counts["refused"];
        return fail(cudaErrorInvalidValue);
    }
    if (!grid.x || !grid.y || !grid.z || grid.y > 65535 || grid.z > 65535 || block.x * block.y * block.z > 1024)
        return fail(cudaErrorInvalidConfiguration);
    if (legacy_copy && !legacy(stream)) {
        ++counts["unordered"];
        last_unordered = name;
    }
    ++launches[name];
    emulate(name, args);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* entry, cudaFuncAttribute attr, int value) {
    Lock lk(mu);
    if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (value > 227 * 1024) return fail(cudaErrorInvalidValue);
        smem_limit[{entry, device}] = value;
    }
    return cudaSuccess;
}

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) {
    if (capturing) return fail(cudaErrorStreamCaptureUnsupported);
    *p = std::aligned_alloc(256, (n + 511) / 256 * 256);
    if (!*p) return fail(cudaErrorMemoryAllocation);
    std::memset(*p, 0, n);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    Lock lk(mu);
    *p = std::calloc(1, n);
    page_locked.insert(*p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) {
    Lock lk(mu);
    page_locked.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind kind) {
    Lock lk(mu);
    std::memcpy(d, s, n);
    legacy_copy = kind == cudaMemcpyHostToDevice && pageable(s);   // the others end the legacy stream's work
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t stream) {
    Lock lk(mu);
    std::memcpy(d, s, n);
    if (kind == cudaMemcpyHostToDevice && pageable(s)) {
        if (legacy(stream)) legacy_copy = true;
        else queued.push_back({stream, s, std::string((const char*)s, n)});
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    for (size_t r = 0; r < h; ++r) std::memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t stream) {
    Lock lk(mu);
    std::memset(d, v, n);
    if (legacy(stream)) legacy_copy = true;
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }
cudaError_t cudaMemcpyToSymbol(const void* symbol, const void* s, size_t n, size_t off, cudaMemcpyKind) {
    Lock lk(mu);
    std::memcpy((char*)var_memory(symbol) + off, s, n);
    legacy_copy = true;
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbolAsync(const void* symbol, const void* s, size_t n, size_t off, cudaMemcpyKind, cudaStream_t stream) {
    Lock lk(mu);
    std::memcpy((char*)var_memory(symbol) + off, s, n);
    if (legacy(stream)) legacy_copy = true;
    return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void* d, const void* symbol, size_t n, size_t off, cudaMemcpyKind) {
    Lock lk(mu);
    std::memcpy(d, (char*)var_memory(symbol) + off, n);
    legacy_copy = false;
    return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbolAsync(void* d, const void* symbol, size_t n, size_t off, cudaMemcpyKind, cudaStream_t) {
    Lock lk(mu);
    std::memcpy(d, (char*)var_memory(symbol) + off, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) {
    Lock lk(mu);
    *p = var_memory(symbol);
    return *p ? cudaSuccess : fail(cudaErrorInvalidSymbol);
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    Lock lk(mu);
    std::memset(a, 0, sizeof(*a));
    a->type = pageable(p) ? cudaMemoryTypeDevice : cudaMemoryTypeHost;
    a->device = device;
    return cudaSuccess;
}

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = static_cast<cudaStream_t>(handle());
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    Lock lk(mu);
    if (capturing) return fail(cudaErrorStreamCaptureUnsupported);
    if (legacy(s)) legacy_copy = false;
    waited(s, false);
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    Lock lk(mu);
    legacy_copy = false;
    waited(nullptr, true);
    return capturing ? fail(cudaErrorStreamCaptureUnsupported) : cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* st) {
    *st = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    capturing = s;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    Lock lk(mu);
    capturing = nullptr;
    ++counts["capture"];
    *g = static_cast<cudaGraph_t>(handle());
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    *x = static_cast<cudaGraphExec_t>(handle());
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
    Lock lk(mu);
    ++counts["replay"];
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    std::free(g);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    std::free(x);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = static_cast<cudaEvent_t>(handle());
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}

// ---- devices and errors
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = device;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d > 1) return fail(cudaErrorInvalidDevice);
    device = d;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 152;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }

// a tensor map nobody reads
static int encode_nothing() { return 0; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
    *f = reinterpret_cast<void*>(&encode_nothing);
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

}  // extern "C"
