// A stand-in for the CUDA runtime, for tests of the library's host side on a
// machine without a GPU: device memory is host memory, kernels do nothing, and
// the order of calls is watched.  Linked with the library's own objects.
//
// Streams are numbered handles; work on them is only counted.  What is
// watched:
//   * fake_hazards: launches made while the clear of a new allocation may
//     still run (cleared as a whole, on another stream than the launch's that
//     nobody has waited for since);
//   * fake_launches, fake_allocated, fake_uploaded: totals;
//   * fake_mapped: bytes of the caller's memory whose pages were asked for.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstring>
#include <map>
#include <set>

namespace {
struct Call {
    dim3 grid, block;
    std::size_t shared;
    cudaStream_t stream;
};
thread_local Call pushed;
thread_local int device = 0;
int devices = 1;
long long launches = 0, hazards = 0;
std::size_t allocated = 0, uploaded = 0, mapped = 0;
std::map<char*, std::size_t> memory;
std::multimap<std::size_t, char*> given_back;  // reused for an equal size, as the allocator does
std::set<cudaStream_t> clearing;               // streams with the clear of an allocation in flight
std::size_t handles = 0;
char symbol[1 << 20];

void* handle() { return reinterpret_cast<void*>(0x1000 + 16 * ++handles); }

void cleared(void* p, std::size_t bytes, cudaStream_t stream) {
    const auto at = memory.find(static_cast<char*>(p));
    if (at != memory.end() && at->second == bytes) clearing.insert(stream);
}
void uploading(std::size_t bytes, cudaMemcpyKind kind) {
    if (kind == cudaMemcpyHostToDevice) uploaded += bytes;
}
}  // namespace

extern "C" {
void fake_devices(int n) { devices = n; }
void fake_device(int n) { device = n; }
long long fake_launches() { return launches; }
long long fake_hazards() { return hazards; }
std::size_t fake_allocated() { return allocated; }
std::size_t fake_uploaded() { return uploaded; }
std::size_t fake_mapped() { return mapped; }
void* fake_stream() { return handle(); }

// The library's requests for pages come here; they change nothing.
int madvise(void*, std::size_t bytes, int) noexcept {
    mapped += bytes;
    return 0;
}

cudaError_t cudaGetDeviceCount(int* n) { *n = devices; return cudaSuccess; }
cudaError_t cudaGetDevice(int* n) { *n = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int n) { device = n; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr attribute, int) {
    *value = attribute == cudaDevAttrMultiProcessorCount ? 152 : 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) { *least = 0; *greatest = -5; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { clearing.clear(); return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }

cudaError_t cudaMalloc(void** p, std::size_t bytes) {
    const auto again = given_back.find(bytes);
    char* at = nullptr;
    if (again != given_back.end()) {
        at = again->second;
        given_back.erase(again);
    } else {
        at = static_cast<char*>(mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0));
        if (at == MAP_FAILED) return cudaErrorMemoryAllocation;
    }
    memory[at] = bytes;
    allocated += bytes;
    *p = at;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    const auto at = memory.find(static_cast<char*>(p));
    if (at != memory.end()) {
        allocated -= at->second;
        given_back.emplace(at->second, at->first);
        memory.erase(at);
    }
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int value, std::size_t bytes) {
    cleared(p, bytes, nullptr);
    std::memset(p, value, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int value, std::size_t bytes, cudaStream_t stream) {
    cleared(p, bytes, stream);
    std::memset(p, value, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* to, const void* from, std::size_t bytes, cudaMemcpyKind kind) {
    clearing.erase(nullptr);
    uploading(bytes, kind);
    std::memcpy(to, from, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, std::size_t bytes, cudaMemcpyKind kind, cudaStream_t) {
    uploading(bytes, kind);
    std::memcpy(to, from, bytes);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = symbol; return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = static_cast<cudaStream_t>(handle()); return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { *s = static_cast<cudaStream_t>(handle()); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { clearing.erase(s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* status) {
    *status = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = static_cast<cudaGraph_t>(handle()); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) { *g = static_cast<cudaGraphExec_t>(handle()); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = static_cast<cudaEvent_t>(handle()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = static_cast<cudaEvent_t>(handle()); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }

cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { std::memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, std::size_t) { *n = 4; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, std::size_t, unsigned) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* result) {
    *f = reinterpret_cast<void*>(+[]() -> int { return 0; });  // a driver call that succeeds, whatever its arguments
    *result = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

void** __cudaRegisterFatBinary(void*) { static void* at = nullptr; return &at; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, std::size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, std::size_t shared, cudaStream_t stream) {
    pushed = Call{grid, block, shared, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, std::size_t* shared, void* stream) {
    *grid = pushed.grid;
    *block = pushed.block;
    *shared = pushed.shared;
    *static_cast<cudaStream_t*>(stream) = pushed.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(void** kernel, const void* function) {
    *kernel = const_cast<void*>(function);
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(void*, dim3, dim3, void**, std::size_t, cudaStream_t stream) {
    ++launches;
    for (cudaStream_t other : clearing) {
        if (other != stream) {
            ++hazards;
            break;
        }
    }
    return cudaSuccess;
}
}
