// Standalone sort + unique of 64-bit keys in device memory: the reference's candidate-pair pass
// radix_std::sort_with_buffer followed by std::unique (godot-avbd src/radixsort.hpp:24-83,
// src/avbd/solver_broadphase.cpp:136-137), as a GPU service over a caller-owned key buffer.

#include <cstring>
#include <mutex>
#include <string>
#include <utility>

#include <cuda.h>

#include "avbdg.h"
#include "prims.cuh"

namespace avbdg {

void setLastError(const std::string &msg); // capi.cu

namespace {

int sortFail(int code, const std::string &msg) {
    setLastError(msg);
    return code;
}

__global__ void copyBackKernel(const uint64_t *src, uint64_t *dst, const int *count) {
    pdlWait();
    pdlTrigger();
    const int n = *count;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        dst[i] = src[i];
}

// Scratch of one call: alternate key buffer, radix counts, block sums of the unique pass, count.
struct SortScratch {
    uint64_t *keysAlt;
    void *radix;
    void *unique;
    int *count;
};

// The places of a call's scratch for n keys in one block of `bytes`.
struct SortLayout {
    size_t radix, unique, count, bytes;
    explicit SortLayout(int n) {
        const auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
        radix = up(static_cast<size_t>(n) * sizeof(uint64_t));
        unique = up(radix + radixScratchBytes(n));
        count = up(unique + uniqueScratchBytes(n));
        bytes = count + 256;
    }
    SortScratch at(void *base) const {
        char *b = static_cast<char *>(base);
        return SortScratch{reinterpret_cast<uint64_t *>(b), b + radix, b + unique, reinterpret_cast<int *>(b + count)};
    }
};

// The sort + unique sequence, enqueued on `stream` with caller-provided scratch.
void enqueueSortUnique(uint64_t *keys, int n, int bits, const SortScratch &s, cudaStream_t stream) {
    radixSortPairs(keys, nullptr, s.keysAlt, nullptr, n, nullptr, 0, bits, s.radix, stream);
    uniqueSorted(keys, n, s.keysAlt, s.count, s.unique, stream);
    const int grid = divUp(n, 256);
    launchK(copyBackKernel, grid < 1184 ? grid : 1184, 256, 0, stream, s.keysAlt, keys, s.count);
}

int checkArgs(uint64_t *keys, int n, int bits, int *uniqueCount) {
    if (!uniqueCount)
        return sortFail(AVBDG_ERR_INVALID, "unique_count must not be NULL");
    if (n < 0 || (n > 0 && !keys))
        return sortFail(AVBDG_ERR_INVALID, "count must be >= 0 and keys non-NULL when count > 0");
    if (bits < 1 || bits > 64)
        return sortFail(AVBDG_ERR_INVALID, "key_bits must be in [1, 64]");
    return AVBDG_OK;
}

// ---- Fixed scratch for callers that cannot allocate ----------------------------------------
//
// Some callers of this library run where device allocation is not available to them: a host
// that hands its physics thread a fixed memory budget and forbids further device allocations,
// a plugin loaded into an engine whose allocator owns all device memory, or code running while
// another component holds a stream in capture (where a cudaMalloc would break the capture).
// They own their key buffer but cannot obtain scratch. For them the sort's scratch is this
// one array in the library's own device image: it exists on every GPU that loads the library
// and stays there until the process exits.
constexpr int kStaticMaxKeys = 1 << 18; // 262,144 keys per call
constexpr size_t kStaticScratchBytes = size_t(9) << 19; // 4.5 MiB
static __device__ __align__(256) unsigned char g_staticSortScratch[kStaticScratchBytes];

// Device address of g_staticSortScratch, per device. In host code the array's name is only a
// host-side stand-in, so the address is looked up once per device, with that device current.
// The cached address lives as long as the device's primary context: cudaDeviceReset ends it
// (with every other device object of this library on that device), and a call made after a
// reset would use a stale address, so the library must not be used on a device after a reset.
constexpr int kMaxDevices = 64;
static void *g_staticScratchAddr[kMaxDevices] = {};
static std::mutex g_staticScratchMutex;

int staticScratchAddress(void **out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return sortFail(AVBDG_ERR_CUDA, "no current CUDA device for the static sort scratch");
    std::lock_guard<std::mutex> lock(g_staticScratchMutex);
    if (!g_staticScratchAddr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_staticSortScratch);
        if (e != cudaSuccess || !p)
            return sortFail(AVBDG_ERR_CUDA, std::string("cudaGetSymbolAddress of the static sort scratch: ") +
                                                cudaGetErrorString(e));
        g_staticScratchAddr[dev] = p;
    }
    *out = g_staticScratchAddr[dev];
    return AVBDG_OK;
}

// ---- Kept scratch -----------------------------------------------------------------------------
//
// A cudaMalloc and a cudaFree of a million keys' scratch take about 155 us, more than the kernels do.
// So a call leaves its block for the next one: at most one a context, of at most kKeptBytes. A
// call takes the block out (a second thread finds none and allocates), and it has waited for its stream
// before it puts it back, so no stream ever shares it. It belongs to the context it was allocated in, which
// is known by its id: no other context takes it, and after a device reset nobody does (its place, of
// kMostKept, stays taken). It is given back when a world, batch or server of its context is destroyed and when
// one of them cannot allocate.
constexpr size_t kKeptBytes = size_t(64) << 20;
constexpr int kMostKept = 64;

struct KeptScratch {
    void *base;
    size_t bytes;
    unsigned long long context;
};
static KeptScratch g_kept[kMostKept] = {};
static std::mutex g_keptMutex;

// The context's block, taken out; none: base is null.
KeptScratch takeKept(unsigned long long context) {
    KeptScratch out{};
    std::lock_guard<std::mutex> lock(g_keptMutex);
    for (KeptScratch &k : g_kept)
        if (k.base && k.context == context) {
            std::swap(out, k);
            break;
        }
    return out;
}

// Keeps a context's block; false where it has one or all places are taken.
bool putKept(const KeptScratch &block) {
    std::lock_guard<std::mutex> lock(g_keptMutex);
    KeptScratch *place = nullptr;
    for (KeptScratch &k : g_kept) {
        if (k.base && k.context == block.context)
            return false;
        if (!k.base && !place)
            place = &k;
    }
    if (place)
        *place = block;
    return place != nullptr;
}

// The id of the current context, unique in the process; 0 where there is none.
unsigned long long contextId() {
    using Fn = CUresult (*)(CUcontext, unsigned long long *);
    static const Fn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
        const cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &found);
        return reinterpret_cast<Fn>(e == cudaSuccess && found == cudaDriverEntryPointSuccess ? p : nullptr);
    }();
    unsigned long long id = 0;
    return fn && fn(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

// Scratch for one call: the kept block of the current context if it is large enough, else a new one.
class ScratchLease {
public:
    explicit ScratchLease(size_t bytes, cudaStream_t stream) {
        // A stream in capture takes none: what is captured would use it later.
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        const bool plain = cudaStreamIsCapturing(stream, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
        if (plain && (block.context = contextId())) {
            const KeptScratch kept = takeKept(block.context);
            if (kept.base && kept.bytes >= bytes) {
                block = kept;
                return;
            }
            if (kept.base)
                cudaFree(kept.base);
        }
        if (cudaMalloc(&block.base, bytes) != cudaSuccess)
            block.base = nullptr;
        block.bytes = bytes;
    }
    ~ScratchLease() {
        if (block.base && block.context && block.bytes <= kKeptBytes && idle && putKept(block))
            return;
        if (block.base)
            cudaFree(block.base);
    }
    ScratchLease(const ScratchLease &) = delete;
    ScratchLease &operator=(const ScratchLease &) = delete;
    void *base() const { return block.base; }
    bool idle = false; // the stream has been waited for: the block may be kept

private:
    KeptScratch block{};
};

} // namespace

void releaseSortScratch() {
    const unsigned long long context = contextId();
    const KeptScratch kept = context ? takeKept(context) : KeptScratch{};
    if (kept.base)
        cudaFree(kept.base);
}

} // namespace avbdg

extern "C" {

int avbdg_sort_unique_keys_static(uint64_t *d_keys, int count, int key_bits, int *unique_count, void *stream) {
    using namespace avbdg;
    int rc = checkArgs(d_keys, count, key_bits, unique_count);
    if (rc)
        return rc;
    if (count > kStaticMaxKeys)
        return sortFail(AVBDG_ERR_CAPACITY, "avbdg_sort_unique_keys_static takes at most 262144 keys per call; "
                                            "use avbdg_sort_unique_keys for larger inputs");
    if (count == 0) {
        *unique_count = 0;
        return AVBDG_OK;
    }
    const SortLayout layout(count);
    if (layout.bytes > kStaticScratchBytes)
        return sortFail(AVBDG_ERR_CAPACITY, "static sort scratch too small for this count");
    void *addr = nullptr;
    rc = staticScratchAddress(&addr);
    if (rc)
        return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const SortScratch s = layout.at(addr);
    // The array keeps whatever the previous call left. Every word this call reads is written by
    // it first (the scan's top kernel writes the count before copyBackKernel reads it); the
    // count is cleared as well, defensively.
    cudaMemsetAsync(s.count, 0, sizeof(int), st);
    enqueueSortUnique(d_keys, count, key_bits, s, st);
    const cudaError_t launch = cudaPeekAtLastError();
    int host = 0;
    cudaMemcpyAsync(&host, s.count, sizeof(int), cudaMemcpyDeviceToHost, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    const cudaError_t bad = e != cudaSuccess ? e : launch;
    if (bad != cudaSuccess) {
        cudaGetLastError(); // the error is reported through the return code
        return sortFail(AVBDG_ERR_CUDA, std::string("static sort: ") + cudaGetErrorString(bad));
    }
    *unique_count = host;
    return AVBDG_OK;
}

int avbdg_sort_unique_keys(uint64_t *d_keys, int count, int key_bits, int *unique_count, void *stream) {
    using namespace avbdg;
    int rc = checkArgs(d_keys, count, key_bits, unique_count);
    if (rc)
        return rc;
    if (count == 0) {
        *unique_count = 0;
        return AVBDG_OK;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const SortLayout layout(count);
    ScratchLease scratch(layout.bytes, st);
    if (!scratch.base())
        return sortFail(AVBDG_ERR_CAPACITY, "cudaMalloc of the sort scratch failed");
    const SortScratch s = layout.at(scratch.base());
    enqueueSortUnique(d_keys, count, key_bits, s, st);
    const cudaError_t launch = cudaPeekAtLastError();
    int host = 0;
    cudaMemcpyAsync(&host, s.count, sizeof(int), cudaMemcpyDeviceToHost, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    scratch.idle = e == cudaSuccess;
    const cudaError_t bad = e != cudaSuccess ? e : launch;
    if (bad != cudaSuccess) {
        cudaGetLastError();
        return sortFail(AVBDG_ERR_CUDA, std::string("sort: ") + cudaGetErrorString(bad));
    }
    *unique_count = host;
    return AVBDG_OK;
}

} // extern "C"
