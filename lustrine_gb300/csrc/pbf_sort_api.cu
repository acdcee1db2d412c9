// pbf_sort_api.cu -- the reference's counting sort (Sorting::counting_sort,
// src/neighbors/Sorting.cpp:12-34) as a C entry point on device arrays.
//
// The sort's kernels take some 30 us for a million keys; what a call cost
// beside them was memory.  Scratch from the device's default pool goes back
// to the system at every synchronisation (its release threshold is 0), so each
// call mapped and unmapped it: 175 of 215 us.  The scratch comes from a pool of
// this library's own instead, which keeps up to SCRATCH_KEPT bytes between
// calls; what a larger call took beyond that goes back when it ends, and
// lustrine_release_scratch gives back the rest.  Whether a key was out of
// range is read from a page-locked word that the histogram writes only then
// (a copy from the device otherwise, when all words are in use).  Both are
// shared by threads: the pool is stream-ordered, a word belongs to one call.
// Both end with the device's context: a call after a device reset (or from a
// second context of the device) finds that they are not its own.
#include <atomic>
#include <cstdio>
#include <mutex>

#include <cuda.h>

#include "lustrine_gb300.h"
#include "pbf_context.h"
#include "pbf_kernels.h"

using namespace lgb;

namespace {

constexpr unsigned long long SCRATCH_KEPT = 128ull << 20;
constexpr int kMaxDevices = 64;
constexpr int kWords = 64;

struct DeviceScratch {
    unsigned long long context = 0;  // the context both belong to
    cudaMemPool_t pool = nullptr;
    int* words = nullptr;  // page-locked, kWords ints
    std::atomic<bool> used[kWords];
};
std::mutex g_lock;
DeviceScratch g_scratch[kMaxDevices];

// The current context's id, never used twice in a process; 0 if unknown.
unsigned long long context_id() {
    static const auto get = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return (CUresult(CUDAAPI*)(CUcontext, unsigned long long*))f;
    }();
    unsigned long long id = 0;
    return get && get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

// Whether the words are still page-locked memory (not after a reset).
bool alive(const int* words) {
    cudaPointerAttributes a = {};
    if (cudaPointerGetAttributes(&a, words) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost && a.hostPointer == words;
}

bool open_scratch(DeviceScratch& d, int dev) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    unsigned long long keep = SCRATCH_KEPT;
    if (cudaMemPoolCreate(&d.pool, &props) == cudaSuccess) {
        if (cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess &&
            cudaHostAlloc((void**)&d.words, kWords * sizeof(int),
                          cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess)
            return true;
        cudaMemPoolDestroy(d.pool);
    }
    cudaGetLastError();
    return false;
}

// The current device's scratch, or nullptr (the default pool and a status word
// on the device serve).
DeviceScratch* device_scratch(bool create) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    if (cudaFree(nullptr) != cudaSuccess) return nullptr;  // the device's context made current
    const unsigned long long context = context_id();
    if (!context) return nullptr;
    std::lock_guard<std::mutex> lock(g_lock);
    DeviceScratch& d = g_scratch[dev];
    if (d.words && alive(d.words)) return d.context == context ? &d : nullptr;
    d.words = nullptr;
    for (auto& u : d.used) u.store(false);
    if (!create || !open_scratch(d, dev)) return nullptr;
    d.context = context;
    return &d;
}

// A page-locked word of this call's own, zero; -1 when none is free.
int take_word(DeviceScratch* d) {
    for (int k = 0; d && k < kWords; k++) {
        bool free = false;
        if (d->used[k].compare_exchange_strong(free, true)) {
            *(volatile int*)&d->words[k] = 0;
            return k;
        }
    }
    return -1;
}

int sort_args_ok(const int* counts, const int* keys, size_t n, size_t num_cells, const int* sorted) {
    if (!counts || num_cells < 1 || num_cells > (size_t)(1 << 30)) return 0;
    if (n > (size_t)(1 << 30)) return 0;
    if (n > 0 && (!keys || !sorted)) return 0;
    return 1;
}

}  // namespace

extern "C" int lustrine_counting_sort(int* counts, const int* keys, size_t num_positions,
                                      size_t num_cells, int* sorted_indices, void* stream) {
    if (!sort_args_ok(counts, keys, num_positions, num_cells, sorted_indices)) return LUSTRINE_ERR_ARGS;
    cudaStream_t st = (cudaStream_t)stream;
    const int n = (int)num_positions, C = (int)num_cells;
    const bool copy_keys = counting_sort_copies_keys(counts, keys, num_positions, num_cells, sorted_indices);
    const size_t bytes = counting_sort_scratch_ints_for(num_positions, num_cells, copy_keys) * sizeof(int);
    int* scratch = nullptr;
    DeviceScratch* const kept = device_scratch(true);
    cudaError_t e = kept ? cudaMallocFromPoolAsync((void**)&scratch, bytes, kept->pool, st)
                         : cudaMallocAsync((void**)&scratch, bytes, st);
    if (e != cudaSuccess) return lgb_cuda_status(e, "cudaMallocAsync");
    CountingSortScratch w = counting_sort_scratch(scratch, n, C, copy_keys);
    int bad = 0;
    const int word = take_word(kept);
    // the histogram and the status word behind it start at zero
    e = cudaMemsetAsync(w.count, 0, ((size_t)C + 1) * sizeof(int), st);
    if (e == cudaSuccess) {
        int* const device_status = w.status;
        if (word >= 0) w.status = &kept->words[word];
        e = launch_counting_sort(keys, n, C, w, counts, sorted_indices, st);
        if (word < 0 && e == cudaSuccess)
            e = cudaMemcpyAsync(&bad, device_status, sizeof(int), cudaMemcpyDeviceToHost, st);
    }
    const cudaError_t e1 = cudaFreeAsync(scratch, st);
    const cudaError_t e2 = cudaStreamSynchronize(st);
    if (word >= 0) {
        bad = *(volatile int*)&kept->words[word];
        kept->used[word].store(false);
    }
    if (e == cudaSuccess) e = e2 != cudaSuccess ? e2 : e1;
    if (e != cudaSuccess) return lgb_cuda_status(e, "counting_sort");
    return bad ? LUSTRINE_ERR_ARGS : LUSTRINE_OK;
}

extern "C" int lustrine_release_scratch(void) {
    DeviceScratch* const kept = device_scratch(false);
    cudaError_t e = cudaSuccess;
    if (kept && (e = cudaMemPoolTrimTo(kept->pool, 0)) != cudaSuccess) return lgb_cuda_status(e, "cudaMemPoolTrimTo");
    return LUSTRINE_OK;
}
