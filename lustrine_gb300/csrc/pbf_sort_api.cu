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
#include <atomic>
#include <cstdio>
#include <mutex>

#include "lustrine_gb300.h"
#include "pbf_context.h"
#include "pbf_kernels.h"

using namespace lgb;

namespace {

constexpr unsigned long long SCRATCH_KEPT = 128ull << 20;
constexpr int kMaxDevices = 64;
constexpr int kWords = 64;

std::mutex g_lock;
cudaMemPool_t g_pool[kMaxDevices] = {};
int* g_words = nullptr;  // page-locked, kWords ints
std::atomic<bool> g_word_used[kWords];

// The current device's scratch pool, or nullptr (the default pool serves).
cudaMemPool_t scratch_pool() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_lock);
    if (!g_pool[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        unsigned long long keep = SCRATCH_KEPT;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaGetLastError();
            cudaMemPoolDestroy(pool);
            return nullptr;
        }
        g_pool[dev] = pool;
    }
    return g_pool[dev];
}

// A page-locked word of this call's own, zero; -1 when none is free.
int take_word() {
    {
        std::lock_guard<std::mutex> lock(g_lock);
        if (!g_words && cudaHostAlloc((void**)&g_words, kWords * sizeof(int),
                                      cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
            cudaGetLastError();
            g_words = nullptr;
            return -1;
        }
    }
    for (int k = 0; k < kWords; k++) {
        bool free = false;
        if (g_word_used[k].compare_exchange_strong(free, true)) {
            *(volatile int*)&g_words[k] = 0;
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
    const size_t bytes = counting_sort_scratch_ints(n, C) * sizeof(int);
    int* scratch = nullptr;
    cudaMemPool_t pool = scratch_pool();
    cudaError_t e = pool ? cudaMallocFromPoolAsync((void**)&scratch, bytes, pool, st)
                         : cudaMallocAsync((void**)&scratch, bytes, st);
    if (e != cudaSuccess) return lgb_cuda_status(e, "cudaMallocAsync");
    CountingSortScratch w = counting_sort_scratch(scratch, n, C);
    int bad = 0;
    const int word = take_word();
    // the histogram and the status word behind it start at zero
    e = cudaMemsetAsync(w.count, 0, ((size_t)C + 1) * sizeof(int), st);
    if (e == cudaSuccess) {
        int* const device_status = w.status;
        if (word >= 0) w.status = &g_words[word];
        const cudaError_t before = cudaPeekAtLastError();  // an earlier call's error is not this one's
        launch_counting_sort(keys, n, C, w, counts, sorted_indices, st);
        if (before == cudaSuccess) e = cudaPeekAtLastError();
        if (word < 0 && e == cudaSuccess)
            e = cudaMemcpyAsync(&bad, device_status, sizeof(int), cudaMemcpyDeviceToHost, st);
    }
    const cudaError_t e1 = cudaFreeAsync(scratch, st);
    const cudaError_t e2 = cudaStreamSynchronize(st);
    if (word >= 0) {
        bad = *(volatile int*)&g_words[word];
        g_word_used[word].store(false);
    }
    if (e == cudaSuccess) e = e2 != cudaSuccess ? e2 : e1;
    if (e != cudaSuccess) return lgb_cuda_status(e, "counting_sort");
    return bad ? LUSTRINE_ERR_ARGS : LUSTRINE_OK;
}

extern "C" int lustrine_release_scratch(void) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return lgb_cuda_status(e, "cudaGetDevice");
    cudaMemPool_t pool = nullptr;
    if (dev >= 0 && dev < kMaxDevices) {
        std::lock_guard<std::mutex> lock(g_lock);
        pool = g_pool[dev];
    }
    if (pool && (e = cudaMemPoolTrimTo(pool, 0)) != cudaSuccess) return lgb_cuda_status(e, "cudaMemPoolTrimTo");
    return LUSTRINE_OK;
}
