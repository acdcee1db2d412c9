// The counting sort's entry points over a CUDA runtime made of the functions
// below, whose k-th kernel launch fails and, as the real one, leaves its error
// pending: every call must return an error, launch nothing after the failure,
// and not take an error that was pending before it for its own.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

enum cudaError { OK = 0, MEM = 2, BAD = 9 };
int g_launches = 0, g_fail_at = -1, g_pending = 0, g_after = 0;
static int launch() {
    if (g_fail_at >= 0 && g_launches > g_fail_at) g_after++;
    return g_launches++ == g_fail_at ? (g_pending = BAD) : 0;
}
int lgb_cuda_status(cudaError e, const char*) { return e == MEM ? 7 : 6; }

extern "C" {
int lustrine_counting_sort(int*, const int*, size_t, size_t, int*, void*);
int lustrine_counting_sort_noalloc(int*, const int*, size_t, size_t, int*, void*);

int cudaLaunchKernelExC(const void*, const void*, void**) { return launch(); }
int __cudaLaunchKernel() { return launch(); }
int cudaLaunchKernel() { return launch(); }
int __cudaGetKernel(void** k, const void* f) { return *k = (void*)f, 0; }
int __cudaPopCallConfiguration() { return 0; }
unsigned __cudaPushCallConfiguration() { return 0; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction() {}
void __cudaRegisterVar() {}
int cudaGetSymbolAddress(void** p, const void*) { return *p = malloc(64 << 20), 0; }
int cudaGetDevice(int* d) { return *d = 0, 0; }
int cudaFree(void*) { return 0; }
int cudaFreeAsync(void* p, void*) { return free(p), 0; }
int cudaMallocAsync(void** p, size_t n, void*) { return *p = malloc(n), 0; }
int cudaMallocFromPoolAsync(void** p, size_t n, void*, void*) { return *p = malloc(n), 0; }
int cudaMemPoolCreate(void** p, const void*) { return *p = &g_pending, 0; }
int cudaMemPoolDestroy(void*) { return 0; }
int cudaMemPoolSetAttribute(void*, int, void*) { return 0; }
int cudaMemPoolTrimTo(void*, size_t) { return 0; }
int cudaHostAlloc(void** p, size_t n, unsigned) { return *p = calloc(1, n), 0; }
int cudaPointerGetAttributes() { return 0; }
int cudaMemcpyAsync(void* d, const void*, size_t, int, void*) { return *(int*)d = 0; }
int cudaMemsetAsync(void*, int, size_t, void*) { return 0; }
int cudaStreamSynchronize(void*) { return 0; }
int cudaPeekAtLastError() { return g_pending; }
int cudaGetLastError() { int e = g_pending; return g_pending = 0, e; }
int cuCtxGetIdFake(void*, unsigned long long* id) { return *id = 1, 0; }
int cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long, int* q) {
    return *f = KNOWN_CONTEXT ? (void*)cuCtxGetIdFake : nullptr, *q = 0;
}
}

int main() {
    static int counts[50000], keys[1000], order[1000];
    int bad = 0;
    for (auto sort : {lustrine_counting_sort, lustrine_counting_sort_noalloc})
        for (int off : {0, 1})  // both scans
            for (size_t n : {(size_t)0, (size_t)1000}) {
                auto call = [&](int fail_at) {
                    g_launches = g_after = 0;
                    g_fail_at = fail_at;
                    return sort(counts + off, keys, n, 40000, order, nullptr);
                };
                const int all = (call(-1), g_launches);
                for (int k = -1; k < all; k++)
                    for (int again = 0; again < 3; again++) {
                        const int rc = call(k);
                        if ((rc != 0) != (k >= 0) || g_after || (k < 0 && g_launches != all)) {
                            std::printf("launch %d of %d, n %zu, call %d: status %d, %d after it\n", k, all, n, again, rc,
                                        g_after);
                            bad = 1;
                        }
                    }
                if (all < 2) bad = 1;
            }
    return bad;
}
