// Every non-negative float through both forms of inv_r_of (infinity included):
// prints how many differ, with one of them.
#include <cstdio>

#include "pbf_device.cuh"

__global__ void k_compare(unsigned long long* differing, unsigned* one) {
    const unsigned b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > 0x7f800000u) return;
    const float r2 = __uint_as_float(b);
    if (__float_as_uint(lgb::inv_r_of<true>(r2)) != __float_as_uint(lgb::inv_r_of<false>(r2))) {
        atomicAdd(differing, 1ull);
        *one = b;
    }
}

int main() {
    struct {
        unsigned long long differing;
        unsigned one;
    } *d = nullptr, h = {};
    cudaError_t e = cudaMalloc((void**)&d, sizeof(h));
    if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(h));
    k_compare<<<0x7f800000u / 256 + 1, 256>>>(&d->differing, &d->one);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
    std::printf("%s, %llu differ, bits %08x\n", cudaGetErrorString(e), h.differing, h.one);
    return e != cudaSuccess || h.differing != 0;
}
