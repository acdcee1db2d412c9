// The CUDA runtime of launch_shapes.cu: launches are recorded, not made.
struct Launch {
    const void* kernel;
    unsigned grid, block;
    int count;
};
struct Config {  // the start of cudaLaunchConfig_t
    unsigned grid[3], block[3];
};

extern "C" {
Launch g_launch = {};
int cudaLaunchKernelExC(const Config* c, const void* kernel, void**) {
    g_launch = {kernel, c->grid[0], c->block[0], g_launch.count + 1};
    return 0;
}
int __cudaLaunchKernel() { return 0; }
int cudaLaunchKernel() { return 0; }
int __cudaGetKernel(void** k, const void* f) { return *k = (void*)f, 0; }
int __cudaPopCallConfiguration() { return 0; }
unsigned __cudaPushCallConfiguration() { return 0; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction() {}
void __cudaRegisterVar() {}
int cudaMemsetAsync(void*, int, unsigned long, void*) { return 0; }
int cudaPointerGetAttributes() { return 0; }
int cudaGetLastError() { return 0; }
}
