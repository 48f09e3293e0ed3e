// Stand-in for the CUDA runtime under the launch functions of the step's kernels: devices with
// function attributes of their own, launches that are checked and not made.
#include <cuda_runtime_api.h>

#include <map>
#include <utility>

namespace {
int device = 0;
std::map<std::pair<int, const void *>, int> shared_limit;   // opt-in, per device and kernel
int launches = 0, refused = 0;
unsigned last_grid = 0, last_block = 0;
}  // namespace

extern "C" {
void fake_set_device(int d) { device = d; }
int fake_launches() { return launches; }
int fake_refused() { return refused; }
unsigned fake_last_grid() { return last_grid; }
unsigned fake_last_block() { return last_block; }

cudaError_t cudaGetDevice(int *d) {
    *d = device;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int value) {
    shared_limit[{device, f}] = value;
    return cudaSuccess;
}
// three blocks fit an SM of device 0, two one of device 1
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = device == 0 ? 3 : 2;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
    launches++;
    last_grid = c->gridDim.x;
    last_block = c->blockDim.x;
    const auto it = shared_limit.find({device, f});
    if (c->dynamicSmemBytes > 48 * 1024 && (it == shared_limit.end() || (size_t)it->second < c->dynamicSmemBytes)) {
        refused++;
        return cudaErrorInvalidValue;
    }
    return cudaSuccess;
}

// what nvcc's registration and <<<>>> stubs call
void **__cudaRegisterFatBinary(void *) {
    static void *handle = nullptr;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction() {}
int __cudaGetKernel(const void **kernel, const void *f) {
    *kernel = f;
    return 0;
}
unsigned __cudaPushCallConfiguration() { return 0; }
unsigned __cudaPopCallConfiguration() { return 0; }
int __cudaLaunchKernel() { return 0; }
}
