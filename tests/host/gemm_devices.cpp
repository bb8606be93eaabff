// Launches of the tensor-core GEMM's host code (mlp_gemm.cu) against a fake CUDA runtime with two
// devices: a kernel's shared-memory limit belongs to the device it was raised on, and a launch
// that asks for more than its device allows fails, as on a GPU.  Nothing runs on a device.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <map>
#include <string>
#include <utility>

#include "../../tdp1375_b200/csrc/mlp.h"

namespace {
int gDevice = 0, gLaunches = 0;
bool gRefuse = false;  // cudaFuncSetAttribute fails
cudaError_t gLast = cudaSuccess;
std::map<std::pair<int, const void *>, int> gLimit;  // (device, kernel) -> dynamic shared memory
dim3 gGrid, gBlock;
size_t gShared = 0;
cudaStream_t gStream = nullptr;

CUresult encode(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    return CUDA_SUCCESS;
}
}  // namespace

extern "C" {
void **__cudaRegisterFatBinary(void *) {
    static void *handle = nullptr;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t stream) {
    gGrid = grid, gBlock = block, gShared = shared, gStream = stream;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *shared, void *stream) {
    *grid = gGrid, *block = gBlock, *shared = gShared;
    *static_cast<cudaStream_t *>(stream) = gStream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *kernel, dim3, dim3, void **, size_t shared, cudaStream_t) {
    const auto it = gLimit.find({gDevice, kernel});
    if (shared > (it == gLimit.end() ? 48u << 10 : (size_t)it->second)) return gLast = cudaErrorInvalidValue;
    ++gLaunches;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *kernel, cudaFuncAttribute, int value) {
    if (gRefuse) return cudaErrorInvalidDeviceFunction;
    gLimit[{gDevice, kernel}] = value;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *device) {
    *device = gDevice;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = gLast;
    gLast = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake runtime error"; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **fn, unsigned long long, cudaDriverEntryPointQueryResult *q) {
    *fn = reinterpret_cast<void *>(&encode);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
}

int main() {
    alignas(16) static unsigned char buffer[16];
    auto gemm = [&](int device, int fp32) {
        gDevice = device;
        std::string err;
        const int rc = tdp::mlp::gemm_bf16(buffer, buffer, 256, 256, 64, nullptr, 0, buffer, fp32, 256,
                                           reinterpret_cast<int *>(buffer), nullptr, err);
        if (rc != 0) std::printf("device %d: %s\n", device, err.c_str());
        return rc == 0;
    };
    if (!gemm(0, 0)) return 1;
    // a failed set-up is reported and tried again by the next call
    gRefuse = true;
    if (gemm(1, 0)) return 2;
    gRefuse = false;
    const bool ok = gemm(1, 0) && gemm(0, 1) && gemm(1, 1);
    std::printf("launches %d\n", gLaunches);
    return ok && gLaunches == 4 ? 0 : 3;
}
