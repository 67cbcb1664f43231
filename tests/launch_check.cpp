// launch_chained against a stand-in of the CUDA runtime whose launches fail or
// succeed on request and leave the failure's code standing, as the runtime does.

#include <cstddef>
#include <cstdio>

#define __device__
#define __forceinline__ inline
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidConfiguration = 9 };
enum { cudaLaunchAttributeProgrammaticStreamSerialization = 6 };
using cudaStream_t = void*;
struct dim3 {
    unsigned x = 1, y = 1, z = 1;
    dim3(unsigned x_ = 1, unsigned y_ = 1, unsigned z_ = 1) : x(x_), y(y_), z(z_) {}
};
struct cudaLaunchAttribute {
    int id;
    struct { int programmaticStreamSerializationAllowed; } val;
};
struct cudaLaunchConfig_t {
    dim3 gridDim, blockDim;
    size_t dynamicSmemBytes;
    cudaStream_t stream;
    cudaLaunchAttribute* attrs;
    unsigned numAttrs;
};

static cudaError_t standing = cudaSuccess;
static cudaError_t cudaGetLastError() {
    const cudaError_t err = standing;
    standing = cudaSuccess;
    return err;
}
template <typename... P>
static cudaError_t cudaLaunchKernelEx(const cudaLaunchConfig_t* config, void (*kernel)(P...), P... args) {
    if (config->blockDim.x > 1024) return standing = cudaErrorInvalidConfiguration;
    kernel(args...);
    return cudaSuccess;
}

#include "launch.cuh"

static void set(int* out) { *out = 1; }

int main() {
    int value = 0;
    if (skb::launch_chained(set, dim3(1), 2048, 0, nullptr, &value) != cudaErrorInvalidConfiguration)
        return std::puts("the refusal was not returned"), 1;
    if (standing != cudaSuccess) return std::puts("the refused launch's error is still standing"), 1;
    if (skb::launch_chained(set, dim3(1), 32, 0, nullptr, &value) != cudaSuccess || value != 1)
        return std::puts("a valid launch failed"), 1;
    std::puts("ok");
    return 0;
}
