// A refused chained launch is reported once: the runtime's error state is clear
// afterwards, and the next launch and its cudaGetLastError() succeed.

#include <cstdio>

#include "launch.cuh"

__global__ void set_kernel(int* out) {
    skb::grid_wait();
    *out = 1;
}

int main() {
    int* out = nullptr;
    int value = 0;
    if (cudaMalloc(&out, sizeof(int)) != cudaSuccess) return std::puts("cudaMalloc failed"), 1;
    // The host refuses a block of 2048 threads.
    if (skb::launch_chained(set_kernel, dim3(1), 2048, 0, nullptr, out) == cudaSuccess)
        return std::puts("the launch was not refused"), 1;
    if (cudaPeekAtLastError() != cudaSuccess) return std::puts("the refused launch's error is still standing"), 1;
    if (skb::launch_chained(set_kernel, dim3(1), 1, 0, nullptr, out) != cudaSuccess)
        return std::puts("a valid launch failed"), 1;
    if (cudaGetLastError() != cudaSuccess) return std::puts("an old error was reported again"), 1;
    if (cudaMemcpy(&value, out, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess || value != 1)
        return std::puts("wrong result"), 1;
    cudaFree(out);
    std::puts("ok");
    return 0;
}
