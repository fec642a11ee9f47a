// Every FP32 uniform of [0.5, 1], and small ones, through the packed Box-Muller pair: results that
// are not finite, and results that differ from the one-sample form's.
#include "scphd_kernels.cuh"

namespace {

__global__ void k_check(unsigned long long* bad, unsigned n, unsigned step, unsigned first) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t wa0 = first + step * i, wa1 = ~0u - i, wb0 = 2654435761u * i, wb1 = 40503u * i + 12345u;
    scphd::F2 z0, z1;
    scphd::normals_pair(wa0, wb0, wa1, wb1, z0, z1);
    const float got[4] = {scphd::f2_lo(z0), scphd::f2_lo(z1), scphd::f2_hi(z0), scphd::f2_hi(z1)};
    float want[4];
    scphd::Pair<float>::two(wa0, wb0, want[0], want[1]);
    scphd::Pair<float>::two(wa1, wb1, want[2], want[3]);
    for (int k = 0; k < 4; ++k) {
        if (!isfinite(got[k])) atomicAdd(bad, 1ull);
        if (got[k] != want[k]) atomicAdd(bad + 1, 1ull);
    }
}

}  // namespace

extern "C" int check_normals(unsigned long long out[2]) {
    unsigned long long* bad = nullptr;
    if (cudaMalloc(&bad, 16) != cudaSuccess) return 1;
    cudaMemset(bad, 0, 16);
    // words from 2^31 up in steps of 64: all 2^23 values of [0.5, 1) and those that round to 1
    const unsigned many = 1u << 25, few = 1u << 20;
    k_check<<<many / 256, 256>>>(bad, many, 64u, 0x80000000u);
    k_check<<<few / 256, 256>>>(bad, few, 1u, 0u);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaMemcpy(out, bad, 16, cudaMemcpyDeviceToHost);
    cudaFree(bad);
    return e != cudaSuccess;
}
