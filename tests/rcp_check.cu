// Checks rcp_nr (evp_newton.cu's reciprocal, in evp_vox.cuh) against the correctly rounded division.
#include "evp_vox.cuh"

#include <cstdio>

__global__ void worst(unsigned long long seed, int n, double* out) {
    unsigned long long s = seed + 0x9E3779B97F4A7C15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1);
    double w = 0.0;
    for (int i = 0; i < n; i++) {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        const int e = (int)((s >> 53) % 1800ull) - 900;  // normal x with a normal reciprocal
        const double x = ldexp(1.0 + (double)(s >> 12) * 0x1p-52, e) * ((i & 1) ? -1.0 : 1.0);
        const double r = __drcp_rn(x);
        w = fmax(w, fabs(evp::rcp_nr(x) - r) / fabs(r));
    }
    out[blockIdx.x * blockDim.x + threadIdx.x] = w;
}

int main() {
    constexpr int T = 64 * 128;
    static double h[T];
    double* d;
    cudaMalloc(&d, sizeof(h));
    worst<<<64, 128>>>(20240607ull, 2000, d);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    double w = 0.0;
    for (double x : h) w = x > w ? x : w;
    std::printf("%.17g\n", w);
    return 0;
}
