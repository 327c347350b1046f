// Device-side check of the wall function's small-integer operations (d3q19.cuh) against the general ones on
// the host: div_small for n = 1..75 over quotients of every size that float32 velocities give, sqrt_small for
// 0..12, int_double for -4096..4096.  Prints results compared and those whose bits differ.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include <cuda_runtime.h>
#include "../../water_flow_simulation_b200/csrc/d3q19.cuh"
using namespace wfs;

__global__ void divide(const double* p, int n, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y + 1;
    if (i < n) out[(size_t)(k - 1) * n + i] = div_small(p[i], k);
}
__global__ void integers(double* root, double* value)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= 12) root[i] = sqrt_small(i);
    if (i <= 8192) value[i] = int_double(i - 4096);
}

static long long compared = 0, differ = 0;
static void same(double a, double b)
{
    ++compared;
    differ += std::memcmp(&a, &b, sizeof a) != 0;
}

int main()
{
    constexpr int N = 20000, K = 75;
    std::mt19937_64 rng(5);
    std::uniform_real_distribution<double> mantissa(1.0, 2.0);
    std::vector<double> p{0.0, 0.1, 1.0 / 3.0, std::nextafter(1.0, 0.0), std::nextafter(75.0, 100.0)};
    while ((int)p.size() < N)                              // sums of float32 products with -5..5
        p.push_back(std::ldexp(mantissa(rng), (int)(rng() % 160) - 149) * (rng() % 2 ? 1.0 : -1.0));
    double *dp, *dq, *dr, *dv;
    cudaMalloc(&dp, N * sizeof(double));
    cudaMalloc(&dq, sizeof(double) * N * K);
    cudaMalloc(&dr, 13 * sizeof(double));
    cudaMalloc(&dv, 8193 * sizeof(double));
    cudaMemcpy(dp, p.data(), N * sizeof(double), cudaMemcpyHostToDevice);
    divide<<<dim3((N + 255) / 256, K), 256>>>(dp, N, dq);
    integers<<<(8193 + 255) / 256, 256>>>(dr, dv);
    std::vector<double> q((size_t)N * K), r(13), v(8193);
    cudaMemcpy(q.data(), dq, sizeof(double) * N * K, cudaMemcpyDeviceToHost);
    cudaMemcpy(r.data(), dr, 13 * sizeof(double), cudaMemcpyDeviceToHost);
    cudaMemcpy(v.data(), dv, 8193 * sizeof(double), cudaMemcpyDeviceToHost);
    if (cudaGetLastError() != cudaSuccess) return 1;
    for (int k = 0; k < K; ++k)
        for (int i = 0; i < N; ++i) same(q[(size_t)k * N + i], p[i] / (k + 1));
    for (int i = 0; i <= 12; ++i) same(r[i], std::sqrt((double)i));
    for (int i = 0; i <= 8192; ++i) same(v[i], (double)(i - 4096));
    std::printf("%lld %lld\n", compared, differ);
    return 0;
}
