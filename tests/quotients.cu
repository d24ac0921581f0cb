// How often divide_neg differs from a division, over random operands: host and
// device builds of the same header.
#include <cuda_runtime.h>
#include <cmath>
#include <cstring>
#include "divide.cuh"

using u64 = unsigned long long;

__host__ __device__ static u64 mix(u64 z) {   // splitmix64
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
template <typename A, typename B> __host__ __device__ static A as(B b) {
    A a;
    memcpy(&a, &b, sizeof a);
    return a;
}
// a positive double with a random mantissa and an exponent in [-e, e]
__host__ __device__ static double positive(u64 h, int e) {
    return as<double>((u64)(1023 - e + (int)(mix(h) % (2 * e + 1))) << 52 | (h & 0xfffffffffffffull));
}
template <typename R> __host__ __device__ static bool same(R a, R b) { return (a != a && b != b) || (a == b && signbit(a) == signbit(b)); }

// operand i: FP32 takes every bit pattern, over ordinary and extreme ks; FP64
// 2^-200 .. 2^200 over the same, zeros, infinities and NaNs among them
__host__ __device__ static bool differs(int fp32, u64 i, u64 seed) {
    const u64 h = mix(seed + 2 * i), g = mix(seed + 2 * i + 1);
    if (fp32) {
        const double ks = i % 8 == 0 ? positive(h, 1000) : positive(h, 60);
        const float f = as<float>((unsigned)g);
        const float2 q = ps3d::divide_neg<float>(make_float2(f, f), ks);
        const float want = (float)(-(double)f / ks);
        return !same(q.x, want) || !same(q.y, want);
    }
    const double ks = i % 8 == 0 ? positive(h, 200) : positive(h, 40);
    double f = positive(g, i % 8 == 0 ? 200 : 40) * (g >> 63 ? -1.0 : 1.0);
    if (i % 64 == 1) f = i & 64 ? 0.0 : -0.0;
    if (i % 64 == 2) f = i & 64 ? INFINITY : -INFINITY;
    if (i % 64 == 3) f = NAN;
    const double2 q = ps3d::divide_neg<double>(make_double2(f, f), ks);
    const double want = -f / ks;
    return !same(q.x, want) || !same(q.y, want);
}

__global__ static void k_count(int fp32, u64 n, u64 seed, u64* bad) {
    u64 c = 0;
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) c += differs(fp32, i, seed);
    if (c) atomicAdd(bad, c);
}

// operands that differ among n; negative: a CUDA error
extern "C" long long quotients_differ(int device, int fp32, u64 n, u64 seed) {
    u64 bad = 0;
    if (!device) {
        for (u64 i = 0; i < n; ++i) bad += differs(fp32, i, seed);
        return (long long)bad;
    }
    u64* d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof *d);
    if (!e) e = cudaMemset(d, 0, sizeof *d);
    if (!e) k_count<<<148 * 8, 256>>>(fp32, n, seed, d);
    if (!e) e = cudaGetLastError();
    if (!e) e = cudaMemcpy(&bad, d, sizeof *d, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e ? -(long long)e : (long long)bad;
}
