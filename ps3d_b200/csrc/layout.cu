// layout.cu — conversion between the host's halo layout and the device's
// interior-only layout, done on the device so a host array crosses the bus
// in one contiguous copy.
//
// Host layout: Fortran bounds (1-2:nx+2, 1-2:ny+2, 1-2:nz+2), x fastest
// (main_module.f90:124-127).  Interior point (i, j, k) (0-based) sits at
// array index (i+2, j+2, k+2).  On download every halo point is the periodic
// copy of an interior point, as border_exchg_3D leaves it on one rank
// (parallel_mpi.f90:70-211); for p under a rigid lid the z ghost levels copy
// the nearest interior level instead (pressure_solver.f90:82-93).
#include "engine.h"

namespace ps3d {

// Both kernels move pairs of neighbouring points along x: nx is even and the
// halo is two points wide, so a pair never straddles the periodic seam and is
// 16-byte aligned on both sides.  Pairs are numbered over the whole array and
// split into (row, pair) and (level, row) by multiplications with 32-bit
// reciprocals; every thread has kLB pairs in flight.  Bound by HBM: 16 bytes
// a point (FP64), 19.4 us a download at 256x256x128, against 57.6 us with one
// point a thread and 64-bit divisions for every index.
constexpr int kLayoutThreads = 256, kLB = 4;

struct HaloDims {
    int nx, ny, nz;
    unsigned npairs;        // pairs moved: interior (from) or whole array (to)
    FastDiv row, lev;       // pairs per row, rows per level
};

template <typename T> struct pair2;
template <> struct pair2<double> { using type = double2; };
template <> struct pair2<float> { using type = float2; };

template <typename T>
__global__ void __launch_bounds__(kLayoutThreads) k_from_halo(const double* __restrict__ h, T* __restrict__ dst,
                                                              const HaloDims d) {
    using T2 = typename pair2<T>::type;
    const unsigned stride = gridDim.x * kLayoutThreads;
    for (unsigned t0 = blockIdx.x * kLayoutThreads + threadIdx.x; t0 < d.npairs; t0 += kLB * stride) {
        double2 v[kLB];
#pragma unroll
        for (int q = 0; q < kLB; ++q) {
            const unsigned t = t0 + q * stride;
            if (t < d.npairs) {
                const unsigned r = fdiv(t, d.row), i = t - r * d.row.d;
                const unsigned k = fdiv(r, d.lev), j = r - k * d.lev.d;
                v[q] = __ldg(reinterpret_cast<const double2*>(h + 2 * (i + 1)) +
                             ((long)(k + 2) * (d.ny + 4) + j + 2) * ((d.nx + 4) / 2));
            }
        }
#pragma unroll
        for (int q = 0; q < kLB; ++q) {
            const unsigned t = t0 + q * stride;
            if (t < d.npairs) {
                T2 o;
                o.x = (T)v[q].x; o.y = (T)v[q].y;
                reinterpret_cast<T2*>(dst)[t] = o;
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kLayoutThreads) k_to_halo(const T* __restrict__ src, double* __restrict__ h,
                                                            const HaloDims d, int pghost) {
    using T2 = typename pair2<T>::type;
    const unsigned stride = gridDim.x * kLayoutThreads;
    // halos of up to two points around a grid of at least two: one wrap a side
    auto wr = [](int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); };
    for (unsigned t0 = blockIdx.x * kLayoutThreads + threadIdx.x; t0 < d.npairs; t0 += kLB * stride) {
        T2 v[kLB];
#pragma unroll
        for (int q = 0; q < kLB; ++q) {
            const unsigned t = t0 + q * stride;
            if (t < d.npairs) {
                const unsigned r = fdiv(t, d.row), x = t - r * d.row.d;
                const unsigned z = fdiv(r, d.lev), y = r - z * d.lev.d;
                const int i = wr(2 * (int)x - 2, d.nx), j = wr((int)y - 2, d.ny);
                const int k = pghost ? min(max((int)z - 2, 0), d.nz - 1) : wr((int)z - 2, d.nz);
                v[q] = __ldg(reinterpret_cast<const T2*>(src + ((long)k * d.ny + j) * d.nx + i));
            }
        }
#pragma unroll
        for (int q = 0; q < kLB; ++q) {
            const unsigned t = t0 + q * stride;
            if (t < d.npairs) reinterpret_cast<double2*>(h)[t] = make_double2((double)v[q].x, (double)v[q].y);
        }
    }
}

static int grid_of(unsigned n) {
    return (int)std::min<unsigned>((n + kLayoutThreads - 1) / kLayoutThreads, 148u * 8);   // a wave of full SMs
}
static HaloDims dims_of(int nx, int ny, int nz, int halo) {
    HaloDims d;
    d.nx = nx; d.ny = ny; d.nz = nz;
    d.row = make_fastdiv((unsigned)(nx + halo) / 2);
    d.lev = make_fastdiv((unsigned)(ny + halo));
    d.npairs = (unsigned)(nx + halo) / 2 * (unsigned)(ny + halo) * (unsigned)(nz + halo);
    return d;
}

cudaError_t launch_from_halo(const double* h_dev, void* dst, int nx, int ny, int nz, bool f32, cudaStream_t s) {
    const HaloDims d = dims_of(nx, ny, nz, 0);
    if (f32) k_from_halo<float><<<grid_of(d.npairs), kLayoutThreads, 0, s>>>(h_dev, (float*)dst, d);
    else k_from_halo<double><<<grid_of(d.npairs), kLayoutThreads, 0, s>>>(h_dev, (double*)dst, d);
    return cudaGetLastError();
}
cudaError_t launch_to_halo(const void* src, double* h_dev, int nx, int ny, int nz, bool pghost, bool f32,
                           cudaStream_t s) {
    const HaloDims d = dims_of(nx, ny, nz, 4);
    if (f32) k_to_halo<float><<<grid_of(d.npairs), kLayoutThreads, 0, s>>>((const float*)src, h_dev, d, pghost ? 1 : 0);
    else k_to_halo<double><<<grid_of(d.npairs), kLayoutThreads, 0, s>>>((const double*)src, h_dev, d, pghost ? 1 : 0);
    return cudaGetLastError();
}

}  // namespace ps3d
