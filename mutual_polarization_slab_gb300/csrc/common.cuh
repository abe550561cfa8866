// Shared helpers for the GB300 spectral-Ewald kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/mps_gb300.h"

#define MPS_PI 3.14159265358979323846

namespace mps {

constexpr int kWarp = 32;

// Status plumbing: CUDA errors become MPS_CUDA_ERR, never exceptions.
#define MPS_CUDA_TRY(expr)                                   \
    do {                                                     \
        cudaError_t _e = (expr);                             \
        if (_e != cudaSuccess) {                             \
            mps::set_last_error(_e, #expr, __FILE__, __LINE__); \
            return MPS_CUDA_ERR;                             \
        }                                                    \
    } while (0)

#define MPS_LAUNCH_CHECK()                                   \
    do {                                                     \
        mps::count_launch();                                 \
        cudaError_t _e = cudaGetLastError();                 \
        if (_e != cudaSuccess) {                             \
            mps::set_last_error(_e, "kernel launch", __FILE__, __LINE__); \
            return MPS_CUDA_ERR;                             \
        }                                                    \
    } while (0)

void set_last_error(cudaError_t e, const char *what, const char *file, int line);
void count_launch();
// Kernels enqueued while this thread captures a CUDA graph are not launches:
// between capture_count_begin and capture_count_end count_launch counts them
// for the caller (the launches per graph execution) instead of the process total.
void capture_count_begin();
long long capture_count_end();
void add_launches(long long k);

// A device copy of bytes of host memory (cudaMalloc), complete on return, whatever stream reads it next: a plain
// cudaMemcpy from pageable memory may return with the device's write still pending on the legacy stream, which no
// non-blocking stream waits for.  MPS_NO_MEMORY or MPS_CUDA_ERR (and no copy) otherwise.
int upload_table(const void *host, size_t bytes, void **out);

inline unsigned grid_for(int64_t work, int block, int64_t cap = 152 * 32) {
    int64_t g = (work + block - 1) / block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (unsigned)g;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One float (or two or four, aligned) from global to shared memory without a register in between: a staging loop issues
// all its loads at once (copy_async_wait before the barrier that publishes them).
__device__ __forceinline__ void copy_async(float *smem, const float *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void copy_async(float2 *smem, const float2 *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void copy_async(float4 *smem, const float4 *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// C sums over the warp (C <= 32), one to a lane: each halving of the warp halves the values a lane still carries, so C
// sums take about C + 4 shuffles and additions instead of 5 C, and what follows (the conversion to float64, the
// scaling, the store) is one instruction for all of them: on GB300 a float64 instruction of a warp, a conversion too,
// costs the same for one active lane as for 32.  Each sum adds the same pairs in the same order as warp_sum.
// warp_sums_index tells which sum a lane holds (-1: none, or the same as another lane).
template <typename T>
__device__ __forceinline__ T lane_xor(T v, int o) {
    return __shfl_xor_sync(0xffffffffu, v, o);
}

template <int C, int O = 16, typename T>
__device__ __forceinline__ T warp_sums(const T (&v)[C], int lane) {
    if constexpr (O == 0) {
        static_assert(C == 1, "more sums than lanes");
        return v[0];
    } else {
        constexpr int H = (C + 1) / 2;
        const bool hi = lane & O;
        T u[H];
#pragma unroll
        for (int k = 0; k < H; ++k) {
            const T up = v[k + H < C ? k + H : k];
            u[k] = (hi ? up : v[k]) + lane_xor(hi ? v[k] : up, O);
        }
        return warp_sums<H, O / 2>(u, lane);
    }
}

template <int C, int O = 16>
__device__ __forceinline__ int warp_sums_index(int lane) {
    if constexpr (O == 0) {
        return 0;
    } else {
        constexpr int H = (C + 1) / 2;
        const int i = warp_sums_index<H, O / 2>(lane);
        if (C == 1) return (lane & O) ? -1 : i;
        const int k = i + ((lane & O) ? H : 0);
        return i < 0 || k >= C ? -1 : k;
    }
}

// Four sums over the warp in 6 additions instead of 20 (float64 additions are what a warp's reductions cost on GB300):
// halves of the warp take half of the values each.  Lane 0 returns a's sum, lane 8 b's, lane 16 c's, lane 24 d's.
template <typename T>
__device__ __forceinline__ T warp_sum4(T a, T b, T c, T d, int lane) {
    const bool hi = lane & 16, mid = lane & 8;
    T x = (hi ? c : a) + __shfl_xor_sync(0xffffffffu, hi ? a : c, 16);
    T y = (hi ? d : b) + __shfl_xor_sync(0xffffffffu, hi ? b : d, 16);
    T z = (mid ? y : x) + __shfl_xor_sync(0xffffffffu, mid ? x : y, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    return z;
}

// numpy float mod: result carries the sign of the divisor.
__device__ __forceinline__ double np_mod(double a, double b) {
    double r = fmod(a, b);
    if (r != 0.0) {
        if ((b < 0.0) != (r < 0.0)) r = __dadd_rn(r, b);
    } else {
        r = copysign(0.0, b);
    }
    return r;
}

// Integer frequency of unshifted FFT index i with the fftshift convention
// k in [-ceil((n-1)/2), floor((n-1)/2)] (the Nyquist bin of an even axis is negative).
__device__ __forceinline__ int fft_freq(int i, int n) {
    int c = n / 2;
    int p = i + c;
    if (p >= n) p -= n;
    return p - c;
}

// Quarter of an R2C half spectrum (Nx/2+1, Ny, Nz; x fastest): the points with
// iy <= Ny/2 and iz <= Nz/2.  Index N - i has frequency -fft_freq(i, N), so a
// coefficient that depends on k only through kx^2, ky^2, kz^2 is the same at
// (ix, +-iy, +-iz); mirror_points calls f(linear index, sy, sz) once for each
// distinct such point, sy / sz = -1 where the y / z index was mirrored.
struct HalfQuarter {
    int Nxh, Ny, Nz, Nyq, Nzq;
    __host__ __device__ explicit HalfQuarter(const int N[3])
        : Nxh(N[0] / 2 + 1), Ny(N[1]), Nz(N[2]), Nyq(N[1] / 2 + 1), Nzq(N[2] / 2 + 1) {}
    __host__ __device__ int64_t size() const { return (int64_t)Nxh * Nyq * Nzq; }
    __device__ void point(int64_t t, int *ix, int *iy, int *iz) const {
        *ix = (int)(t % Nxh);
        *iy = (int)((t / Nxh) % Nyq);
        *iz = (int)(t / ((int64_t)Nxh * Nyq));
    }
};

template <class F>
__device__ __forceinline__ void mirror_points(const HalfQuarter &q, int ix, int iy, int iz, F &&f) {
    const int my = (q.Ny - iy) % q.Ny, mz = (q.Nz - iz) % q.Nz;
    const int na = my == iy ? 1 : 2, nb = mz == iz ? 1 : 2;
    for (int a = 0; a < na; ++a)
        for (int b = 0; b < nb; ++b)
            f(((int64_t)(b ? mz : iz) * q.Ny + (a ? my : iy)) * q.Nxh + ix, a ? -1 : 1, b ? -1 : 1);
}

// Rows of stacked grids taken two at a time as the real and the imaginary part of one complex line.  No pair reaches
// from one grid into the next (a grid with an odd number of rows ends with a row by itself): the two rows share a
// rounding error, and an infinity or NaN, and grids of different vectors have nothing to do with each other.
struct RowPairs {
    unsigned rows, pairs;   // of one grid
    __host__ __device__ explicit RowPairs(int64_t grid_rows)
        : rows((unsigned)grid_rows), pairs((unsigned)((grid_rows + 1) / 2)) {}
    // The lines from pair p0 on: first row of the first one, and of line l after that; two = it has a second row.
    struct Lines {
        unsigned q0, pairs;
        bool odd;
        int64_t row0;
        __device__ __forceinline__ unsigned row(unsigned l, bool *two) const {
            *two = true;
            if (!odd) return 2 * l;
            const unsigned c = (q0 + l) / pairs;
            *two = q0 + l - c * pairs != pairs - 1;
            return 2 * l - c;
        }
    };
    __device__ __forceinline__ Lines from(int64_t p0) const {
        const bool odd = rows & 1;
        const int64_t c0 = odd ? p0 / pairs : 0;
        return {(unsigned)(p0 - c0 * pairs), pairs, odd, 2 * p0 - c0};
    }
};

__device__ __forceinline__ int64_t wrap_index(int64_t i, int64_t n) {
    int64_t r = i % n;
    return r < 0 ? r + n : r;
}

// Exclusive scan of int64 counts (n may be large); tmp is scan_workspace() bytes.
size_t scan_workspace(int64_t n);
int exclusive_scan_i64(const int64_t *in, int64_t *out, int64_t n, void *tmp, cudaStream_t s);
int exclusive_scan_i32_to_i64(const int32_t *in, int64_t *out, int64_t n, void *tmp, cudaStream_t s);

}  // namespace mps
