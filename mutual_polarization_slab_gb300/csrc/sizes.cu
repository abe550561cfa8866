// Polydisperse dipole operator (spheres of different radii; the MATLAB variant
// Capacitance_Sizes, cited CS/).
//
//   real space   dielectric 3/(4 pi a^3 (eps - 1)), self value of the (a_i, a_i)
//                coupling, pair couplings of the two radii (CS/RealSpace.m:18-76)
//                either interpolated from the per-radius-pair tables of
//                CS/RealSpaceTable.m or evaluated in closed form at the exact
//                separation (continuous radii)
//   wave space   the dipoles are spread as charges onto ONE scalar grid with the
//                sphere kernel K(d) r-hat.p (CS/Spread.m:39-72), scaled by
//                exp(-(1-eta) q^2 / 4 xi^2) / q^2 (CS/Scale.m:16-21; even in q, so
//                the half-spectrum real transforms are exact), and contracted with
//                prod(h) sum K(d) r-hat (CS/Contract.m:39-73)
//
// The kernel values K(d)/d of every particle's P^3 stencil are computed once
// per system; the spread and contract rebuild r = node - x from the particle's
// base offset.
#include <math.h>

#include <cstdlib>

#include "sizes.cuh"

namespace mps {

// ---------------------------------------------------------------------------
// Couplings (CS/RealSpaceTable.m:34-146), written with shared subexpressions.
// ---------------------------------------------------------------------------
__host__ __device__ inline void cs_couplings(double r, double ai, double aj, double xi, double *perp, double *para) {
    const double pi = MPS_PI;
    const double sp3 = pi * sqrt(pi);
    const double x2 = xi * xi, x4 = x2 * x2, x6 = x4 * x2;
    const double s = ai + aj, d = ai - aj;
    const double ai2 = ai * ai, aj2 = aj * aj, ai3 = ai2 * ai, aj3 = aj2 * aj;
    const double A3 = ai3 * aj3;
    const double c1 = 4 * ai3 - 3 * ai2 * aj - 3 * ai * aj2 + 4 * aj3;
    const double c2 = 4 * ai3 + 3 * ai2 * aj - 3 * ai * aj2 - 4 * aj3;
    const double c3 = ai3 - 3 * ai2 * aj - 3 * ai * aj2 + aj3;
    const double c4 = ai3 + 3 * ai2 * aj - 3 * ai * aj2 - aj3;
    const double q1 = ai2 - 4 * ai * aj + aj2;
    const double q2 = ai2 + 4 * ai * aj + aj2;
    const double sq = ai2 + aj2;
    const double dq = (ai2 - aj2) * (ai2 - aj2);
    const double s2 = s * s, d2 = d * d;
    const double r2 = r * r, r3 = r2 * r, r4 = r2 * r2, r5 = r4 * r, r6 = r3 * r3;
    const double e1 = exp(-(r + s) * (r + s) * x2), e2 = exp(-(r - s) * (r - s) * x2);
    const double e3 = exp(-(r - d) * (r - d) * x2), e4 = exp(-(r + d) * (r + d) * x2);
    const double g1 = erfc((r + s) * xi), g2 = erfc((r - s) * xi), g3 = erfc((r - d) * xi), g4 = erfc((r + d) * xi);
    const double base_s = r * (3 - 12 * (ai2 - ai * aj + aj2) * x2 - 4 * s2 * q1 * x4);
    const double tail_s = 3 * s + 4 * c1 * x2 + 4 * s2 * s * q1 * x4;
    const double base_d = r * (-3 + 12 * (ai2 + ai * aj + aj2) * x2 + 4 * d2 * q2 * x4);
    const double tail_d = 3 * d + 4 * c2 * x2 + 4 * d2 * d * q2 * x4;
    // I - rr part
    {
        const double k5 = 1.0 / (1024 * sp3 * A3 * r3 * xi * x4);
        const double mid_s = r3 * (16 * x2 + 8 * (-4 * ai2 + ai * aj - 4 * aj2) * x4);
        const double mid_d = r3 * (-16 * x2 + 8 * (4 * ai2 + ai * aj + 4 * aj2) * x4);
        const double f1 = k5 * (4 * r5 * x4 - 4 * s * r4 * x4 + mid_s + r2 * (-12 * s * x2 - 8 * c1 * x4) + base_s + tail_s);
        const double f2 = k5 * (4 * r5 * x4 + 4 * s * r4 * x4 + mid_s + r2 * (12 * s * x2 + 8 * c1 * x4) + base_s - tail_s);
        const double f3 = k5 * (-4 * r5 * x4 - 4 * d * r4 * x4 + mid_d + r2 * (-12 * d * x2 - 8 * c2 * x4) + base_d + tail_d);
        const double f4 = k5 * (-4 * r5 * x4 + 4 * d * r4 * x4 + mid_d + r2 * (12 * d * x2 + 8 * c2 * x4) + base_d - tail_d);
        const double k6 = 1.0 / (2048 * pi * A3 * r3 * x6);
        const double gs = r2 * (-18 * x2 + 72 * sq * x4 + 72 * dq * x6) + 3 - 18 * sq * x2 - 36 * dq * x4;
        const double t4 = 36 * r4 * x4 * (-1 + 2 * sq * x2);
        const double f5 = k6 * (-8 * r6 * x6 + t4 + 128 * (ai3 + aj3) * r3 * x6 + gs - 8 * s2 * s2 * q1 * x6);
        const double f6 = k6 * (-8 * r6 * x6 + t4 - 128 * (ai3 + aj3) * r3 * x6 + gs - 8 * s2 * s2 * q1 * x6);
        const double f7 = k6 * (8 * r6 * x6 - t4 + 128 * (ai3 - aj3) * r3 * x6 - gs + 8 * d2 * d2 * q2 * x6);
        const double f8 = k6 * (8 * r6 * x6 - t4 - 128 * (ai3 - aj3) * r3 * x6 - gs + 8 * d2 * d2 * q2 * x6);
        double reg = 0.0;
        if (r < s && r >= d && r >= -d)
            reg = (s - r) * (s - r) * (s - r) / (128 * pi * A3 * r3) * (-r3 - 3 * s * r2 + 3 * q1 * r + c3);
        else if (r < -d && r > d)
            reg = (r3 - aj3) / (4 * pi * aj3 * r3);
        else if (r < d && r > -d)
            reg = (r3 - ai3) / (4 * pi * ai3 * r3);
        *perp = f1 * e1 + f2 * e2 + f3 * e3 + f4 * e4 + f5 * g1 + f6 * g2 + f7 * g3 + f8 * g4 + reg;
    }
    // rr part
    {
        const double k5 = 1.0 / (512 * sp3 * A3 * r3 * xi * x4);
        const double mid_s = r3 * (14 * x2 - 4 * (7 * ai2 - 4 * ai * aj + 7 * aj2) * x4);
        const double mid_d = r3 * (-14 * x2 + 4 * (7 * ai2 + 4 * ai * aj + 7 * aj2) * x4);
        const double f1 = k5 * (8 * r5 * x4 - 8 * s * r4 * x4 + mid_s + r2 * (-6 * s * x2 - 4 * c3 * x4) - base_s - tail_s);
        const double f2 = k5 * (8 * r5 * x4 + 8 * s * r4 * x4 + mid_s + r2 * (6 * s * x2 + 4 * c3 * x4) - base_s + tail_s);
        const double f3 = k5 * (-8 * r5 * x4 - 8 * d * r4 * x4 + mid_d + r2 * (-6 * d * x2 - 4 * c4 * x4) - base_d - tail_d);
        const double f4 = k5 * (-8 * r5 * x4 + 8 * d * r4 * x4 + mid_d + r2 * (6 * d * x2 + 4 * c4 * x4) - base_d + tail_d);
        const double k6 = 1.0 / (1024 * pi * A3 * r3 * x6);
        const double hs = -3 + 18 * sq * x2 + 36 * dq * x4;
        const double t4 = 36 * r4 * x4 * (-1 + 2 * sq * x2);
        const double f5 = k6 * (-16 * r6 * x6 + t4 + 64 * (ai3 + aj3) * r3 * x6 + hs + 8 * s2 * s2 * q1 * x6);
        const double f6 = k6 * (-16 * r6 * x6 + t4 - 64 * (ai3 + aj3) * r3 * x6 + hs + 8 * s2 * s2 * q1 * x6);
        const double f7 = k6 * (16 * r6 * x6 - t4 + 64 * (ai3 - aj3) * r3 * x6 - hs - 8 * d2 * d2 * q2 * x6);
        const double f8 = k6 * (16 * r6 * x6 - t4 - 64 * (ai3 - aj3) * r3 * x6 - hs - 8 * d2 * d2 * q2 * x6);
        double reg = 0.0;
        if (r < s && r >= d && r >= -d)
            reg = -1.0 / (64 * pi * A3 * r3) * (s2 * s2 * q1 - 8 * (ai3 + aj3) * r3 + 9 * sq * r4 - 2 * r6);
        else if (r < -d && r > d)
            reg = (r3 + 2 * aj3) / (4 * pi * aj3 * r3);
        else if (r < d && r > -d)
            reg = (r3 + 2 * ai3) / (4 * pi * ai3 * r3);
        *para = f1 * e1 + f2 * e2 + f3 * e3 + f4 * e4 + f5 * g1 + f6 * g2 + f7 * g3 + f8 * g4 + reg;
    }
}

// r -> 0 value of both parts (CS/RealSpaceTable.m:87-89).
__host__ __device__ inline double cs_self(double ai, double aj, double xi) {
    const double pi = MPS_PI;
    const double x2 = xi * xi;
    const double ai3 = ai * ai * ai, aj3 = aj * aj * aj;
    return 1.0 / (16 * pi * sqrt(pi) * ai3 * aj3 * xi * x2) *
               ((1 - 2 * ai * ai * x2 + 2 * ai * aj * x2 - 2 * aj * aj * x2) * exp(-(ai + aj) * (ai + aj) * x2) +
                (-1 + 2 * ai * ai * x2 + 2 * ai * aj * x2 + 2 * aj * aj * x2) * exp(-(ai - aj) * (ai - aj) * x2)) +
           1.0 / (8 * pi * ai3 * aj3) * ((ai3 - aj3) * erf((ai - aj) * xi) - (ai3 + aj3) * erf((ai + aj) * xi)) +
           fmin(ai3, aj3) / (4 * pi * ai3 * aj3);
}

// Column of the radius pair (i, j): upper triangle in row order.
__host__ __device__ inline int64_t cs_column(int64_t i, int64_t j, int64_t M) {
    if (i > j) {
        const int64_t t = i;
        i = j;
        j = t;
    }
    return i * M - i * (i - 1) / 2 + (j - i);
}

__global__ void k_cs_table(const double *__restrict__ r, int64_t n, const double *__restrict__ a, int64_t M,
                           double xi, double *__restrict__ perp, double *__restrict__ para) {
    const int64_t m = M * (M + 1) / 2;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n * m; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t % n, col = t / n;
        // invert the column index
        int64_t ci = 0, rem = col;
        while (rem >= M - ci) {
            rem -= M - ci;
            ++ci;
        }
        const int64_t cj = ci + rem;
        double pp, pa;
        if (i == 0) {
            pp = pa = cs_self(a[ci], a[cj], xi);
        } else {
            cs_couplings(r[i], a[ci], a[cj], xi, &pp, &pa);
        }
        perp[col * n + i] = pp;
        para[col * n + i] = pa;
    }
}

// First table entry >= d (search from a uniform-spacing guess).
__device__ __forceinline__ int64_t cs_search(const double *__restrict__ rv, int64_t n, double d) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (rv[mid] < d)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Per-pair couplings of the CSR list: A (I - rr) and B - A, float64 and float32, a pair to a thread, its row by a
// search in row_ptr: the couplings' float64 instructions bound it, and each costs a warp the same for one active lane
// as for 32, however many pairs a row has.  With a thread a row 3,000 spheres filled 94 warps of the chip (60 pairs
// each: 1.58 ms); with a warp a row (0.25 ms) rows of few pairs left most lanes idle (a system of 29,791 spheres with 6
// pairs a row 2.91 ms a thread a row, 3.61 a warp a row, 2.72 so, of 50,653 with 71 10.5, 10.0 and 8.5).
__global__ void k_cs_pair_coefs(const int64_t *__restrict__ row_ptr, const int32_t *__restrict__ nbr,
                                const double *__restrict__ dist, int64_t n, int64_t np,
                                const double *__restrict__ radius, const int32_t *__restrict__ cls, int64_t M,
                                const double *__restrict__ tab, const double *__restrict__ rv, int64_t ntab, double xi,
                                double *__restrict__ A64, double *__restrict__ BA64, float *__restrict__ A32,
                                float *__restrict__ BA32, int *__restrict__ err) {
    const int64_t m = M * (M + 1) / 2;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < np; e += (int64_t)gridDim.x * blockDim.x) {
        int64_t a = 0, hi = n - 1;   // the last row that starts at e or before
        while (a < hi) {
            const int64_t mid = (a + hi + 1) >> 1;
            if (row_ptr[mid] <= e)
                a = mid;
            else
                hi = mid - 1;
        }
        const int32_t b = nbr[e];
        const double d = dist[e];
        double A = 0.0, B = 0.0;
        if (tab) {
            const int64_t col = cs_column(cls[a], cls[b], M);
            const int64_t i = cs_search(rv, ntab, d);
            if (i <= 0 || i >= ntab) {
                atomicExch(err, 1);
            } else {
                const double rl = rv[i - 1], rh = rv[i];
                const double *pp = tab + col * ntab, *pa = tab + (m + col) * ntab;
                A = pp[i - 1] * (rh - d) / (rh - rl) + pp[i] * (d - rl) / (rh - rl);
                B = pa[i - 1] * (rh - d) / (rh - rl) + pa[i] * (d - rl) / (rh - rl);
            }
        } else {
            cs_couplings(d, radius[a], radius[b], xi, &A, &B);
        }
        A64[e] = A;
        BA64[e] = B - A;
        A32[e] = (float)A;
        BA32[e] = (float)(B - A);
    }
}

__global__ void k_cs_diag(const double *__restrict__ lam, int64_t n, int64_t nsets, const double *__restrict__ radius,
                          const int32_t *__restrict__ cls, int64_t M, const double *__restrict__ tab, int64_t ntab,
                          double xi, double *__restrict__ diag) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n * nsets; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = t % n;
        const double ra = radius[a];
        const double self = tab ? tab[cs_column(cls[a], cls[a], M) * ntab] : cs_self(ra, ra, xi);
        diag[t] = 3.0 / (4.0 * MPS_PI * ra * ra * ra * (lam[t] - 1.0)) + self;
    }
}

// Half-away-from-zero rounding of x / h (the MATLAB round of CS/Spread.m:37).
__device__ __forceinline__ double cs_round(double v) {
    const double a = floor(fabs(v) + 0.5);
    return v > 0 ? a : (v < 0 ? -a : 0.0 * a);
}

// Per particle: wrapped index of stencil column 0, base = node0 h - x, and the
// kernel K(d)/d at every node of the P^3 stencil (x fastest).
__global__ void k_cs_geom(const double *__restrict__ x, int64_t n, GridParams gp, const double *__restrict__ radius,
                          double xi, double eta, int32_t *__restrict__ start, double *__restrict__ base,
                          double *__restrict__ g64, float *__restrict__ g32) {
    const int P = gp.P;
    const int64_t P3 = (int64_t)P * P * P;
    const int lo = (P - 1) / 2;
    const double pi = MPS_PI;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n * P3; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = t / P3;
        const int64_t l = t % P3;
        const int o[3] = {(int)(l % P) - lo, (int)((l / P) % P) - lo, (int)(l / ((int64_t)P * P)) - lo};
        double r[3];
        for (int k = 0; k < 3; ++k) {
            const double xv = x[3 * a + k];
            const double node0 = cs_round(__ddiv_rn(xv, gp.h[k]));
            if (l == 0) {
                start[3 * a + k] = (int32_t)wrap_index((int64_t)node0 - lo - 1, gp.N[k]);
                base[3 * a + k] = node0 * gp.h[k] - xv;
            }
            r[k] = (node0 * gp.h[k] + (double)o[k] * gp.h[k]) - xv;
        }
        const double d = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
        const double ra = radius[a];
        double v;
        if (d < 1e-6) {
            // small-d form as the reference writes it (CS/Spread.m:60-61)
            v = 8 * sqrt(2.0) * pow(xi, 5) * exp(-2 * ra * xi * xi / eta) / (pi * sqrt(pi) * pow(eta, 2.5));
        } else {
            const double K = 3.0 / (8 * sqrt(2.0) * pi * sqrt(pi) * ra * ra * ra * sqrt(eta) * xi * d * d) *
                             ((eta + 4 * ra * xi * xi * d) * exp(-2 * (d + ra) * (d + ra) * xi * xi / eta) -
                              (eta - 4 * ra * xi * xi * d) * exp(-2 * (d - ra) * (d - ra) * xi * xi / eta));
            v = K / d;
        }
        g64[t] = v;
        if (g32) g32[t] = (float)v;
    }
}

__global__ void k_cs_green(GridParams gp, double eta, double xi, double *__restrict__ c64, float *__restrict__ c32) {
    const int Nxh = gp.N[0] / 2 + 1;
    const int64_t Gc = (int64_t)Nxh * gp.N[1] * gp.N[2];
    const double invG = 1.0 / (double)gp.G;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < Gc; t += (int64_t)gridDim.x * blockDim.x) {
        const int ix = (int)(t % Nxh);
        const int iy = (int)((t / Nxh) % gp.N[1]);
        const int iz = (int)(t / ((int64_t)Nxh * gp.N[1]));
        const double kx = fft_freq(ix, gp.N[0]) * gp.kfac[0];
        const double ky = fft_freq(iy, gp.N[1]) * gp.kfac[1];
        const double kz = fft_freq(iz, gp.N[2]) * gp.kfac[2];
        const double q2 = kx * kx + ky * ky + kz * kz;
        const double v = q2 > 0 ? exp(-(1 - eta) * q2 / (4 * xi * xi)) / q2 * invG : 0.0;
        c64[t] = v;
        if (c32) c32[t] = (float)v;
    }
}

// Spread: a warp per (particle, block of RB vectors); lanes walk the (x, y)
// footprint.  The particle's node weights K(d)/d (P^3 per particle) are read once
// per block of vectors instead of once per vector: with a spectrum batch (3 fields x
// K contrasts) they were the dominant read.
template <typename T, int RB, int MB = 1>
__global__ void __launch_bounds__(256, MB) k_spread_cs(const double *__restrict__ m, int64_t n, int nrhs,
                                                   const int32_t *__restrict__ start, const double *__restrict__ base,
                                                   const T *__restrict__ g, GridParams gp, T *__restrict__ grid) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int P = gp.P;
    const int lo = (P - 1) / 2;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const int64_t P3 = (int64_t)P * P * P;
    const int nblk = (nrhs + RB - 1) / RB;
    for (int64_t t = warp; t < n * nblk; t += nw) {
        const int64_t a = gp.order ? (int64_t)gp.order[t % n] : t % n;
        const int r0 = (int)(t / n) * RB;
        const int cnt = min(RB, nrhs - r0);
        const int sx = start[3 * a], sy = start[3 * a + 1], sz = start[3 * a + 2];
        // every lane loads all the vectors' moments: handed round by shuffles from a lane each, the kernel took up to
        // twice as long (12 vectors, N = 4000, 64^3, P = 16 215 us so, 430 by shuffles; N = 20,000, 80^3, P = 8 171 and
        // 269)
        T px[RB], py[RB], pz[RB];
#pragma unroll
        for (int q = 0; q < RB; ++q) {
            const double *ma = m + ((int64_t)(r0 + (q < cnt ? q : 0)) * n + a) * 3;
            px[q] = (T)ma[0];
            py[q] = (T)ma[1];
            pz[q] = (T)ma[2];
        }
        const T bx = (T)(base[3 * a] - lo * gp.h[0]), by = (T)(base[3 * a + 1] - lo * gp.h[1]),
                bz = (T)(base[3 * a + 2] - lo * gp.h[2]);
        const T hx = (T)gp.h[0], hy = (T)gp.h[1], hz = (T)gp.h[2];
        const T *ga = g + a * P3;
        T *gr = grid + (int64_t)r0 * gp.G;
        for (int row0 = 0; row0 < P * P; row0 += 32) {
            int idx, sub, lpp;
            if (!stencil_row(row0, P, lane, &idx, &sub, &lpp)) continue;
            const int jx = idx % P, jy = idx / P;
            int ix = sx + jx;
            if (ix >= Nx) ix -= Nx;
            int iy = sy + jy;
            if (iy >= Ny) iy -= Ny;
            const T rx = bx + (T)jx * hx, ry = by + (T)jy * hy;
            T pxy[RB];
#pragma unroll
            for (int q = 0; q < RB; ++q) pxy[q] = rx * px[q] + ry * py[q];
            const int64_t rowb = (int64_t)ix + (int64_t)Nx * iy;
            for (int jz = sub; jz < P; jz += lpp) {
                int iz = sz + jz;
                if (iz >= Nz) iz -= Nz;
                const T rz = bz + (T)jz * hz;
                const T wv = ga[jx + P * (jy + P * jz)];
                T *node = gr + rowb + (int64_t)Nx * Ny * iz;
#pragma unroll
                for (int q = 0; q < RB; ++q)
                    if (q < cnt) atomicAdd(node + (int64_t)q * gp.G, wv * (pxy[q] + rz * pz[q]));
            }
        }
    }
}

template <typename T>
struct CsCplx;
template <>
struct CsCplx<float> {
    using type = float2;
};
template <>
struct CsCplx<double> {
    using type = double2;
};

// spec[r][k] *= coef[k]: a thread takes one spectrum point of a few vectors (blockIdx.y), with one complex (8 or 16
// byte) load and store per value; with all vectors to a thread a small grid's points filled the chip too thinly (48
// vectors on 40^3: 13.7 -> 4.0 us).
constexpr int kScaleVec = 4;

template <typename T>
__global__ void k_scale_cs(T *__restrict__ spec, int nrhs, int64_t Gc, const T *__restrict__ coef, T factor) {
    using C = typename CsCplx<T>::type;
    const int r0 = blockIdx.y * kScaleVec, cnt = min(kScaleVec, nrhs - r0);
    C *sp = reinterpret_cast<C *>(spec) + (int64_t)r0 * Gc;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < Gc; t += (int64_t)gridDim.x * blockDim.x) {
        const T c = factor * coef[t];
        C v[kScaleVec];
#pragma unroll
        for (int r = 0; r < kScaleVec; ++r)
            if (r < cnt) v[r] = sp[(int64_t)r * Gc + t];
#pragma unroll
        for (int r = 0; r < kScaleVec; ++r)
            if (r < cnt) {
                v[r].x *= c;
                v[r].y *= c;
                sp[(int64_t)r * Gc + t] = v[r];
            }
    }
}

// Contract: out = prod(h) sum_nodes K(d)/d (node - x) E~(node)  (overwrites).
// A warp per (particle, block of RB vectors): the node weights are read once per
// block; each vector's sums run in the same order as with one vector per warp.
template <typename T, int RB, int MB = 1>
__global__ void __launch_bounds__(256, MB) k_contract_cs(const T *__restrict__ grid, int64_t n, int nrhs,
                                                     const int32_t *__restrict__ start,
                                                     const double *__restrict__ base, const T *__restrict__ g,
                                                     GridParams gp, double *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int P = gp.P;
    const int lo = (P - 1) / 2;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const int64_t P3 = (int64_t)P * P * P;
    const int nblk = (nrhs + RB - 1) / RB;
    const int oc = warp_sums_index<3 * RB>(lane);   // the sum this lane writes
    for (int64_t t = warp; t < n * nblk; t += nw) {
        const int64_t a = gp.order ? (int64_t)gp.order[t % n] : t % n;
        const int r0 = (int)(t / n) * RB;
        const int cnt = min(RB, nrhs - r0);
        const int sx = start[3 * a], sy = start[3 * a + 1], sz = start[3 * a + 2];
        const T bx = (T)(base[3 * a] - lo * gp.h[0]), by = (T)(base[3 * a + 1] - lo * gp.h[1]),
                bz = (T)(base[3 * a + 2] - lo * gp.h[2]);
        const T hx = (T)gp.h[0], hy = (T)gp.h[1], hz = (T)gp.h[2];
        const T *ga = g + a * P3;
        const T *gr = grid + (int64_t)r0 * gp.G;
        T acc[3 * RB];
#pragma unroll
        for (int q = 0; q < 3 * RB; ++q) acc[q] = 0;
        for (int row0 = 0; row0 < P * P; row0 += 32) {
            int idx, sub, lpp;
            if (!stencil_row(row0, P, lane, &idx, &sub, &lpp)) continue;
            const int jx = idx % P, jy = idx / P;
            int ix = sx + jx;
            if (ix >= Nx) ix -= Nx;
            int iy = sy + jy;
            if (iy >= Ny) iy -= Ny;
            const T rx = bx + (T)jx * hx, ry = by + (T)jy * hy;
            const int64_t rowb = (int64_t)ix + (int64_t)Nx * iy;
            T sxy[RB], szz[RB];
#pragma unroll
            for (int q = 0; q < RB; ++q) sxy[q] = szz[q] = 0;
            for (int jz = sub; jz < P; jz += lpp) {
                int iz = sz + jz;
                if (iz >= Nz) iz -= Nz;
                const T wv = ga[jx + P * (jy + P * jz)];
                const T wz = wv * (bz + (T)jz * hz);
                const T *node = gr + rowb + (int64_t)Nx * Ny * iz;
#pragma unroll
                for (int q = 0; q < RB; ++q) {
                    if (q < cnt) {
                        const T v = node[(int64_t)q * gp.G];
                        sxy[q] += wv * v;
                        szz[q] += wz * v;
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < RB; ++q) {
                acc[3 * q] += rx * sxy[q];
                acc[3 * q + 1] += ry * sxy[q];
                acc[3 * q + 2] += szz[q];
            }
        }
        const T v = warp_sums(acc, lane);
        if (oc >= 0 && oc < 3 * cnt) out[((int64_t)(r0 + oc / 3) * n + a) * 3 + oc % 3] = (double)v * gp.hprod;
    }
}

// ---------------------------------------------------------------------------
// Many vectors (a spectrum or sweep batch).
//
// Spread: a block owns an 8 x 4 x 4 tile of nodes and walks the particles whose stencils reach it (TileBins), 32 at
// a time with their moments in shared memory; a warp owns two rows of 8 nodes, one above the other, four lanes to a
// pair of nodes, and takes the particles that reach its rows (a ballot), four at a time: one weight K(d)/d a node
// serves 16 vectors a group, V groups to a block.  Every node is written once, in the planes that the transforms read,
// in a fixed order of sums: no atomics, no zeroing.  48 vectors, 3,000 spheres, 40^3, P = 8: 87 us with float atomics
// from a warp a particle (78 with four-vector atomics on interleaved grids), 54 so.  Reading the moments from shared
// memory bounds it, so a lane keeps two nodes along z for each read (one: 73).
//
// Contraction: the grids lie side by side, node by node, four vectors to a float4.  From planes, a warp touched a line
// in L1 for every vector and row of the stencil; here four lanes take a node's 16 vectors (64 contiguous bytes), eight
// nodes of the stencil at a time, the weights are read once for all 16, and no sum crosses more than eight lanes.  103
// -> 50 us, the L2's bandwidth, and 7 us for the transposition.
// ---------------------------------------------------------------------------
constexpr int kCsGroup = 16;
constexpr int kCsTileX = 8, kCsTileY = 4, kCsTileZ = 4, kCsChunk = 32;

// mv[a][axis][v] = m[v][a][axis], v < 4 vq (zeros beyond nrhs).
__global__ void k_cs_moments(const double *__restrict__ m, int64_t n, int nrhs, int vq, float *__restrict__ mv) {
    const int64_t total = n * 12 * vq;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a3 = t / (4 * vq);   // 3 a + axis
        const int v = (int)(t - a3 * (4 * vq));
        mv[t] = v < nrhs ? (float)m[(int64_t)v * n * 3 + a3] : 0.f;
    }
}

template <int V>
__global__ void __launch_bounds__(256, 4) k_spread_cs_nodes(const float4 *__restrict__ mv, int nrhs, int vq,
                                                         const int32_t *__restrict__ start,
                                                         const double *__restrict__ base, const float *__restrict__ g,
                                                         GridParams gp, const int64_t *__restrict__ tstart,
                                                         const int32_t *__restrict__ entries, int ntx, int nty,
                                                         float *__restrict__ grid) {
    __shared__ float4 s_m[kCsChunk][3][4 * V];
    __shared__ float4 s_b[kCsChunk];    // node0 - x of the stencil's first node, particle id
    __shared__ int s_o[kCsChunk][3];    // stencil index of the tile's first node
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, lv = lane & 3, xn = lane >> 2;
    const int64_t t = blockIdx.x;
    const int X0 = (int)(t % ntx) * kCsTileX, Y0 = (int)((t / ntx) % nty) * kCsTileY,
              Z0 = (int)(t / ((int64_t)ntx * nty)) * kCsTileZ;
    const int yr = wid & (kCsTileY - 1), zr = 2 * (wid / kCsTileY);   // the warp's rows: (yr, zr) and (yr, zr + 1)
    const int P = gp.P, lo = (P - 1) / 2;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const bool inx = X0 + xn < Nx, row_in = Y0 + yr < Ny && Z0 + zr < Nz;
    const int q0 = (int)blockIdx.y * 4 * V;   // first float4 of the block's vectors
    const float hx = (float)gp.h[0], hy = (float)gp.h[1], hz = (float)gp.h[2];
    float acc[2][V][4];
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[0][v][k] = acc[1][v][k] = 0.f;
    const int64_t e0 = tstart[t], e1 = tstart[t + 1];
    for (int64_t cb = e0; cb < e1; cb += kCsChunk) {
        const int cnt = (int)min((int64_t)kCsChunk, e1 - cb);
        // a warp copies four particles' moments; the first works out the geometry too
        int32_t id[kCsChunk / 8];
#pragma unroll
        for (int k = 0; k < kCsChunk / 8; ++k) id[k] = wid + 8 * k < cnt ? entries[cb + wid + 8 * k] : -1;
#pragma unroll
        for (int k = 0; k < kCsChunk / 8; ++k)
            if (id[k] >= 0)
                for (int i = lane; i < 12 * V; i += 32) {
                    const int c = i / (4 * V), q = i - c * (4 * V);
                    if (q0 + q < vq)
                        copy_async(&s_m[wid + 8 * k][c][q], mv + (3 * (int64_t)id[k] + c) * vq + q0 + q);
                    else
                        s_m[wid + 8 * k][c][q] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
        if (threadIdx.x < cnt) {
            const int32_t a = entries[cb + threadIdx.x];
            const double *b = base + 3 * (int64_t)a;
            s_b[threadIdx.x] = make_float4((float)(b[0] - lo * gp.h[0]), (float)(b[1] - lo * gp.h[1]),
                                           (float)(b[2] - lo * gp.h[2]), __int_as_float(a));
            const int32_t *sa = start + 3 * (int64_t)a;
            s_o[threadIdx.x][0] = X0 - sa[0] + (X0 < sa[0] ? Nx : 0);
            s_o[threadIdx.x][1] = Y0 - sa[1] + (Y0 < sa[1] ? Ny : 0);
            s_o[threadIdx.x][2] = Z0 - sa[2] + (Z0 < sa[2] ? Nz : 0);
        }
        copy_async_wait();
        __syncthreads();
        // the chunk's particles whose stencils hold one of the rows
        bool on = false;
        if (lane < cnt && row_in) {
            int jy = s_o[lane][1] + yr, jz = s_o[lane][2] + zr;
            jy -= jy >= Ny ? Ny : 0;
            jz -= jz >= Nz ? Nz : 0;
            on = jy < P && (jz < P || jz == Nz - 1);   // (the second row holds the stencil's first plane)
        }
        unsigned list = __ballot_sync(0xffffffffu, on);
        // four particles at a time: each of a node's lanes works out one of them, shuffles hand its weights round
        while (list) {
            int pk[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                pk[k] = __ffs(list) - 1;   // -1 when the list is done
                list &= list - 1;
            }
            const int p = lv == 0 ? pk[0] : lv == 1 ? pk[1] : lv == 2 ? pk[2] : pk[3];
            float wx[2] = {0.f, 0.f}, wy[2] = {0.f, 0.f}, wz[2] = {0.f, 0.f};
            if (p >= 0) {
                int jx = s_o[p][0] + xn, jy = s_o[p][1] + yr, jz = s_o[p][2] + zr;
                jx -= jx >= Nx ? Nx : 0;
                jy -= jy >= Ny ? Ny : 0;
                jz -= jz >= Nz ? Nz : 0;
                const float4 b = s_b[p];
                const float *ga = g + ((int64_t)__float_as_int(b.w) * P * P + jy) * P + jx;
                const bool in = inx && jx < P;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float wv = in && jz < P ? ga[jz * P * P] : 0.f;
                    wx[h] = wv * (b.x + (float)jx * hx);
                    wy[h] = wv * (b.y + (float)jy * hy);
                    wz[h] = wv * (b.z + (float)jz * hz);
                    if (++jz >= Nz) jz = 0;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (pk[k] < 0) break;   // the whole warp
                const int src = (lane & 28) | k;
                float u[2][3];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    u[h][0] = __shfl_sync(0xffffffffu, wx[h], src);
                    u[h][1] = __shfl_sync(0xffffffffu, wy[h], src);
                    u[h][2] = __shfl_sync(0xffffffffu, wz[h], src);
                }
#pragma unroll
                for (int v = 0; v < V; ++v)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float4 mc = s_m[pk[k]][c][4 * v + lv];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            acc[h][v][0] += u[h][c] * mc.x;
                            acc[h][v][1] += u[h][c] * mc.y;
                            acc[h][v][2] += u[h][c] * mc.z;
                            acc[h][v][3] += u[h][c] * mc.w;
                        }
                    }
            }
        }
        __syncthreads();
    }
    if (inx && row_in) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (Z0 + zr + h >= Nz) break;
            float *o = grid + ((int64_t)(Z0 + zr + h) * Ny + Y0 + yr) * Nx + X0 + xn;
#pragma unroll
            for (int v = 0; v < V; ++v)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int r = 4 * (q0 + 4 * v + lv) + k;
                    if (r < nrhs) o[r * gp.G] = acc[h][v][k];
                }
        }
    }
}

__global__ void __launch_bounds__(256) k_contract_cs_il(const float4 *__restrict__ il, int64_t n, int nrhs, int vq,
                                                        const int32_t *__restrict__ start,
                                                        const double *__restrict__ base, const float *__restrict__ g,
                                                        GridParams gp, double *__restrict__ out) {
    const int lane = threadIdx.x & 31, lv = lane & 3, ni = lane >> 2;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int P = gp.P, PP = P * P, lo = (P - 1) / 2;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const int64_t plane = (int64_t)Nx * Ny * vq;
    const int nblk = (nrhs + kCsGroup - 1) / kCsGroup;
    for (int64_t t = warp; t < n * nblk; t += nw) {
        const int64_t a = gp.order ? (int64_t)gp.order[t % n] : t % n;
        const int r0 = (int)(t / n) * kCsGroup, vec = min(r0 / 4 + lv, vq - 1);   // (surplus lanes repeat the last four)
        const int sx = start[3 * a], sy = start[3 * a + 1], sz = start[3 * a + 2];
        const float bx = (float)(base[3 * a] - lo * gp.h[0]), by = (float)(base[3 * a + 1] - lo * gp.h[1]),
                    bz = (float)(base[3 * a + 2] - lo * gp.h[2]);
        const float hx = (float)gp.h[0], hy = (float)gp.h[1], hz = (float)gp.h[2];
        const float *ga = g + a * PP * P;
        float acc[12];   // 3 vector + axis
#pragma unroll
        for (int k = 0; k < 12; ++k) acc[k] = 0.f;
        for (int col = ni; col < PP; col += 8) {
            const int jy = col / P, jx = col - jy * P;
            int ix = sx + jx, iy = sy + jy;
            if (ix >= Nx) ix -= Nx;
            if (iy >= Ny) iy -= Ny;
            const float rx = bx + (float)jx * hx, ry = by + (float)jy * hy;
            const float4 *row = il + ((int64_t)ix + (int64_t)Nx * iy) * vq + vec;
            float s[4] = {0.f, 0.f, 0.f, 0.f}, z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int jz = 0; jz < P; ++jz) {
                int iz = sz + jz;
                if (iz >= Nz) iz -= Nz;
                const float wv = ga[col + PP * jz], wz = wv * (bz + (float)jz * hz);
                const float4 v = __ldg(row + plane * iz);
                s[0] += wv * v.x;
                s[1] += wv * v.y;
                s[2] += wv * v.z;
                s[3] += wv * v.w;
                z[0] += wz * v.x;
                z[1] += wz * v.y;
                z[2] += wz * v.z;
                z[3] += wz * v.w;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc[3 * k] += rx * s[k];
                acc[3 * k + 1] += ry * s[k];
                acc[3 * k + 2] += z[k];
            }
        }
        // sums over the eight node lanes, halving what a lane carries: 12 -> 6 -> 3 -> one or two
        const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
        float b[6], c[3];
#pragma unroll
        for (int k = 0; k < 6; ++k)
            b[k] = (h16 ? acc[k + 6] : acc[k]) + __shfl_xor_sync(0xffffffffu, h16 ? acc[k] : acc[k + 6], 16);
#pragma unroll
        for (int k = 0; k < 3; ++k) c[k] = (h8 ? b[k + 3] : b[k]) + __shfl_xor_sync(0xffffffffu, h8 ? b[k] : b[k + 3], 8);
        const float d0 = (h4 ? c[2] : c[0]) + __shfl_xor_sync(0xffffffffu, h4 ? c[0] : c[2], 4);
        const float d1 = c[1] + __shfl_xor_sync(0xffffffffu, c[1], 4);
        const int k0 = (h16 ? 2 : 0) + (h8 ? 1 : 0), r = r0 + 4 * lv + k0;
        if (r < nrhs) {
            double *o = out + ((int64_t)r * n + a) * 3;
            o[h4 ? 2 : 0] = (double)d0 * gp.hprod;
            if (!h4) o[1] = (double)d1 * gp.hprod;
        }
    }
}

// Planes to interleaved: 32 nodes and 64 vectors of them to a block, through shared memory.
__global__ void __launch_bounds__(256) k_cs_interleave(const float *__restrict__ grid, int nrhs, int64_t G, int vq,
                                                       float4 *__restrict__ il) {
    __shared__ float s[64][33];
    const int64_t t0 = (int64_t)blockIdx.x * 32;
    const int v0 = (int)blockIdx.y * 64, lane = threadIdx.x & 31;
    for (int v = threadIdx.x >> 5; v < 64; v += 8)
        s[v][lane] = v0 + v < nrhs && t0 + lane < G ? grid[(int64_t)(v0 + v) * G + t0 + lane] : 0.f;
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * 16; e += 256) {
        const int node = e >> 4, q = e & 15;
        if (t0 + node < G && v0 / 4 + q < vq)
            il[(t0 + node) * vq + v0 / 4 + q] = make_float4(s[4 * q][node], s[4 * q + 1][node], s[4 * q + 2][node],
                                                            s[4 * q + 3][node]);
    }
}

// ---------------------------------------------------------------------------
// Host wrappers
// ---------------------------------------------------------------------------
int cs_pair_coefs(const int64_t *row_ptr, const int32_t *nbr, const double *dist, int64_t n, int64_t np,
                  const double *radius, const int32_t *cls, int64_t M, const double *tab, const double *rv,
                  int64_t ntab, double xi, PairData<double> p64, PairData<float> p32, int *err, cudaStream_t s) {
    k_cs_pair_coefs<<<grid_for(np, 128), 128, 0, s>>>(row_ptr, nbr, dist, n, np, radius, cls, M, tab, rv, ntab, xi,
                                                      p64.A, p64.BA, p32.A, p32.BA, err);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int cs_diag(const double *lam, int64_t n, int64_t nsets, const double *radius, const int32_t *cls, int64_t M,
            const double *tab, int64_t ntab, double xi, double *diag, cudaStream_t s) {
    k_cs_diag<<<grid_for(n * nsets, 256), 256, 0, s>>>(lam, n, nsets, radius, cls, M, tab, ntab, xi, diag);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int cs_geometry(const double *x, int64_t n, const GridParams &gp, const double *radius, double xi, double eta,
                int32_t *start, double *base, double *g64, float *g32, cudaStream_t s) {
    const int64_t P3 = (int64_t)gp.P * gp.P * gp.P;
    k_cs_geom<<<grid_for(n * P3, 256), 256, 0, s>>>(x, n, gp, radius, xi, eta, start, base, g64, g32);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int cs_green(const GridParams &gp, double eta, double xi, double *c64, float *c32, cudaStream_t s) {
    const int64_t Gc = (int64_t)(gp.N[0] / 2 + 1) * gp.N[1] * gp.N[2];
    k_cs_green<<<grid_for(Gc, 256), 256, 0, s>>>(gp, eta, xi, c64, c32);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template <typename T>
int spread_cs(const double *m, int64_t n, int nrhs, const int32_t *start, const double *base, const T *g,
              const GridParams &gp, T *grid, cudaStream_t s) {
    MPS_CUDA_TRY(cudaMemsetAsync(grid, 0, sizeof(T) * (size_t)nrhs * gp.G, s));
    if (n == 0) return MPS_OK;
    // 8 vectors per warp pass (the node weights read once per 8 vectors); 4 and 16 measured slower.  Fewer vectors take
    // passes of their own width: the surplus vectors' loads and conversions cost a warp as much as the real ones' (one
    // vector, 8000 particles, 54^3, P = 8 33 -> 22 us; in float64 1728, 31^3, P = 12 56 -> 46;
    // three and four in float64 were slower on larger grids, 64^3, P = 12 151 -> 181)
    const int64_t items = n * ((nrhs + 7) / 8);
    // float: bounds of 4 blocks per SM (72.8 ms over the 16-configuration batch's float32 matvecs against 75.8
    // unbounded); double: unbounded (a 64-register cap spills it)
    constexpr int MB = sizeof(T) == 4 ? 4 : 1;
    const auto kernel = nrhs == 1   ? k_spread_cs<T, 1, MB>
                        : nrhs == 2 ? k_spread_cs<T, 2, MB>
                        : nrhs <= 4 && sizeof(T) == 4 ? k_spread_cs<T, 4, MB>
                                                      : k_spread_cs<T, 8, MB>;
    kernel<<<grid_for(items * 32, 256, 152 * 64), 256, 0, s>>>(m, n, nrhs, start, base, g, gp, grid);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

// What both kernels of many vectors take: a group of vectors, stencils that wrap once, the scratch's size.
static bool cs_many(const GridParams &gp, int64_t n, int nrhs) {
    if (nrhs < kCsGroup || n < 1 || 3 * n > gp.G || gp.P > kMaxP) return false;
    const int T[3] = {kCsTileX, kCsTileY, kCsTileZ};
    for (int d = 0; d < 3; ++d)
        if (gp.N[d] < T[d] || gp.N[d] < gp.P) return false;
    return true;
}

// Spread by tiles: with fewer than two tiles for every SM a tile's list is the time it takes, and on a large grid with
// few particles every tile's own time is.  By warps a particle / by tiles, us: 16 vectors, P = 8, 40^3, 3000 and 216
// particles 39 / 34 and 21 / 14; 96^3, P = 6, 16 vectors, 1105 particles 27 / 45, 8847 66 / 76; 48 vectors, 500
// particles, P = 8 66 / 66.
bool cs_many_spread(const GridParams &gp, int64_t n, int nrhs) {
    return cs_many(gp, n, nrhs) && gp.G >= 300 * kCsTileX * kCsTileY * kCsTileZ &&
           (gp.G < 150000 || (double)n * gp.P * gp.P * gp.P * nrhs >= 30.0 * gp.G);
}

// Contraction of interleaved grids: the transposition costs by nodes, the gather that it speeds up by particles, and a
// group that is not full costs as much as a full one.  By planes / interleaved, us: 48 vectors, 40^3, 3000 spheres, P =
// 8 85 / 60, 216 16 / 25; 16 vectors, 40^3, P = 8, 4000 43 / 37, 1600 23 / 25; 96^3, P = 6, 1105 27 / 69.
bool cs_many_contract(const GridParams &gp, int64_t n, int nrhs) {
    const int lanes = (nrhs + kCsGroup - 1) / kCsGroup * kCsGroup;
    return cs_many(gp, n, nrhs) && (double)n * gp.P * gp.P * (2 * nrhs - lanes) >= 20.0 * gp.G && n * nrhs >= 40000;
}

size_t cs_many_floats(int nrhs, int64_t G) {
    return nrhs < kCsGroup ? 0 : (size_t)((nrhs + 3) / 4) * 4 * (size_t)G;   // (fewer vectors never take these kernels)
}

int cs_bins_build(const int32_t *start, int64_t n, const GridParams &gp, TileBins &tb, cudaStream_t s) {
    return bins_build(start, n, gp, kCsTileX, kCsTileY, kCsTileZ, tb, s);
}

int spread_cs_many(const double *m, int64_t n, int nrhs, const int32_t *start, const double *base, const float *g,
                   const GridParams &gp, const TileBins &tb, float *scratch, float *grid, cudaStream_t s) {
    if (tb.tx != kCsTileX || tb.ty != kCsTileY || tb.tz != kCsTileZ) return MPS_BAD_ARG;
    const int vq = (nrhs + 3) / 4, groups = (nrhs + kCsGroup - 1) / kCsGroup;
    k_cs_moments<<<grid_for(n * 12 * vq, 256), 256, 0, s>>>(m, n, nrhs, vq, scratch);
    MPS_LAUNCH_CHECK();
    const float4 *mv = (const float4 *)scratch;
    // as many groups to a block as leave the fewest lanes without a vector, more rather than fewer
    const int V = groups % 3 == 0 || groups > 4 ? 3 : (groups % 2 == 0 ? 2 : 1);
    const dim3 blocks((unsigned)tb.ntiles, (groups + V - 1) / V);
    if (V == 3)
        k_spread_cs_nodes<3><<<blocks, 256, 0, s>>>(mv, nrhs, vq, start, base, g, gp, tb.tile_start, tb.entries, tb.ntx,
                                                    tb.nty, grid);
    else if (V == 2)
        k_spread_cs_nodes<2><<<blocks, 256, 0, s>>>(mv, nrhs, vq, start, base, g, gp, tb.tile_start, tb.entries, tb.ntx,
                                                    tb.nty, grid);
    else
        k_spread_cs_nodes<1><<<blocks, 256, 0, s>>>(mv, nrhs, vq, start, base, g, gp, tb.tile_start, tb.entries, tb.ntx,
                                                    tb.nty, grid);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int contract_cs_many(const float *grid, int64_t n, int nrhs, const int32_t *start, const double *base, const float *g,
                     const GridParams &gp, float *scratch, double *out, cudaStream_t s) {
    const int vq = (nrhs + 3) / 4;
    k_cs_interleave<<<dim3((unsigned)((gp.G + 31) / 32), (vq + 15) / 16), 256, 0, s>>>(grid, nrhs, gp.G, vq,
                                                                                       (float4 *)scratch);
    MPS_LAUNCH_CHECK();
    const int64_t items = n * ((nrhs + kCsGroup - 1) / kCsGroup);
    k_contract_cs_il<<<grid_for(items * 32, 256, 152 * 64), 256, 0, s>>>((const float4 *)scratch, n, nrhs, vq, start,
                                                                         base, g, gp, out);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template <typename T>
int scale_cs(void *spec, int nrhs, const GridParams &gp, const T *coef, cudaStream_t s, double factor) {
    const int64_t Gc = (int64_t)(gp.N[0] / 2 + 1) * gp.N[1] * gp.N[2];
    k_scale_cs<T><<<dim3(grid_for(Gc, 256), (nrhs + kScaleVec - 1) / kScaleVec), 256, 0, s>>>((T *)spec, nrhs, Gc, coef,
                                                                                                   (T)factor);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template <typename T>
int contract_cs(const T *grid, int64_t n, int nrhs, const int32_t *start, const double *base, const T *g,
                const GridParams &gp, double *out, cudaStream_t s) {
    if (n == 0) return MPS_OK;
    // 4 vectors per warp pass (5 x 4 accumulators per lane): 99 ms against 104 for 8 over the 16-configuration
    // batch's float32 matvecs; 16 spills
    const int64_t items = n * ((nrhs + 3) / 4);
    // float: bounds of 3 blocks per SM (76 registers: 83 ms over the batch's float32 matvecs against 99 at 64)
    constexpr int MB = sizeof(T) == 4 ? 3 : 1;
    k_contract_cs<T, 4, MB><<<grid_for(items * 32, 256, 152 * 64), 256, 0, s>>>(grid, n, nrhs, start, base, g, gp, out);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template int spread_cs<float>(const double *, int64_t, int, const int32_t *, const double *, const float *,
                              const GridParams &, float *, cudaStream_t);
template int spread_cs<double>(const double *, int64_t, int, const int32_t *, const double *, const double *,
                               const GridParams &, double *, cudaStream_t);
template int scale_cs<float>(void *, int, const GridParams &, const float *, cudaStream_t, double);
template int scale_cs<double>(void *, int, const GridParams &, const double *, cudaStream_t, double);
template int contract_cs<float>(const float *, int64_t, int, const int32_t *, const double *, const float *,
                                const GridParams &, double *, cudaStream_t);
template int contract_cs<double>(const double *, int64_t, int, const int32_t *, const double *, const double *,
                                 const GridParams &, double *, cudaStream_t);

}  // namespace mps

using namespace mps;

extern "C" int mps_sizes_table(const double *r, int64_t n, const double *a_uniq, int64_t M, double xi, double *perp,
                               double *para, mps_stream_t stream) {
    if (n < 1 || M < 1 || !r || !a_uniq || !perp || !para || !(xi > 0)) return MPS_BAD_ARG;
    const int64_t m = M * (M + 1) / 2;
    k_cs_table<<<grid_for(n * m, 256), 256, 0, (cudaStream_t)stream>>>(r, n, a_uniq, M, xi, perp, para);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}
