// Adjoint forces of the polarisation energy E = -1/2 m . H0 with A(x) m = H0.
//
// Because the operator is symmetric, dE/dx_k = 1/2 m^T (dA/dx_k) m with the
// converged moments held fixed (no second solve), so
//   F_k = -dE/dx_k = -sum_j grad_r [m_k . M(r) m_j]            (real space)
//                    - h^3 sum_n grad_x w_k(n) (m_k . phi(n))  (wave space)
// with M(r) = A(r)(I - r r) + B(r) r r, r = x_k - x_j (minimum image), A and B
// the linearly interpolated tables (their derivatives are the segment slopes,
// i.e. the exact derivative of the operator that was solved), w_k the Gaussian
// spreading weight and phi the convolved grid the contraction reads
// (IFFT(scale(FFT(spread(m))))).  The dielectric, self and slab terms do not
// depend on positions.  dE/d eps_k = 1/2 |m_k|^2 dD_k/d eps_k with
// D_k = 3 / (4 pi (eps_k - 1)) + self.
#include <math.h>

#include "cells.cuh"
#include "grid.cuh"

namespace mps {

// Slopes of the tables' segments, sl[i] = (perp, para) slope between rows i - 1 and i; sl[0].x = the index guess's
// 1 / spacing.  Per pair they would cost two float64 divisions.
__global__ void k_table_slopes(const double *__restrict__ perp, const double *__restrict__ para,
                               const double *__restrict__ rv, int64_t ntab, double2 *__restrict__ sl) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ntab; i += (int64_t)gridDim.x * blockDim.x) {
        if (i == 0) {
            sl[0] = make_double2(rv[ntab - 1] > 0 ? (double)(ntab - 1) / rv[ntab - 1] : 0.0, 0.0);
        } else {
            const double dr = rv[i] - rv[i - 1];
            sl[i] = make_double2((perp[i] - perp[i - 1]) / dr, (para[i] - para[i - 1]) / dr);
        }
    }
}

// First index with rv[i] >= d (ntab where there is none), from the uniform-spacing guess; the binary search where that
// misses by more than a few rows.
__device__ __forceinline__ int64_t seg_index(const double *__restrict__ rv, int64_t n, double d, double inv_dr) {
    const double gf = d * inv_dr;
    int64_t lo = 0, hi = n, g = gf > 0.0 ? (gf < (double)n ? (int64_t)gf : n) : 0;
    for (int it = 0; it < 4; ++it) {
        if (g < n && rv[g] < d) {
            lo = ++g;
        } else if (g > 0 && !(rv[g - 1] < d)) {
            hi = --g;
        } else {
            return g;
        }
    }
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (rv[mid] < d)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// One group of 8 lanes per particle over its CSR row (N = 200,000, 12 million pairs: 1.75 ms and 0.39 for the float64
// copy of the list before, 1.21 ms with the slopes from a table, the guessed index, no division and the list read as it
// is; 1.04 with the part along the particle's own moment summed as a scalar and one multiply-add a term).  T: the pair
// data's type; the double-float list of a system that has made no float64 copy is read as it is, its values joined by
// one float64 addition each.
template <typename T>
__global__ void __launch_bounds__(256) k_rs_force(const double *__restrict__ m, int64_t n,
                                                  const int64_t *__restrict__ row_ptr, PairData<T> pd,
                                                  const double2 *__restrict__ slope, const double *__restrict__ rv,
                                                  int64_t ntab, const int32_t *__restrict__ order,
                                                  double *__restrict__ F, int *__restrict__ err) {
    constexpr int G = 8;
    const int lane = threadIdx.x % G;
    const int oc = warp_sums_index<4, G / 2>(lane);   // the sum this lane holds at the end
    const int64_t grp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int64_t ngrp = ((int64_t)gridDim.x * blockDim.x) / G;
    const double inv_dr = slope[0].x;
    for (int64_t i0 = grp; i0 < n; i0 += ngrp) {
        const int64_t a = order ? (int64_t)order[i0] : i0;
        const double amx = m[3 * a], amy = m[3 * a + 1], amz = m[3 * a + 2];
        double f[4] = {0.0, 0.0, 0.0, 0.0};   // the force without its part along the particle's own moment; that part
        for (int64_t e = row_ptr[a] + lane; e < row_ptr[a + 1]; e += G) {
            const int32_t b = pd.nbr[e];
            const double d = (double)pd.dist[e];
            const int64_t i = seg_index(rv, ntab, d, inv_dr);
            if (i <= 0 || i >= ntab) {
                atomicExch(err, 1);
                continue;
            }
            const double2 sl = slope[i];
            const double BA = (double)pd.BA[e];
            const double rx = (double)pd.rx[e], ry = (double)pd.ry[e], rz = (double)pd.rz[e];
            const double mbx = m[3 * b], mby = m[3 * b + 1], mbz = m[3 * b + 2];
            const double ar = amx * rx + amy * ry + amz * rz;
            const double br = mbx * rx + mby * ry + mbz * rz;
            const double ab = amx * mbx + amy * mby + amz * mbz;
            double inv = (double)(1.0f / (float)d);   // Newton from the float32 reciprocal: two steps reach float64
            inv = inv * (2.0 - d * inv);
            inv = inv * (2.0 - d * inv);
            const double s = BA * inv, arbr = ar * br;
            // grad_r [A (ma.mb) + (B - A)(ma.r)(mb.r)]
            const double cr = sl.x * ab + (sl.y - sl.x - 2.0 * s) * arbr;
            const double sb = s * br, sa = s * ar;
            f[0] -= cr * rx;
            f[1] -= cr * ry;
            f[2] -= cr * rz;
            f[0] -= sa * mbx;
            f[1] -= sa * mby;
            f[2] -= sa * mbz;
            f[3] -= sb;
        }
        const double v = warp_sums<4, G / 2>(f, lane), own = __shfl_sync(0xffffffffu, v, 6, G);   // lane 6 holds f[3]
        if (oc >= 0 && oc < 3) F[3 * a + oc] = v + own * (oc == 0 ? amx : (oc == 1 ? amy : amz));
    }
}

// Half-away-from-zero rounding, as the grid geometry uses.
__device__ __forceinline__ double round_half_away(double v) {
    const double a = floor(fabs(v) + 0.5);
    return v > 0 ? a : (v < 0 ? -a : 0.0 * a);
}

// g[a][d][j] = -(4 xi^2 / eta_d) r_d w_d, the derivative of the Gaussian factor w_d with respect to r_d = node - x.
__global__ void k_wave_factors(const double *__restrict__ x, int64_t n, const double *__restrict__ w, GridParams gp,
                               double *__restrict__ g) {
    const int P = gp.P, lo = (P - 1) / 2;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n * 3; t += (int64_t)gridDim.x * blockDim.x) {
        const int d = (int)(t % 3);
        const double h = gp.h[d], xv = x[t];
        const double base = __dsub_rn(__dmul_rn(round_half_away(__ddiv_rn(xv, h)), h), xv);
        const double c = -4.0 * gp.xi * gp.xi / gp.eta[d];
        for (int j = 0; j < P; ++j) g[t * P + j] = c * (base + (double)(j - lo) * h) * w[t * P + j];
    }
}

// Wave-space part: warp per particle (in the visiting order) over its P^3 stencil; phi = the three convolved component
// grids of one vector.  A node costs five float64 multiply-adds -- m . phi, and its sums along z with w_z and with its
// derivative -- where the position vector at every node cost thirteen (N = 200,000, P = 10: 5.27 -> 2.07 ms).
__global__ void __launch_bounds__(128) k_wave_force(const double *__restrict__ phi, const double *__restrict__ m,
                                                    int64_t n, const int32_t *__restrict__ start,
                                                    const double *__restrict__ w, const double *__restrict__ g,
                                                    GridParams gp, double *__restrict__ F) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int P = gp.P;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const int64_t G = gp.G, plane = (int64_t)Nx * Ny;
    for (int64_t i = warp; i < n; i += nw) {
        const int64_t a = gp.order ? (int64_t)gp.order[i] : i;
        const int sx = start[3 * a], sy = start[3 * a + 1], sz = start[3 * a + 2];
        const double *wa = w + a * 3 * P, *ga = g + a * 3 * P;
        const double mx = m[3 * a], my = m[3 * a + 1], mz = m[3 * a + 2];
        double fx = 0.0, fy = 0.0, fz = 0.0;
        for (int row0 = 0; row0 < P * P; row0 += 32) {
            int idx, sub, lpp;
            if (!stencil_row(row0, P, lane, &idx, &sub, &lpp)) continue;
            const int jx = idx % P, jy = idx / P;
            int ix = sx + jx;
            if (ix >= Nx) ix -= Nx;
            int iy = sy + jy;
            if (iy >= Ny) iy -= Ny;
            const double *pr = phi + ix + (int64_t)Nx * iy;
            double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
            for (int jz = sub; jz < P; jz += lpp) {
                int iz = sz + jz;
                if (iz >= Nz) iz -= Nz;
                const double *p = pr + plane * iz;
                const double v = mx * p[0] + my * p[G] + mz * p[2 * G];
                s0 += wa[2 * P + jz] * v;
                s1 += ga[2 * P + jz] * v;
            }
            const double wx = wa[jx], wy = wa[P + jy];
            fx += ga[jx] * wy * s0;
            fy += wx * ga[P + jy] * s0;
            fz += wx * wy * s1;
        }
        const double v = warp_sum4(fx, fy, fz, 0.0, lane);
        if ((lane & 7) == 0 && lane < 24) F[3 * a + lane / 8] += gp.hprod * v;
    }
}

// dD/d eps = -3 / (4 pi (eps - 1)^2) = -(4 pi / 3) (D - self)^2, from the stored diagonal.
__global__ void k_eps_grad(const double *__restrict__ m, const double *__restrict__ diag, double self, int64_t n,
                           double *__restrict__ dE) {
    for (int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; a < n; a += (int64_t)gridDim.x * blockDim.x) {
        const double m2 = m[3 * a] * m[3 * a] + m[3 * a + 1] * m[3 * a + 1] + m[3 * a + 2] * m[3 * a + 2];
        const double dl = diag[a] - self;
        dE[a] = 0.5 * m2 * (-(4.0 * MPS_PI / 3.0) * dl * dl);
    }
}

template <typename T>
int rs_force(const double *m, int64_t n, const int64_t *row_ptr, const PairData<T> &pd, const double *perp,
             const double *para, const double *rv, int64_t ntab, double2 *slopes, const int32_t *order, double *F,
             int *err, cudaStream_t s) {
    k_table_slopes<<<grid_for(ntab, 256), 256, 0, s>>>(perp, para, rv, ntab, slopes);
    MPS_LAUNCH_CHECK();
    k_rs_force<T><<<grid_for(n * 8, 256, 152 * 64), 256, 0, s>>>(m, n, row_ptr, pd, slopes, rv, ntab, order, F, err);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}
template int rs_force<double>(const double *, int64_t, const int64_t *, const PairData<double> &, const double *,
                              const double *, const double *, int64_t, double2 *, const int32_t *, double *, int *,
                              cudaStream_t);
template int rs_force<dfv>(const double *, int64_t, const int64_t *, const PairData<dfv> &, const double *,
                           const double *, const double *, int64_t, double2 *, const int32_t *, double *, int *,
                           cudaStream_t);

int wave_force(const double *phi, const double *x, const double *m, int64_t n, const int32_t *start, const double *w,
               double *g, const GridParams &gp, double *F, cudaStream_t s) {
    k_wave_factors<<<grid_for(3 * n, 256), 256, 0, s>>>(x, n, w, gp, g);
    MPS_LAUNCH_CHECK();
    k_wave_force<<<grid_for(n * 32, 128, 152 * 128), 128, 0, s>>>(phi, m, n, start, w, g, gp, F);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int eps_grad(const double *m, const double *diag, double self, int64_t n, double *dE, cudaStream_t s) {
    k_eps_grad<<<grid_for(n, 256), 256, 0, s>>>(m, diag, self, n, dE);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

}  // namespace mps
