// Dipole + quadrupole operator: 8 moments per sphere, S (x, y, z) and the
// traceless quadrupole Q stored as (xx, xy, xz, yy, yz), zz = -(xx + yy)
// (Capacitance_Quadrupole/MatrixVectorMultiply.m:31-77).
//
//   spread / contract   the dipole path's Gaussian on 8 component grids
//                       (CQ/Spread.m:41-71, CQ/Contract.m:49-77)
//   scale               E~ = (HES k.fS + HEQ Qd.fQ) k,  G~ = (HGS k.fS + HGQ Qd.fQ) Qf
//                       with HES = 9 j1^2, HEQ = -45/2 i j1 j2, HGS = 45 i j2 j1,
//                       HGQ = 225/2 j2^2, times exp(-sum(1-eta)k^2/4xi^2)/k^2
//                       (CQ/Scale.m:19-72); on the half spectrum of real grids
//                       the unpaired Nyquist bins get the average of the
//                       coupling at k and at its conjugate partner (the real
//                       part of the reference's complex pipeline)
//   real space          nine interpolated couplings per pair (CQ/RealSpace.m:27-100)
#include <math.h>

#include "quad.cuh"

#include <algorithm>

namespace mps {

__device__ __forceinline__ double to_double(float v) { return float_to_double(v); }
__device__ __forceinline__ double to_double(double v) { return v; }

// ---------------------------------------------------------------------------
// Spread / contract for ncomp (<= 8) moment components per particle.
// ---------------------------------------------------------------------------
// Spread: a warp to a particle and vector or, SPLIT, to every parts-th pass over its (x, y) rows, 32 rows at a time
// (spread_parts).
template <typename T, bool SPLIT>
__global__ void __launch_bounds__(256) k_spread_gen(const double *__restrict__ m, int64_t n, int nrhs, int ncomp,
                                                    int parts, const int32_t *__restrict__ start,
                                                    const T *__restrict__ w, GridParams gp, T *__restrict__ grid) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int P = gp.P;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const int64_t G = gp.G;
    if (!SPLIT) parts = 1;
    for (int64_t u = warp; u < n * nrhs * parts; u += nw) {
        const int64_t t = SPLIT ? u / parts : u;
        const int part = (int)(u - t * parts);
        const int64_t a = gp.order ? (int64_t)gp.order[t % n] : t % n;
        const int r = (int)(t / n);
        const int sx = start[3 * a], sy = start[3 * a + 1], sz = start[3 * a + 2];
        const T *wa = w + a * 3 * P;
        T mv[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) mv[c] = c < ncomp ? (T)m[((int64_t)r * n + a) * ncomp + c] : (T)0;
        T *g0 = grid + (int64_t)r * ncomp * G;
        for (int row0 = 32 * part; row0 < P * P; row0 += 32 * parts) {
            int idx, sub, lpp;
            if (!stencil_row(row0, P, lane, &idx, &sub, &lpp)) continue;
            const int jx = idx % P, jy = idx / P;
            int ix = sx + jx;
            if (ix >= Nx) ix -= Nx;
            int iy = sy + jy;
            if (iy >= Ny) iy -= Ny;
            const T wxy = wa[jx] * wa[P + jy];
            const int64_t rowb = (int64_t)ix + (int64_t)Nx * iy;
            for (int jz = sub; jz < P; jz += lpp) {
                int iz = sz + jz;
                if (iz >= Nz) iz -= Nz;
                const T wv = wxy * wa[2 * P + jz];
                const int64_t node = rowb + (int64_t)Nx * Ny * iz;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if (c < ncomp) atomicAdd(g0 + c * G + node, wv * mv[c]);
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_contract_gen(const T *__restrict__ grid, int64_t n, int nrhs, int ncomp,
                                                      const int32_t *__restrict__ start, const T *__restrict__ w,
                                                      GridParams gp, double *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int P = gp.P;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const int64_t G = gp.G;
    const int oc = warp_sums_index<8>(lane);   // the component this lane writes
    for (int64_t t = warp; t < n * nrhs; t += nw) {
        const int64_t a = gp.order ? (int64_t)gp.order[t % n] : t % n;
        const int r = (int)(t / n);
        const int sx = start[3 * a], sy = start[3 * a + 1], sz = start[3 * a + 2];
        const T *wa = w + a * 3 * P;
        const T *g0 = grid + (int64_t)r * ncomp * G;
        T acc[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] = (T)0;
        for (int row0 = 0; row0 < P * P; row0 += 32) {
            int idx, sub, lpp;
            if (!stencil_row(row0, P, lane, &idx, &sub, &lpp)) continue;
            const int jx = idx % P, jy = idx / P;
            int ix = sx + jx;
            if (ix >= Nx) ix -= Nx;
            int iy = sy + jy;
            if (iy >= Ny) iy -= Ny;
            const T wxy = wa[jx] * wa[P + jy];
            const int64_t rowb = (int64_t)ix + (int64_t)Nx * iy;
            for (int jz = sub; jz < P; jz += lpp) {
                int iz = sz + jz;
                if (iz >= Nz) iz -= Nz;
                const T wv = wxy * wa[2 * P + jz];
                const int64_t node = rowb + (int64_t)Nx * Ny * iz;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if (c < ncomp) acc[c] += wv * g0[c * G + node];
            }
        }
        const T v = warp_sums(acc, lane);
        if (oc >= 0 && oc < ncomp) out[((int64_t)r * n + a) * ncomp + oc] = to_double(v) * gp.hprod;
    }
}

// Contraction of the eight float32 grids of a vector by home blocks: a block takes the particles whose stencils start
// in one 8^3 block of nodes and four of the components; it stages the nodes that they reach, the block grown by P - 1
// per axis, as float4 (the four components side by side), then a warp per particle sums over its stencil from shared
// memory, the lanes on the P^2 columns.  Rows of P + 8 nodes: consecutive columns of a warp then lie 16 bytes apart
// modulo the banks, whatever P.  The gather from the grids (k_contract_gen) reads a line per row, plane and component
// of every particle through L1, which bounds it; here the staging does (the blocks' chains of loads).  N = 50,320, 90 x
// 90 x 96, P = 6: 96 us by the gather (with its sums converted by one lane), 60 so (with an interleaved copy of the
// grids, staged 16 bytes at a time or gathered from, 63 and 68).
constexpr int kHome8Chunk = 32;
constexpr int kHome8Warps = 8;

__global__ void __launch_bounds__(kHome8Warps * 32, 5) k_contract_home8(
    const float *__restrict__ grid, int64_t n, const int64_t *__restrict__ hstart,
    const int32_t *__restrict__ hentries, int nbx, int nby, const int32_t *__restrict__ start,
    const float *__restrict__ w, GridParams gp, double *__restrict__ out) {
    const int P = gp.P, F = 3 * P;
    const int R = kHomeBlock + P - 1, RS = R + 1, RP = R * RS;   // nodes per axis, row and plane strides
    extern __shared__ float4 s_reg4[];                            // [R][R][RS]
    float *s_w = (float *)(s_reg4 + R * RP);                      // [kHome8Chunk][3 P]
    int *s_p = (int *)(s_w + kHome8Chunk * F);                    // [kHome8Chunk][2]: first node in the region, particle id
    const int64_t hb = blockIdx.x;
    const int64_t e0 = hstart[hb], e1 = hstart[hb + 1];
    if (e0 == e1) return;   // the whole block leaves: no barrier is left waiting
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const int X0 = (int)(hb % nbx) * kHomeBlock, Y0 = (int)((hb / nbx) % nby) * kHomeBlock,
              Z0 = (int)(hb / ((int64_t)nbx * nby)) * kHomeBlock;
    const int r = blockIdx.y >> 1, c0 = 4 * (blockIdx.y & 1);
    const int64_t G = gp.G;
    const float *g0 = grid + (int64_t)blockIdx.y * 4 * G;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // origin + offset < 3 N (the host requires N >= 8 and N >= P): at most two wraps
    auto wrap2 = [](int i, int N) {
        i -= i >= N ? N : 0;
        return i - (i >= N ? N : 0);
    };
    const int LX = R <= 16 ? 16 : 32, x = lane & (LX - 1);
    if (x < R) {
        const float *gx = g0 + wrap2(X0 + x, Nx);
        const int rpw = 32 / LX;   // rows a warp takes at a time
        for (int row = wid * rpw + lane / LX; row < R * R; row += kHome8Warps * rpw) {
            const int z = row / R, y = row - z * R;
            const float *src = gx + ((int64_t)wrap2(Z0 + z, Nz) * Ny + wrap2(Y0 + y, Ny)) * Nx;
            float *dst = (float *)(s_reg4 + row * RS + x);
#pragma unroll
            for (int c = 0; c < 4; ++c) copy_async(dst + c, src + c * G);
        }
    }
    const int full = P * P / 32 * 32, rem = P * P - full;   // columns of the whole rounds and of the last one,
    const int lz = rem ? 32 / rem : 1;                      // whose lanes share a column's planes
    const int lcol = rem ? full + lane / lz : 0, lsub = lane - lane / lz * lz;
    const int ljy = lcol / P, ljx = lcol - ljy * P;
    const int oc = warp_sums_index<4>(lane);
    for (int64_t b0 = e0; b0 < e1; b0 += kHome8Chunk) {
        const int cnt = (int)min((int64_t)kHome8Chunk, e1 - b0);
        for (int q = threadIdx.x; q < cnt * F; q += kHome8Warps * 32) {
            const int p = q / F;
            s_w[q] = w[(int64_t)hentries[b0 + p] * F + (q - p * F)];
        }
        if (threadIdx.x < cnt) {
            const int32_t a = hentries[b0 + threadIdx.x];
            const int32_t *sa = start + 3 * (int64_t)a;
            s_p[2 * threadIdx.x] = (sa[2] - Z0) * RP + (sa[1] - Y0) * RS + sa[0] - X0;
            s_p[2 * threadIdx.x + 1] = a;
        }
        copy_async_wait();
        __syncthreads();   // the region (first pass) and this chunk's particles are in place
        for (int p = wid; p < cnt; p += kHome8Warps) {
            const float *wa = s_w + p * F;
            const float4 *base = s_reg4 + s_p[2 * p];
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            for (int q = lane; q < full; q += 32) {
                const int jy = q / P, jx = q - jy * P;
                const float4 *col = base + jy * RS + jx;
                float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
                for (int jz = 0; jz < P; ++jz) {
                    const float wz = wa[2 * P + jz];
                    const float4 v = col[jz * RP];
                    s[0] += wz * v.x;
                    s[1] += wz * v.y;
                    s[2] += wz * v.z;
                    s[3] += wz * v.w;
                }
                const float wxy = wa[jx] * wa[P + jy];
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[c] += wxy * s[c];
            }
            if (rem && lcol < P * P) {
                const float4 *col = base + ljy * RS + ljx;
                const float wxy = wa[ljx] * wa[P + ljy];
                for (int jz = lsub; jz < P; jz += lz) {
                    const float wv = wxy * wa[2 * P + jz];
                    const float4 v = col[jz * RP];
                    acc[0] += wv * v.x;
                    acc[1] += wv * v.y;
                    acc[2] += wv * v.z;
                    acc[3] += wv * v.w;
                }
            }
            __syncwarp();
            const float v = warp_sums(acc, lane);
            if (oc >= 0) out[((int64_t)r * n + s_p[2 * p + 1]) * 8 + c0 + oc] = float_to_double(v) * gp.hprod;
        }
        __syncthreads();   // this chunk's particles are read before the next overwrites them
    }
}

// ---------------------------------------------------------------------------
// Wave space
// ---------------------------------------------------------------------------
// The couplings depend on k only through its components' squares: worked out once for the quarter spectrum and written
// for its mirror images.  The float32 table holds the unit wave vector too (the float64 square root and division of a
// point cost the float32 scale kernel more than reading 16 bytes: 25 -> 12 us on 90 x 90 x 96); the float64 kernel
// works it out.
__global__ void k_quad_kcoef(GridParams gp, double *__restrict__ c64, float4 *__restrict__ c32) {
    const HalfQuarter hq(gp.N);
    const double invG = 1.0 / (double)gp.G;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < hq.size();
         t += (int64_t)gridDim.x * blockDim.x) {
        int ix, iy, iz;
        hq.point(t, &ix, &iy, &iz);
        const double kx = fft_freq(ix, gp.N[0]) * gp.kfac[0];
        const double ky = fft_freq(iy, gp.N[1]) * gp.kfac[1];
        const double kz = fft_freq(iz, gp.N[2]) * gp.kfac[2];
        const double k2 = kx * kx + ky * ky + kz * kz;
        double v[4] = {0, 0, 0, 0};
        float q[3] = {0, 0, 0};
        if (k2 > 0) {
            const double k = sqrt(k2);
            const double s = sin(k), c = cos(k);
            const double j1 = s / k2 - c / k;
            const double j2 = (3.0 / k2 - 1.0) * s / k - 3.0 * c / k2;
            const double etak2 = (1 - gp.eta[0]) * kx * kx + (1 - gp.eta[1]) * ky * ky + (1 - gp.eta[2]) * kz * kz;
            const double g = exp(-etak2 / (4 * gp.xi * gp.xi)) / k2 * invG;
            v[0] = 9.0 * j1 * j1 * g;        // HES
            v[1] = -22.5 * j1 * j2 * g;      // HEQ / i
            v[2] = 45.0 * j2 * j1 * g;       // HGS / i
            v[3] = 112.5 * j2 * j2 * g;      // HGQ
            for (int i = 0; i < 4; ++i)
                if (!isfinite(v[i])) v[i] = 0.0;
            const double inv = 1.0 / k;
            q[0] = (float)(kx * inv);
            q[1] = (float)(ky * inv);
            q[2] = (float)(kz * inv);
        }
        const float4 lo = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
        mirror_points(hq, ix, iy, iz, [&](int64_t lin, int sy, int sz) {
            for (int i = 0; i < 4; ++i) c64[4 * lin + i] = v[i];
            if (c32) {
                c32[2 * lin] = lo;
                c32[2 * lin + 1] = make_float4(q[0], sy * q[1], sz * q[2], 0.f);
            }
        });
    }
}

template <typename T>
struct C2T;
template <>
struct C2T<float> {
    using type = float2;
};
template <>
struct C2T<double> {
    using type = double2;
};

// out = M(q) f for unit wave vector q; cconj flips the imaginary couplings.
template <typename T, typename C>
__device__ __forceinline__ void quad_couple(const T q[3], const T cf[4], bool cconj, const C f[8], C out[8]) {
    const T qd[5] = {q[0] * q[0] - q[2] * q[2], 2 * q[0] * q[1], 2 * q[0] * q[2], q[1] * q[1] - q[2] * q[2],
                     2 * q[1] * q[2]};
    const T qf[5] = {q[0] * q[0] - (T)(1.0 / 3.0), q[0] * q[1], q[0] * q[2], q[1] * q[1] - (T)(1.0 / 3.0),
                     q[1] * q[2]};
    C dS, dQ;
    dS.x = q[0] * f[0].x + q[1] * f[1].x + q[2] * f[2].x;
    dS.y = q[0] * f[0].y + q[1] * f[1].y + q[2] * f[2].y;
    dQ.x = dQ.y = (T)0;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        dQ.x += qd[k] * f[3 + k].x;
        dQ.y += qd[k] * f[3 + k].y;
    }
    const T eq = cconj ? -cf[1] : cf[1];
    const T gs = cconj ? -cf[2] : cf[2];
    // a = HES dS + i eq dQ ; b = i gs dS + HGQ dQ
    C a, b;
    a.x = cf[0] * dS.x - eq * dQ.y;
    a.y = cf[0] * dS.y + eq * dQ.x;
    b.x = -gs * dS.y + cf[3] * dQ.x;
    b.y = gs * dS.x + cf[3] * dQ.y;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        out[k].x = a.x * q[k];
        out[k].y = a.y * q[k];
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        out[3 + k].x = b.x * qf[k];
        out[3 + k].y = b.y * qf[k];
    }
}

template <typename T>
__global__ void k_scale_quad(typename C2T<T>::type *__restrict__ spec, int nrhs, GridParams gp,
                             const T *__restrict__ coef, T factor) {
    using C = typename C2T<T>::type;
    const int Nxh = gp.N[0] / 2 + 1;
    const int64_t Gc = (int64_t)Nxh * gp.N[1] * gp.N[2];
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < Gc; t += (int64_t)gridDim.x * blockDim.x) {
        const int ix = (int)(t % Nxh);
        const int iy = (int)((t / Nxh) % gp.N[1]);
        const int iz = (int)(t / ((int64_t)Nxh * gp.N[1]));
        T q[3] = {0, 0, 0}, cf[4];
        if constexpr (sizeof(T) == 4) {
            const float4 *c4 = (const float4 *)coef + 2 * t;
            const float4 lo = c4[0], hi = c4[1];
            cf[0] = factor * lo.x;
            cf[1] = factor * lo.y;
            cf[2] = factor * lo.z;
            cf[3] = factor * lo.w;
            q[0] = hi.x;
            q[1] = hi.y;
            q[2] = hi.z;
        } else {
            const double kx = fft_freq(ix, gp.N[0]) * gp.kfac[0];
            const double ky = fft_freq(iy, gp.N[1]) * gp.kfac[1];
            const double kz = fft_freq(iz, gp.N[2]) * gp.kfac[2];
            const double k2 = kx * kx + ky * ky + kz * kz;
            if (k2 > 0) {
                const double inv = 1.0 / sqrt(k2);
                q[0] = kx * inv;
                q[1] = ky * inv;
                q[2] = kz * inv;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) cf[i] = factor * coef[4 * t + i];
        }
        const bool ny[3] = {(gp.N[0] % 2 == 0) && ix == gp.N[0] / 2, (gp.N[1] % 2 == 0) && iy == gp.N[1] / 2,
                            (gp.N[2] % 2 == 0) && iz == gp.N[2] / 2};
        const bool nyq = ny[0] || ny[1] || ny[2];
        // conjugate partner: non-Nyquist components flip sign
        const T qp[3] = {ny[0] ? q[0] : -q[0], ny[1] ? q[1] : -q[1], ny[2] ? q[2] : -q[2]};
        for (int r = 0; r < nrhs; ++r) {
            C *s = spec + (int64_t)(8 * r) * Gc + t;
            C f[8], o1[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) f[c] = s[c * Gc];
            quad_couple<T, C>(q, cf, false, f, o1);
            if (nyq) {
                C o2[8];
                quad_couple<T, C>(qp, cf, true, f, o2);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    o1[c].x = (T)0.5 * (o1[c].x + o2[c].x);
                    o1[c].y = (T)0.5 * (o1[c].y + o2[c].y);
                }
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) s[c * Gc] = o1[c];
        }
    }
}

// ---------------------------------------------------------------------------
// Real space
// ---------------------------------------------------------------------------
__device__ __forceinline__ void load8(const float *__restrict__ p, float v[8]) {   // 32-byte aligned rows
    const float4 a = ((const float4 *)p)[0], b = ((const float4 *)p)[1];
    v[0] = a.x;
    v[1] = a.y;
    v[2] = a.z;
    v[3] = a.w;
    v[4] = b.x;
    v[5] = b.y;
    v[6] = b.z;
    v[7] = b.w;
}
__device__ __forceinline__ void load8(const double *__restrict__ p, double v[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = p[i];
}

__device__ __forceinline__ int64_t qsearch(const double *__restrict__ rv, int64_t n, double d, double inv_dr) {
    double gf = d * inv_dr;
    int64_t g = gf < 0 ? 0 : (gf > (double)(n - 1) ? n - 1 : (int64_t)gf);
    for (int it = 0; it < 64; ++it) {
        if (g < n && rv[g] < d) {
            ++g;
            continue;
        }
        if (g > 0 && rv[g - 1] >= d) {
            --g;
            continue;
        }
        return g;
    }
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

// coef[9][np] = (A, B, C, D, E, F, G, H, I) interpolated at the pair separations.
__global__ void k_quad_pair_coefs(const double *__restrict__ dist, int64_t np, const double *__restrict__ perp,
                                  const double *__restrict__ para, const double *__restrict__ qt,
                                  const double *__restrict__ rv, int64_t ntab, double inv_dr,
                                  double *__restrict__ c64, float *__restrict__ c32, int *__restrict__ err) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np; p += (int64_t)gridDim.x * blockDim.x) {
        const double d = dist[p];
        const int64_t i = qsearch(rv, ntab, d, inv_dr);
        double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        if (i <= 0 || i >= ntab) {
            atomicExch(err, 1);
        } else {
            const double t = (d - rv[i - 1]) / (rv[i] - rv[i - 1]);
            const double u = 1.0 - t;
            v[0] = perp[i - 1] * u + perp[i] * t;
            v[1] = para[i - 1] * u + para[i] * t;
            for (int k = 0; k < 7; ++k) v[2 + k] = qt[k * ntab + i - 1] * u + qt[k * ntab + i] * t;
        }
        for (int k = 0; k < 9; ++k) {
            c64[k * np + p] = v[k];
            if (c32) c32[k * np + p] = (float)v[k];
        }
    }
}

// Float32 copy of the moments for the pair sum: a pair converts nothing (eight conversions a pair on the float64 pipe
// had been two thirds of the float32 sum) and gathers two aligned float4 instead of eight doubles.
__global__ void k_moments8(const double *__restrict__ m, int64_t total, float *__restrict__ m32) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
        m32[i] = (float)m[i];
}

// mp: the moments the pairs read (T), m: those of the diagonal.  G lanes to a row, its pairs in turn; the couplings are
// nine arrays of n_pairs, so a row's reads are contiguous.  The row's eight sums end one to a lane.  3 million pairs in
// 50,320 rows: 79 us with the conversions, 48 so (memory bound at 26; a warp to a row took 66).
template <typename T, int G>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) k_rs_quad(const double *__restrict__ m, const T *__restrict__ mp,
                                                 double *__restrict__ out, int64_t n,
                                                 int nrhs, int64_t np, const int64_t *__restrict__ row_ptr,
                                                 const int32_t *__restrict__ nbr, const T *__restrict__ rxs,
                                                 const T *__restrict__ rys, const T *__restrict__ rzs,
                                                 const T *__restrict__ coef, const double *__restrict__ diagS,
                                                 const double *__restrict__ diagQ,
                                                 const int32_t *__restrict__ diag_of_rhs) {
    const int lane = threadIdx.x % G;
    const int oc = warp_sums_index<8, G / 2>(lane);
    const int64_t grp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int64_t ngrp = ((int64_t)gridDim.x * blockDim.x) / G;
    // every lane of a warp walks its rows the same number of times: the sums at the end take all of them
    const int64_t trips = (n * nrhs + ngrp - 1) / ngrp;
    for (int64_t it = 0; it < trips; ++it) {
        const int64_t t = it * ngrp + grp;
        const bool on = t < n * nrhs;
        const int64_t a = on ? t % n : 0;
        const int r = on ? (int)(t / n) : 0;
        T acc[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] = (T)0;
        const int64_t e1 = on ? row_ptr[a + 1] : 0;
        int64_t e = on ? row_ptr[a] + lane : 0;
        int32_t next = e < e1 ? nbr[e] : 0;
        // what the row's end takes, loaded before its pairs
        const bool wr = on && oc >= 0;
        const int64_t di0 = (int64_t)(diag_of_rhs && on ? diag_of_rhs[r] : 0) * n + a, o = ((int64_t)r * n + a) * 8 + oc;
        const double d = wr ? (oc < 3 ? diagS[di0] : diagQ[di0]) : 0.0, mo = wr ? m[o] : 0.0, prev = wr ? out[o] : 0.0;
        for (; e < e1; e += G) {
            const int32_t b = next;
            next = e + G < e1 ? nbr[e + G] : 0;   // the neighbour's moments wait for its id only once a row
            const T rx = rxs[e], ry = rys[e], rz = rzs[e];
            const T *cf = coef + e;
            const T A = cf[0], B = cf[np], Cc = cf[2 * np], D = cf[3 * np], E = cf[4 * np], F = cf[5 * np],
                    Gg = cf[6 * np], H = cf[7 * np], I = cf[8 * np];
            T mb[8];
            load8(mp + ((int64_t)r * n + b) * 8, mb);
            const T Sx = mb[0], Sy = mb[1], Sz = mb[2];
            const T Q0 = mb[3], Q1 = mb[4], Q2 = mb[5], Q3 = mb[6], Q4 = mb[7];
            const T sr = Sx * rx + Sy * ry + Sz * rz;
            const T Qr0 = Q0 * rx + Q1 * ry + Q2 * rz;
            const T Qr1 = Q1 * rx + Q3 * ry + Q4 * rz;
            const T Qr2 = Q2 * rx + Q4 * ry - (Q0 + Q3) * rz;
            const T rQr = Q0 * (rx * rx - rz * rz) + 2 * Q1 * rx * ry + 2 * Q2 * rx * rz + Q3 * (ry * ry - rz * rz) +
                          2 * Q4 * ry * rz;
            // field: A S + (B-A)(S.r) r - (C rQr r)/2 - D Q.r
            const T sE = (B - A) * sr - (T)0.5 * Cc * rQr;
            acc[0] += A * Sx;
            acc[1] += A * Sy;
            acc[2] += A * Sz;
            acc[0] += sE * rx;
            acc[1] += sE * ry;
            acc[2] += sE * rz;
            acc[0] -= D * Qr0;
            acc[1] -= D * Qr1;
            acc[2] -= D * Qr2;
            // gradient, 5-component (xx, xy, xz, yy, yz)
            const T q5[5] = {rx * rx, rx * ry, rx * rz, ry * ry, ry * rz};
            const T srs[5] = {2 * Sx * rx, Sx * ry + rx * Sy, Sx * rz + rx * Sz, 2 * Sy * ry, Sy * rz + ry * Sz};
            const T qq[5] = {4 * Qr0 * rx, 2 * (Qr0 * ry + rx * Qr1), 2 * (Qr0 * rz + rx * Qr2), 4 * Qr1 * ry,
                             2 * (Qr1 * rz + ry * Qr2)};
            const T Qv[5] = {Q0, Q1, Q2, Q3, Q4};
            const T cq = Cc * sr + (T)0.5 * I * rQr;
            const T di = (D + E) * sr + (T)0.5 * (F + H) * rQr;
            const T hG = (T)0.5 * Gg, hH = (T)0.5 * H;
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                acc[3 + k] += cq * q5[k];
                acc[3 + k] += D * srs[k];
                acc[3 + k] += hG * Qv[k];
                acc[3 + k] += hH * qq[k];
                if (k == 0 || k == 3) acc[3 + k] += di;
            }
        }
        const T v = warp_sums<8, G / 2>(acc, lane);
        if (wr) out[o] = prev + (d * mo + to_double(v));
    }
}

// Gradient/quadrupole diagonal: 15 / (8 pi (eps - 1)) + grad_quad_2(0) / 2
// (CQ/MatrixVectorMultiply.m and CQ/RealSpace.m self terms).
__global__ void k_quad_diag(const double *__restrict__ lam, int64_t total, double self_q, double *__restrict__ diag) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
        diag[i] = 15.0 / (8.0 * MPS_PI * (lam[i] - 1.0)) + 0.5 * self_q;
}

// ---------------------------------------------------------------------------
// Host wrappers
// ---------------------------------------------------------------------------
// Warps to a particle and vector: a stencil of many rows is a long chain of atomics, and few particles leave most SMs
// without one; its passes over 32 rows go to warps of their own while the GPU has room for them (64 to an SM).
static int spread_parts(int64_t items, int P) {
    const int64_t room = 152 * 64 / std::max<int64_t>(items, 1);
    return (int)std::max<int64_t>(1, std::min<int64_t>(room, (P * P + 31) / 32));
}

template <typename T>
int spread_gen(const double *m, int64_t n, int nrhs, int ncomp, const int32_t *start, const T *w,
               const GridParams &gp, T *grid, cudaStream_t s) {
    MPS_CUDA_TRY(cudaMemsetAsync(grid, 0, sizeof(T) * (size_t)ncomp * nrhs * gp.G, s));
    const int parts = spread_parts(n * nrhs, gp.P);
    const auto kernel = parts > 1 ? k_spread_gen<T, true> : k_spread_gen<T, false>;
    kernel<<<grid_for(n * nrhs * parts * 32, 256, 152 * 64), 256, 0, s>>>(m, n, nrhs, ncomp, parts, start, w, gp, grid);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template <typename T>
int contract_gen(const T *grid, int64_t n, int nrhs, int ncomp, const int32_t *start, const T *w,
                 const GridParams &gp, double *out, cudaStream_t s) {
    k_contract_gen<T><<<grid_for(n * nrhs * 32, 256, 152 * 64), 256, 0, s>>>(grid, n, nrhs, ncomp, start, w, gp, out);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

// The staging costs so much a block, the gather so much a particle; on 96^3 with P = 6 (10) 33 us and 0.53 a thousand
// particles (87 and 1.8) against 1.8 (5.0) a thousand: even at 16 particles a block.
bool contract_home8_pays(const GridParams &gp, int64_t n) {
    if (gp.P > kMaxP) return false;
    int64_t blocks = 1;
    for (int d = 0; d < 3; ++d) {
        if (gp.N[d] < kHomeBlock || gp.N[d] < gp.P) return false;
        blocks *= (gp.N[d] + kHomeBlock - 1) / kHomeBlock;
    }
    return n >= 16 * blocks;
}

static size_t home8_smem(int P) {
    const size_t R = kHomeBlock + P - 1;
    return sizeof(float4) * R * R * (R + 1) + sizeof(float) * kHome8Chunk * 3 * P + sizeof(int) * 2 * kHome8Chunk;
}

int contract_home8(const float *grid, int64_t n, int nrhs, const int32_t *start, const float *w, const GridParams &gp,
                   const TileBins &tb, double *out, cudaStream_t s) {
    if (!tb.has_home) return MPS_BAD_ARG;
    const size_t smem = home8_smem(gp.P);
    // one limit for every launch (the largest support's): a thread that sets its own lower one between another's
    // request and launch would make that launch fail
    if (smem > 48 * 1024)
        MPS_CUDA_TRY(cudaFuncSetAttribute(k_contract_home8, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)home8_smem(kMaxP)));
    k_contract_home8<<<dim3((unsigned)tb.nhome, 2 * nrhs), kHome8Warps * 32, smem, s>>>(
        grid, n, tb.hstart, tb.hentries, tb.nhb[0], tb.nhb[1], start, w, gp, out);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int quad_diag(const double *lam, int64_t total, const double *gq2, double *diag, cudaStream_t s) {
    double self_q = 0.0;
    MPS_CUDA_TRY(cudaMemcpyAsync(&self_q, gq2, sizeof(double), cudaMemcpyDeviceToHost, s));
    MPS_CUDA_TRY(cudaStreamSynchronize(s));
    k_quad_diag<<<grid_for(total, 256), 256, 0, s>>>(lam, total, self_q, diag);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int quad_kcoef(const GridParams &gp, double *c64, float *c32, cudaStream_t s) {
    k_quad_kcoef<<<grid_for(HalfQuarter(gp.N).size(), 128), 128, 0, s>>>(gp, c64, (float4 *)c32);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template <typename T>
int scale_quad(void *spec, int nrhs, const GridParams &gp, const T *coef, cudaStream_t s, double factor) {
    const int64_t Gc = (int64_t)(gp.N[0] / 2 + 1) * gp.N[1] * gp.N[2];
    k_scale_quad<T><<<grid_for(Gc, 256), 256, 0, s>>>((typename C2T<T>::type *)spec, nrhs, gp, coef,
                                                        (T)factor);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int quad_pair_coefs(const double *dist, int64_t np, const double *perp, const double *para, const double *qt,
                    const double *rv, int64_t ntab, double *c64, float *c32, int *err, cudaStream_t s) {
    if (np == 0) return MPS_OK;
    double rv_last = 0.0;
    MPS_CUDA_TRY(cudaMemcpyAsync(&rv_last, rv + ntab - 1, sizeof(double), cudaMemcpyDeviceToHost, s));
    MPS_CUDA_TRY(cudaStreamSynchronize(s));
    const double inv_dr = rv_last > 0 ? (double)(ntab - 1) / rv_last : 0.0;
    k_quad_pair_coefs<<<grid_for(np, 256), 256, 0, s>>>(dist, np, perp, para, qt, rv, ntab, inv_dr, c64, c32, err);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template <typename T>
int real_space_quad(const double *m, float *m32, double *out, int64_t n, int nrhs, const int64_t *row_ptr, int64_t np,
                    const int32_t *nbr, const T *rx, const T *ry, const T *rz, const T *coef, const double *diagS,
                    const double *diagQ, const int32_t *diag_of_rhs, cudaStream_t s) {
    const T *mp;
    if constexpr (sizeof(T) == 4) {
        const int64_t total = 8 * n * nrhs;
        k_moments8<<<grid_for(total, 256), 256, 0, s>>>(m, total, m32);
        MPS_LAUNCH_CHECK();
        mp = m32;
    } else {
        mp = m;
    }
    constexpr int G = 8;
    k_rs_quad<T, G><<<grid_for(n * nrhs * G, 256, 152 * 64), 256, 0, s>>>(m, mp, out, n, nrhs, np, row_ptr, nbr, rx, ry,
                                                                          rz, coef, diagS, diagQ, diag_of_rhs);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template int spread_gen<float>(const double *, int64_t, int, int, const int32_t *, const float *, const GridParams &,
                               float *, cudaStream_t);
template int spread_gen<double>(const double *, int64_t, int, int, const int32_t *, const double *,
                                const GridParams &, double *, cudaStream_t);
template int contract_gen<float>(const float *, int64_t, int, int, const int32_t *, const float *, const GridParams &,
                                 double *, cudaStream_t);
template int contract_gen<double>(const double *, int64_t, int, int, const int32_t *, const double *,
                                  const GridParams &, double *, cudaStream_t);
template int scale_quad<float>(void *, int, const GridParams &, const float *, cudaStream_t, double);
template int scale_quad<double>(void *, int, const GridParams &, const double *, cudaStream_t, double);
template int real_space_quad<float>(const double *, float *, double *, int64_t, int, const int64_t *, int64_t,
                                    const int32_t *, const float *, const float *, const float *, const float *,
                                    const double *, const double *, const int32_t *, cudaStream_t);
template int real_space_quad<double>(const double *, float *, double *, int64_t, int, const int64_t *, int64_t,
                                     const int32_t *, const double *, const double *, const double *, const double *,
                                     const double *, const double *, const int32_t *, cudaStream_t);

}  // namespace mps
