// K1/K2: cell binning by counting sort, candidate neighbour lists and the
// cutoff-filtered pair lists (EW/ewald.py:84-199, 939-1016).
//
// Integer outputs are bit-exact with the reference: the cell coordinate uses
// the same float64 operations (numpy mod, divide, multiply, floor) and the pair
// order reproduces the reference's emission order (occupied cells by linear
// index, 27 neighbour cells with the x offset outermost, home particle, then
// neighbour particle, both by increasing id).  Floating-point pair data use
// explicitly rounded operations (no FMA contraction) so they match numpy's.
#include <string.h>

#include "cells.cuh"
#include "cellwalk.cuh"

namespace mps {

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------
__global__ void k_cell_assign(const double *__restrict__ x, int64_t n, double Lx, double Ly, double Lz,
                              int64_t ncx, int64_t ncy, int64_t ncz, int64_t *__restrict__ cell3) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double L[3] = {Lx, Ly, Lz};
        const int64_t nc[3] = {ncx, ncy, ncz};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            double w = np_mod(x[3 * i + d], L[d]);
            double f = floor(__dmul_rn(__ddiv_rn(w, L[d]), (double)nc[d]));
            cell3[3 * i + d] = (int64_t)f;
        }
    }
}

__global__ void k_cell_lin(const int64_t *__restrict__ cell3, int64_t n, int64_t ncx, int64_t ncy, int64_t ncz,
                           int32_t *__restrict__ lin, int32_t *__restrict__ counts) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        // clamp: a coordinate rounding up to exactly L lands in the last cell
        int64_t cx = min(max(cell3[3 * i + 0], (int64_t)0), ncx - 1);
        int64_t cy = min(max(cell3[3 * i + 1], (int64_t)0), ncy - 1);
        int64_t cz = min(max(cell3[3 * i + 2], (int64_t)0), ncz - 1);
        int32_t c = (int32_t)(cx + ncx * (cy + ncy * cz));
        lin[i] = c;
        atomicAdd(&counts[c], 1);
    }
}

__global__ void k_cell_scatter(const int32_t *__restrict__ lin, int64_t n, const int64_t *__restrict__ starts,
                               int32_t *__restrict__ cursor, int32_t *__restrict__ unsorted) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t c = lin[i];
        int64_t p = starts[c] + atomicAdd(&cursor[c], 1);
        unsorted[p] = (int32_t)i;
    }
}

// One warp per cell: rank each member by id (ids are unique) -> stable order.
__global__ void k_cell_rank(const int32_t *__restrict__ unsorted, const int32_t *__restrict__ counts,
                            const int64_t *__restrict__ starts, int64_t ncells, int32_t *__restrict__ sorted) {
    const int lane = threadIdx.x & 31;
    int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t c = warp; c < ncells; c += nwarps) {
        int32_t len = counts[c];
        int64_t s0 = starts[c];
        for (int32_t e = lane; e < len; e += 32) {
            int32_t v = unsorted[s0 + e];
            int32_t rank = 0;
            for (int32_t j = 0; j < len; ++j) rank += (unsorted[s0 + j] < v);
            sorted[s0 + rank] = v;
        }
    }
}

// Screen positions (near_position) of n points in sorted order, so that a walk's candidates are consecutive 16-byte
// loads, and of ne more as they come.
__global__ void k_near_positions(const double *__restrict__ x, const int32_t *__restrict__ sorted, int64_t n,
                                 const double *__restrict__ xe, int64_t ne, Box3 box, NearBox nb, float4 *__restrict__ xs,
                                 float4 *__restrict__ es) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n + ne; t += (int64_t)gridDim.x * blockDim.x) {
        if (t < n)
            xs[t] = near_position(x, sorted[t], box, nb);
        else
            es[t - n] = near_position(xe, t - n, box, nb);
    }
}

// Row of the first table separation >= d, at least 1 (the callers have checked d <= rv[ntab - 1]), from the
// uniform-spacing guess (d - r0) inv_dr; a table that is far from uniform takes the binary search.
__device__ __forceinline__ int64_t probe_row(const double *__restrict__ rv, int64_t ntab, double d, double inv_dr,
                                             double r0 = 0.0) {
    int64_t lo = 1, hi = ntab - 1;
    const double gf = (d - r0) * inv_dr;
    int64_t g = gf > 1.0 ? (gf < (double)hi ? (int64_t)gf : hi) : 1;
    for (int it = 0; it < 4; ++it) {
        if (rv[g] < d) {
            lo = ++g;   // g <= hi: rv[hi] >= d
        } else if (g > 1 && rv[g - 1] >= d) {
            hi = --g;
        } else {
            return g;
        }
    }
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (rv[mid] >= d) hi = mid; else lo = mid + 1;
    }
    return lo;
}

// 1/v by Newton's method y <- y (2 - v y) from a float32 seed (two steps).
__device__ __forceinline__ double rcp_newton(double v) {
    double y = (double)(1.0f / (float)v);
    y = y * (2.0 - v * y);
    y = y * (2.0 - v * y);
    return y;
}

// sqrt(d2) and its reciprocal without a float64 division: the square root of a zero separation is 0.
__device__ __forceinline__ double probe_distance(double d2, double *inv) {
    const double y = rsqrt(d2), d = d2 * y;
    *inv = y;
    return d2 > 0.0 ? fma(0.5 * y, fma(-d, d, d2), d) : d2;
}

// Minimum-image vector r - L trunc(2 r / L) of a probe/source pair and its squared length; the comparisons give the
// same value for |r| < L and cost no division.
__device__ __forceinline__ double probe_diff2(const double *__restrict__ xe, int64_t e, const double *__restrict__ xp,
                                              int64_t b, const Box3 &box, double r[3]) {
    double d2 = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double v = xe[3 * e + k] - xp[3 * b + k];
        const double L = box.L[k];
        if (fabs(v) < L) {
            if (v >= 0.5 * L)
                v -= L;
            else if (v <= -0.5 * L)
                v += L;
        } else {
            v -= L * trunc(2.0 * v / L);
        }
        r[k] = v;
        d2 += v * v;
    }
    return d2;
}

// Field at probe points from the dipoles of sources within rc (Compute_Field/RealSpace.m:1-60
// over the probe/source neighbour list of Compute_Field/FieldMap.m:46-52): one warp per probe walks
// the sources of the 27 cells around the probe's cell.  Minimum image r - L trunc(2 r / L); pairs
// with d >= rc or d = 0 are skipped; A, B interpolated between the bracketing table rows (first
// row with rvals >= d); out[e] = sum A m + (B - A) (m . r^) r^ in a fixed order per probe.
// One candidate in seven lies within rc: the walk screens them in float32 (near_walk) and the float64 pair terms, the
// only part that GB300's float64 rate bounds, run on 32 kept pairs at a time (90,000 probes and 10,000 spheres, 29 of
// 203 candidates a probe: 5.62 ms with every candidate in float64, 0.57 ms; the table row comes from the
// uniform-spacing guess instead of 13 float64 comparisons).
__global__ void __launch_bounds__(128) k_probe_real(const double *__restrict__ xe, int64_t ne,
                                                    const int64_t *__restrict__ cell_e,
                                                    const float4 *__restrict__ es,
                                                    const double *__restrict__ xp, const float4 *__restrict__ xs,
                                                    const double *__restrict__ p,
                                                    const int32_t *__restrict__ counts,
                                                    const int64_t *__restrict__ starts, int64_t ncx, int64_t ncy,
                                                    int64_t ncz, Box3 box, NearBox nb, double rc,
                                                    const double *__restrict__ perp,
                                                    const double *__restrict__ para, const double *__restrict__ rv,
                                                    int64_t ntab, double *__restrict__ out, int *__restrict__ err) {
    __shared__ int32_t q[4][kNearQueue];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const double rv_last = rv[ntab - 1], inv_dr = rv_last > 0 ? (double)(ntab - 1) / rv_last : 0.0;
    for (int64_t e = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; e < ne; e += nw) {
        const int32_t c = (int32_t)(cell_e[3 * e] + ncx * (cell_e[3 * e + 1] + ncy * cell_e[3 * e + 2]));
        const CellWalk cw = cell_walk(c, lane, counts, starts, ncx, ncy, ncz);
        double acc[3] = {0.0, 0.0, 0.0};
        near_walk(cw, lane, xs, es[e], -1, nb, q[wid], [&](int32_t b) {
            double r[3];
            double y;
            const double d = probe_distance(probe_diff2(xe, e, xp, b, box, r), &y);
            if (!(d < rc) || !(d > 0.0)) return;
            if (!(rv_last >= d)) {
                atomicExch(err, 1);
                return;
            }
            const int64_t lo = probe_row(rv, ntab, d, inv_dr);
            const double rh = rv[lo], rl = rv[lo - 1], inv = rcp_newton(rh - rl), wl = (rh - d) * inv, wh = (d - rl) * inv;
            const double A = perp[lo - 1] * wl + perp[lo] * wh;
            const double B = para[lo - 1] * wl + para[lo] * wh;
            const double *m = p + 3 * (int64_t)b;
            const double ba = (B - A) * ((m[0] * r[0] + m[1] * r[1] + m[2] * r[2]) * y) * y;
#pragma unroll
            for (int k = 0; k < 3; ++k) {   // (two multiply-adds, not three instructions)
                acc[k] += A * m[k];
                acc[k] += ba * r[k];
            }
        });
        const double v = warp_sum4(acc[0], acc[1], acc[2], 0.0, lane);
        if ((lane & 7) == 0 && lane < 24) out[3 * e + lane / 8] = v;
    }
}

// Field and field gradient at probe points from the dipoles and quadrupoles of sources within rc
// (Compute_Field_Quadrupole/RealSpace.m:1-77 over the probe/particle pairs of FieldMap.m:44-48):
// the couplings A..I of each pair interpolated from the 9 tables (field_dip_1/2, field_quad_1..3,
// grad_quad_1..4; first row with rvals >= d), out[e] = (E (3), G (5)).  A source at the probe
// itself (d = 0) is skipped (the reference divides by d there).
__global__ void __launch_bounds__(128) k_probe_real_quad(const double *__restrict__ xe, int64_t ne,
                                                         const int64_t *__restrict__ cell_e,
                                                         const float4 *__restrict__ es,
                                                         const double *__restrict__ xp,
                                                         const float4 *__restrict__ xs,
                                                         const double *__restrict__ sq,
                                                         const int32_t *__restrict__ counts,
                                                         const int64_t *__restrict__ starts, int64_t ncx,
                                                         int64_t ncy, int64_t ncz, Box3 box, NearBox nb, double rc,
                                                         const double *__restrict__ tab, const double *__restrict__ rv,
                                                         int64_t ntab, double *__restrict__ out, int *__restrict__ err) {
    __shared__ int32_t q[4][kNearQueue];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const double rv_last = rv[ntab - 1], inv_dr = rv_last > 0 ? (double)(ntab - 1) / rv_last : 0.0;
    for (int64_t e = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; e < ne; e += nw) {
        const int32_t c = (int32_t)(cell_e[3 * e] + ncx * (cell_e[3 * e + 1] + ncy * cell_e[3 * e + 2]));
        const CellWalk cw = cell_walk(c, lane, counts, starts, ncx, ncy, ncz);
        double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        near_walk(cw, lane, xs, es[e], -1, nb, q[wid], [&](int32_t b) {
            double r[3];
            double y;
            const double d = probe_distance(probe_diff2(xe, e, xp, b, box, r), &y);
            if (!(d < rc) || !(d > 0.0)) return;
            if (!(rv_last >= d)) {
                atomicExch(err, 1);
                return;
            }
            const int64_t lo = probe_row(rv, ntab, d, inv_dr);
            const double rh = rv[lo], rl = rv[lo - 1], inv = rcp_newton(rh - rl), wl = (rh - d) * inv, wh = (d - rl) * inv;
            double cf[9];
#pragma unroll
            for (int t = 0; t < 9; ++t) cf[t] = tab[t * ntab + lo - 1] * wl + tab[t * ntab + lo] * wh;
            const double A = cf[0], B = cf[1], Cc = cf[2], D = cf[3], E = cf[4], F = cf[5], Gg = cf[6], H = cf[7],
                         I = cf[8];
            const double rx = r[0] * y, ry = r[1] * y, rz = r[2] * y;
            const double *m = sq + 8 * (int64_t)b;
            const double Sx = m[0], Sy = m[1], Sz = m[2], Q0 = m[3], Q1 = m[4], Q2 = m[5], Q3 = m[6], Q4 = m[7];
            const double sr = Sx * rx + Sy * ry + Sz * rz;
            const double Qr0 = Q0 * rx + Q1 * ry + Q2 * rz;
            const double Qr1 = Q1 * rx + Q3 * ry + Q4 * rz;
            const double Qr2 = Q2 * rx + Q4 * ry - (Q0 + Q3) * rz;
            const double rQr = Q0 * (rx * rx - rz * rz) + 2 * Q1 * rx * ry + 2 * Q2 * rx * rz +
                               Q3 * (ry * ry - rz * rz) + 2 * Q4 * ry * rz;
            const double sE = (B - A) * sr - 0.5 * Cc * rQr;
            acc[0] += A * Sx;
            acc[1] += A * Sy;
            acc[2] += A * Sz;
            acc[0] += sE * rx;
            acc[1] += sE * ry;
            acc[2] += sE * rz;
            acc[0] -= D * Qr0;
            acc[1] -= D * Qr1;
            acc[2] -= D * Qr2;
            const double q5[5] = {rx * rx, rx * ry, rx * rz, ry * ry, ry * rz};
            const double srs[5] = {2 * Sx * rx, Sx * ry + rx * Sy, Sx * rz + rx * Sz, 2 * Sy * ry, Sy * rz + ry * Sz};
            const double qq[5] = {4 * Qr0 * rx, 2 * (Qr0 * ry + rx * Qr1), 2 * (Qr0 * rz + rx * Qr2), 4 * Qr1 * ry,
                                  2 * (Qr1 * rz + ry * Qr2)};
            const double Qv[5] = {Q0, Q1, Q2, Q3, Q4};
            const double cq = Cc * sr + 0.5 * I * rQr;
            const double di = (D + E) * sr + 0.5 * (F + H) * rQr;
            const double hG = 0.5 * Gg, hH = 0.5 * H;
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                acc[3 + k] += cq * q5[k];
                acc[3 + k] += D * srs[k];
                acc[3 + k] += hG * Qv[k];
                acc[3 + k] += hH * qq[k];
                if (k == 0 || k == 3) acc[3 + k] += di;
            }
        });
        const double v = warp_sum4(acc[0], acc[1], acc[2], acc[3], lane), w = warp_sum4(acc[4], acc[5], acc[6], acc[7], lane);
        if ((lane & 7) == 0) {
            out[8 * e + lane / 8] = v;
            out[8 * e + 4 + lane / 8] = w;
        }
    }
}

// Polydisperse field map, real space (Compute_Field_Sizes/RealSpace.m:1-77): probes are spheres of the
// smallest radius (class cmin), so the couplings of a probe/source pair come from the table column
// of the classes (cmin, cls[b]) (column order of CS/RealSpaceTable.m: i <= j, row-major over i);
// rvals need not start at 0: a separation below rvals[0] or above rvals[ntab-1] is out of the table.
__global__ void __launch_bounds__(128) k_probe_real_cs(const double *__restrict__ xe, int64_t ne,
                                                       const int64_t *__restrict__ cell_e,
                                                       const float4 *__restrict__ es,
                                                       const double *__restrict__ xp, const float4 *__restrict__ xs,
                                                       const double *__restrict__ p,
                                                       const int32_t *__restrict__ cls, int32_t cmin, int32_t M,
                                                       const int32_t *__restrict__ counts,
                                                       const int64_t *__restrict__ starts, int64_t ncx, int64_t ncy,
                                                       int64_t ncz, Box3 box, NearBox nb, double rc,
                                                       const double *__restrict__ perp,
                                                       const double *__restrict__ para,
                                                       const double *__restrict__ rv, int64_t ntab,
                                                       double *__restrict__ out, int *__restrict__ err) {
    __shared__ int32_t q[4][kNearQueue];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const double rv_first = rv[0], rv_last = rv[ntab - 1];
    // rows start at rv_first, not at zero: the guess is the offset from it
    const double inv_dr = rv_last > rv_first ? (double)(ntab - 1) / (rv_last - rv_first) : 0.0;
    for (int64_t e = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; e < ne; e += nw) {
        const int32_t c = (int32_t)(cell_e[3 * e] + ncx * (cell_e[3 * e + 1] + ncy * cell_e[3 * e + 2]));
        const CellWalk cw = cell_walk(c, lane, counts, starts, ncx, ncy, ncz);
        double acc[3] = {0.0, 0.0, 0.0};
        near_walk(cw, lane, xs, es[e], -1, nb, q[wid], [&](int32_t b) {
            double r[3];
            double y;
            const double d = probe_distance(probe_diff2(xe, e, xp, b, box, r), &y);
            if (!(d < rc)) return;
            if (!(d > rv_first) || !(rv_last >= d)) {
                atomicExch(err, 1);
                return;
            }
            const int64_t lo = probe_row(rv, ntab, d, inv_dr, rv_first);
            const int32_t ci = cmin < cls[b] ? cmin : cls[b], cj = cmin < cls[b] ? cls[b] : cmin;
            const int64_t col = (int64_t)ci * M - (int64_t)ci * (ci - 1) / 2 + (cj - ci);
            const double *tp = perp + col * ntab, *ta = para + col * ntab;
            const double rh = rv[lo], rl = rv[lo - 1], inv = rcp_newton(rh - rl), wl = (rh - d) * inv, wh = (d - rl) * inv;
            const double A = tp[lo - 1] * wl + tp[lo] * wh;
            const double B = ta[lo - 1] * wl + ta[lo] * wh;
            const double *m = p + 3 * (int64_t)b;
            const double ba = (B - A) * ((m[0] * r[0] + m[1] * r[1] + m[2] * r[2]) * y) * y;
#pragma unroll
            for (int k = 0; k < 3; ++k) {   // (two multiply-adds, not three instructions)
                acc[k] += A * m[k];
                acc[k] += ba * r[k];
            }
        });
        const double v = warp_sum4(acc[0], acc[1], acc[2], 0.0, lane);
        if ((lane & 7) == 0 && lane < 24) out[3 * e + lane / 8] = v;
    }
}

// Candidate counts in emission-slot order: slot(s,o) = 27*start[c] + o*count[c] + (s - start[c]).
__global__ void k_candidate_slots(const int32_t *__restrict__ sorted, const int32_t *__restrict__ lin,
                                  const int32_t *__restrict__ counts, const int64_t *__restrict__ starts, int64_t n,
                                  int64_t ncx, int64_t ncy, int64_t ncz, int64_t *__restrict__ slot_count) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < 27 * n; t += (int64_t)gridDim.x * blockDim.x) {
        int64_t s = t / 27;
        int o = (int)(t % 27);
        int32_t a = sorted[s];
        int32_t c = lin[a];
        int32_t nb = nb_cell(c, o, ncx, ncy, ncz);
        int64_t cnt = counts[nb] - (nb == c ? 1 : 0);
        int64_t slot = 27 * starts[c] + (int64_t)o * counts[c] + (s - starts[c]);
        slot_count[slot] = cnt;
    }
}

__global__ void k_candidate_fill(const int32_t *__restrict__ sorted, const int32_t *__restrict__ lin,
                                 const int32_t *__restrict__ counts, const int64_t *__restrict__ starts, int64_t n,
                                 int64_t ncx, int64_t ncy, int64_t ncz, const int64_t *__restrict__ slot_off,
                                 int64_t *__restrict__ p1, int64_t *__restrict__ p2) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < 27 * n; t += (int64_t)gridDim.x * blockDim.x) {
        int64_t s = t / 27;
        int o = (int)(t % 27);
        int32_t a = sorted[s];
        int32_t c = lin[a];
        int32_t nb = nb_cell(c, o, ncx, ncy, ncz);
        int64_t slot = 27 * starts[c] + (int64_t)o * counts[c] + (s - starts[c]);
        int64_t w = slot_off[slot];
        int64_t b0 = starts[nb], len = counts[nb];
        for (int64_t j = 0; j < len; ++j) {
            int32_t b = sorted[b0 + j];
            if (b == a) continue;
            p1[w] = a;
            p2[w] = b;
            ++w;
        }
    }
}

// Minimum-image separation exactly as numpy evaluates r - L*trunc(2r/L) and
// sqrt(sum(r*r)) (left-to-right over x, y, z).
__device__ __forceinline__ double min_image_sep(const double *__restrict__ x, int64_t a, int64_t b, const double *L,
                                                double r[3]) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double v = __dsub_rn(x[3 * a + d], x[3 * b + d]);
        double t = trunc(__ddiv_rn(__dmul_rn(2.0, v), L[d]));
        r[d] = __dsub_rn(v, __dmul_rn(L[d], t));
    }
    double s = __dadd_rn(__dadd_rn(__dmul_rn(r[0], r[0]), __dmul_rn(r[1], r[1])), __dmul_rn(r[2], r[2]));
    return __dsqrt_rn(s);
}

// First index i with rv[i] >= d (numpy searchsorted side='left').
__device__ __forceinline__ int64_t search_left(const double *__restrict__ rv, int64_t n, double d) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (rv[mid] < d)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Same index as search_left, starting from the uniform-spacing guess d * inv_dr
// (inv_dr = (ntab-1)/rv[ntab-1]); falls back to the binary search when the
// table is far from uniform.
__device__ __forceinline__ int64_t search_left_guess(const double *__restrict__ rv, int64_t n, double d,
                                                     double inv_dr) {
    if (!(inv_dr > 0)) return search_left(rv, n, d);
    double gf = d * inv_dr;
    int64_t g = gf < 0 ? 0 : (gf > (double)(n - 1) ? n - 1 : (int64_t)gf);
    for (int it = 0; it < 8; ++it) {
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
    return search_left(rv, n, d);
}

// Interpolated couplings at separation d; returns false when d is outside the table.
__device__ __forceinline__ bool table_lerp(const double *__restrict__ perp, const double *__restrict__ para,
                                           const double *__restrict__ rv, int64_t ntab, double d, double *A,
                                           double *B, double inv_dr = 0.0) {
    int64_t i = search_left_guess(rv, ntab, d, inv_dr);
    if (i <= 0 || i >= ntab) return false;
    double rl = rv[i - 1], rh = rv[i];
    double t = __ddiv_rn(__dsub_rn(d, rl), __dsub_rn(rh, rl));
    double omt = __dsub_rn(1.0, t);
    *A = __dadd_rn(__dmul_rn(perp[i - 1], omt), __dmul_rn(perp[i], t));
    *B = __dadd_rn(__dmul_rn(para[i - 1], omt), __dmul_rn(para[i], t));
    return true;
}

// 1/sqrt(s) by Newton's method y <- y (3 - s y^2) / 2 from a float32 seed: two
// steps take the seed's ~2^-22 relative error below float64 rounding.
__device__ __forceinline__ double rsqrt_newton(double s) {
    double y = (double)rsqrtf((float)s);
    y = y * (1.5 - 0.5 * s * y * y);
    y = y * (1.5 - 0.5 * s * y * y);
    return y;
}

// table_lerp with the segment's reciprocal from Newton iterations (solver lists:
// agreement with table_lerp to float64 rounding, not bit-exact).
__device__ __forceinline__ bool table_lerp_fast(const double *__restrict__ perp, const double *__restrict__ para,
                                                const double *__restrict__ rv, int64_t ntab, double d, double *A,
                                                double *B, double inv_dr) {
    int64_t i = search_left_guess(rv, ntab, d, inv_dr);
    if (i <= 0 || i >= ntab) return false;
    const double rl = rv[i - 1], rh = rv[i];
    const double t = (d - rl) * rcp_newton(rh - rl);
    const double omt = 1.0 - t;
    *A = perp[i - 1] * omt + perp[i] * t;
    *B = para[i - 1] * omt + para[i] * t;
    return true;
}

__global__ void k_pair_flag(const double *__restrict__ x, double Lx, double Ly, double Lz,
                            const int64_t *__restrict__ p1, const int64_t *__restrict__ p2, int64_t ncand, double rc,
                            int32_t *__restrict__ flag) {
    const double L[3] = {Lx, Ly, Lz};
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < ncand; k += (int64_t)gridDim.x * blockDim.x) {
        double r[3];
        double d = min_image_sep(x, p1[k], p2[k], L, r);
        flag[k] = d < rc ? 1 : 0;
    }
}

__global__ void k_pair_fill(const double *__restrict__ x, double Lx, double Ly, double Lz,
                            const int64_t *__restrict__ p1, const int64_t *__restrict__ p2, int64_t ncand,
                            const int32_t *__restrict__ flag, const int64_t *__restrict__ off,
                            const double *__restrict__ perp, const double *__restrict__ para,
                            const double *__restrict__ rv, int64_t ntab, int64_t *__restrict__ p1f,
                            int64_t *__restrict__ p2f, double *__restrict__ rhat, double *__restrict__ A,
                            double *__restrict__ B, int *__restrict__ err) {
    const double L[3] = {Lx, Ly, Lz};
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < ncand; k += (int64_t)gridDim.x * blockDim.x) {
        if (!flag[k]) continue;
        double r[3];
        int64_t a = p1[k], b = p2[k];
        double d = min_image_sep(x, a, b, L, r);
        int64_t w = off[k];
        p1f[w] = a;
        p2f[w] = b;
        rhat[3 * w + 0] = __ddiv_rn(r[0], d);
        rhat[3 * w + 1] = __ddiv_rn(r[1], d);
        rhat[3 * w + 2] = __ddiv_rn(r[2], d);
        double av = 0.0, bv = 0.0;
        if (!table_lerp(perp, para, rv, ntab, d, &av, &bv)) atomicExch(err, 1);
        A[w] = av;
        B[w] = bv;
    }
}

// Cutoff test of the solver's pair list.  A float32 screen on float32 copies
// of the positions sorts candidates into clearly outside / clearly inside /
// near rc (margins bound the float32 rounding); only pairs near rc (and, in
// the fill pass, kept pairs) touch float64, which is scarce on GB300.  The kept
// set is exactly the reference's d < rc set: the float64 path below does the
// reference's operations (r - L trunc(2r/L) by comparisons, which give the same
// value for |r| < L, and sqrt of the left-to-right sum of squares).
struct PairScreen {
    double L[3];
    float Lf[3];
    float rc2_lo, rc2_hi;
    double rc;
};

enum { SCREEN_OUT = 0, SCREEN_IN = 1, SCREEN_NEAR = 2 };

__device__ __forceinline__ int pair_screen(const float4 &a, const float4 &b, const PairScreen &ps) {
    const float pa[3] = {a.x, a.y, a.z}, pb[3] = {b.x, b.y, b.z};
    float s2 = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float v = pa[k] - pb[k];
        if (!(fabsf(v) < ps.Lf[k])) return SCREEN_NEAR;  // far outside the box: exact path decides
        if (v > 0.5f * ps.Lf[k])
            v -= ps.Lf[k];
        else if (v < -0.5f * ps.Lf[k])
            v += ps.Lf[k];
        s2 = fmaf(v, v, s2);
    }
    if (s2 > ps.rc2_hi) return SCREEN_OUT;
    if (s2 < ps.rc2_lo) return SCREEN_IN;
    return SCREEN_NEAR;
}

// Float64 minimum-image vector and distance, same values as min_image_sep for |r| < L.
__device__ __forceinline__ double pair_exact(const double *__restrict__ x, int64_t a, int64_t b, const PairScreen &ps,
                                             double r[3]) {
    bool big = false;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double v = __dsub_rn(x[3 * a + k], x[3 * b + k]);
        big = big || !(fabs(v) < ps.L[k]);
        if (v >= 0.5 * ps.L[k])
            v = __dsub_rn(v, ps.L[k]);
        else if (v <= -0.5 * ps.L[k])
            v = __dadd_rn(v, ps.L[k]);
        r[k] = v;
    }
    if (big) return min_image_sep(x, a, b, ps.L, r);
    const double s = __dadd_rn(__dadd_rn(__dmul_rn(r[0], r[0]), __dmul_rn(r[1], r[1])), __dmul_rn(r[2], r[2]));
    return __dsqrt_rn(s);
}

// Minimum-image difference x_a - x_b (same rounding as pair_exact) and its
// squared length; big = a coordinate difference of a box length or more (then
// the caller uses pair_exact, which wraps by the general rule).
__device__ __forceinline__ double pair_diff2(const double *__restrict__ x, int64_t a, int64_t b, const PairScreen &ps,
                                             double r[3], bool *big) {
    bool bg = false;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double v = __dsub_rn(x[3 * a + k], x[3 * b + k]);
        bg = bg || !(fabs(v) < ps.L[k]);
        if (v >= 0.5 * ps.L[k])
            v = __dsub_rn(v, ps.L[k]);
        else if (v <= -0.5 * ps.L[k])
            v = __dadd_rn(v, ps.L[k]);
        r[k] = v;
    }
    *big = bg;
    return __dadd_rn(__dadd_rn(__dmul_rn(r[0], r[0]), __dmul_rn(r[1], r[1])), __dmul_rn(r[2], r[2]));
}

// Filtered per-particle neighbour counts, slot (a, o) at a*27 + o.  One warp per
// (particle, neighbour cell): lanes take the cell's particles, a ballot counts
// the kept ones.  xs: float positions and ids in cell order, so a round of candidates is one contiguous load; by way of
// the sorted ids every lane's coordinates lay on a line of their own (N = 100,000: 0.26 -> 0.20 ms).
__global__ void __launch_bounds__(256) k_csr_count(const double *__restrict__ x, const float4 *__restrict__ xs,
                                                   PairScreen ps, const int32_t *__restrict__ lin,
                                                   const int32_t *__restrict__ counts,
                                                   const int64_t *__restrict__ starts, int64_t n, int64_t ncx,
                                                   int64_t ncy, int64_t ncz, int64_t *__restrict__ cnt27) {
    __shared__ int hist[8][27];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; s < n; s += nw) {
        const float4 pa = xs[s];
        const int32_t a = __float_as_int(pa.w);
        const CellWalk cw = cell_walk(lin[a], lane, counts, starts, ncx, ncy, ncz);
        if (lane < 27) hist[wid][lane] = 0;
        __syncwarp();
        // two candidates per lane per iteration: their dependent loads (position, then coordinates) overlap
        for (int j0 = 0; j0 < cw.total; j0 += 64) {
            int o[2];
            float4 c[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = j0 + 32 * h + lane;
                int64_t pos;
                walk_at(cw, j < cw.total ? j : cw.total - 1, o[h], pos);
                c[h] = j < cw.total ? xs[pos] : pa;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int32_t b = __float_as_int(c[h].w);
                bool keep = false;
                if (b != a) {
                    const int sc = pair_screen(pa, c[h], ps);
                    if (sc == SCREEN_IN) {
                        keep = true;
                    } else if (sc == SCREEN_NEAR) {
                        double r[3];
                        keep = pair_exact(x, a, b, ps, r) < ps.rc;
                    }
                }
                if (keep) atomicAdd(&hist[wid][o[h]], 1);
            }
        }
        __syncwarp();
        if (lane < 27) cnt27[(int64_t)a * 27 + lane] = hist[wid][lane];
        __syncwarp();
    }
}

template <typename T>
__device__ __forceinline__ void store_pair(PairData<T> &pd, int64_t w, int32_t b, double A, double B,
                                           const double rh[3], double d) {
    pd.nbr[w] = b;
    if (pd.dist) pd.dist[w] = (T)d;
    pd.A[w] = (T)A;
    pd.BA[w] = (T)(B - A);
    pd.rx[w] = (T)rh[0];
    pd.ry[w] = (T)rh[1];
    pd.rz[w] = (T)rh[2];
}

// Traversal of the cells around particle a in the order of k_csr_count, shared by the fill kernels: the screen only
// decides which candidates are kept (float screen, float64 for the few in its margin band) and queues their ids per
// warp in shared memory, in traversal order; drain(cnt, w) then computes the pairs w .. w + cnt - 1 of the row from the
// queue, one per lane (cnt <= 32), instead of by the few lanes of each round that kept one (about one candidate in six
// is kept).  The row lists its pairs by neighbour-cell offset, then by particle id.
constexpr int kFillWarps = 8;

template <class F>
__device__ __forceinline__ void csr_row_walk(const double *__restrict__ x, const float4 *__restrict__ xs,
                                             const PairScreen &ps, const CellWalk &cw, const float4 &pa, int lane,
                                             int64_t w, int32_t *q_b, F &&drain) {
    const int32_t a = __float_as_int(pa.w);
    int qn = 0;                           // kept pairs waiting in the queue (warp-uniform, < 32 between rounds)
    // two candidates per lane per iteration (candidates j0 + lane and j0 + 32 + lane, queued in that order)
    for (int j0 = 0; j0 < cw.total; j0 += 64) {
        float4 c[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = j0 + 32 * h + lane;
            int o;
            int64_t pos;
            walk_at(cw, j < cw.total ? j : cw.total - 1, o, pos);
            (void)o;
            c[h] = j < cw.total ? xs[pos] : pa;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int32_t b = __float_as_int(c[h].w);
            bool keep = false;
            const int sc = b != a ? pair_screen(pa, c[h], ps) : SCREEN_OUT;
            if (sc == SCREEN_IN) {
                keep = true;
            } else if (sc == SCREEN_NEAR) {   // the correctly rounded float64 separation decides
                double r64[3];
                keep = pair_exact(x, a, b, ps, r64) < ps.rc;
            }
            const unsigned mask = __ballot_sync(0xffffffffu, keep);
            if (keep) q_b[qn + __popc(mask & ((1u << lane) - 1u))] = b;
            qn += __popc(mask);
        }
        __syncwarp();
        while (qn >= 32) {
            drain(32, w);
            w += 32;
            qn -= 32;
            __syncwarp();
            if (lane < qn) q_b[lane] = q_b[32 + lane];   // the rest to the front (qn < 64 here)
            if (lane + 32 < qn) q_b[lane + 32] = q_b[64 + lane];
            __syncwarp();
        }
    }
    if (qn > 0) drain(qn, w);
    __syncwarp();
}

// Float64 pair list of the quadrupole and polydisperse operators (50,000 spheres, 60 of about 380 candidates: 1.77 ms
// with the pair terms in the walk, 0.45 ms queued).
__global__ void __launch_bounds__(kFillWarps * 32) k_csr_fill(const double *__restrict__ x,
                                                              const float4 *__restrict__ xs, PairScreen ps,
                                                              const int32_t *__restrict__ lin,
                                                              const int32_t *__restrict__ counts,
                                                              const int64_t *__restrict__ starts, int64_t n,
                                                              int64_t ncx, int64_t ncy, int64_t ncz,
                                                              const int64_t *__restrict__ off27,
                                                              const double *__restrict__ perp,
                                                              const double *__restrict__ para,
                                                              const double *__restrict__ rv, int64_t ntab,
                                                              double inv_dr, PairData<double> p64,
                                                              PairData<float> p32, int *__restrict__ err) {
    __shared__ int32_t q_b[kFillWarps][128];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; s < n; s += nw) {
        const float4 pa = xs[s];
        const int32_t a = __float_as_int(pa.w);
        const CellWalk cw = cell_walk(lin[a], lane, counts, starts, ncx, ncy, ncz);
        csr_row_walk(x, xs, ps, cw, pa, lane, off27[(int64_t)a * 27], q_b[wid], [&](int cnt, int64_t w) {
            if (lane >= cnt) return;
            const int32_t b = q_b[wid][lane];
            double r[3];
            bool big = false;
            double s2 = pair_diff2(x, a, b, ps, r, &big);
            if (big) {   // far-wrapped: the general rule
                const double de = pair_exact(x, a, b, ps, r);
                s2 = __dmul_rn(de, de);
            }
            // the float64 division and square root are slow on GB300: Newton iterations from float32 seeds instead
            const double y = rsqrt_newton(s2);
            const double d = s2 * y;
            const double rh[3] = {r[0] * y, r[1] * y, r[2] * y};
            double A = 0.0, B = 0.0;
            // ntab == 0: the couplings are filled in afterwards from the separations
            if (ntab > 0 && !table_lerp_fast(perp, para, rv, ntab, d, &A, &B, inv_dr)) atomicExch(err, 1);
            store_pair(p64, w + lane, b, A, B, rh, d);
            store_pair(p32, w + lane, b, A, B, rh, d);
        });
    }
}

// ---------------------------------------------------------------------------
// Double-float pair list
// ---------------------------------------------------------------------------
__global__ void k_positions_df(const double *__restrict__ x, int64_t m, float2 *__restrict__ xdf) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const dfv v(x[i]);
        xdf[i] = make_float2(v.hi, v.lo);
    }
}

__global__ void k_df_tab(const double *__restrict__ perp, const double *__restrict__ para,
                         const double *__restrict__ rv, int64_t ntab, float *__restrict__ rvf,
                         float4 *__restrict__ seg_r, float4 *__restrict__ seg_perp, float4 *__restrict__ seg_para) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ntab; i += (int64_t)gridDim.x * blockDim.x) {
        rvf[i] = (float)rv[i];
        if (i == 0) {
            seg_r[0] = seg_perp[0] = seg_para[0] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const dfv rl(rv[i - 1]), inv(1.0 / (rv[i] - rv[i - 1]));
        const dfv p0(perp[i - 1]), dp(perp[i] - perp[i - 1]), q0(para[i - 1]), dq(para[i] - para[i - 1]);
        seg_r[i] = make_float4(rl.hi, rl.lo, inv.hi, inv.lo);
        seg_perp[i] = make_float4(p0.hi, p0.lo, dp.hi, dp.lo);
        seg_para[i] = make_float4(q0.hi, q0.lo, dq.hi, dq.lo);
    }
}

__device__ __forceinline__ dfv df_lo(float4 v) { return dfv(v.x, v.y); }
__device__ __forceinline__ dfv df_hi(float4 v) { return dfv(v.z, v.w); }

// 1/sqrt(s) in double-float by Newton's method y <- y (3 - s y^2) / 2 from the
// float32 reciprocal square root (two steps).
__device__ __forceinline__ dfv df_rsqrt(dfv s) {
    dfv y(rsqrtf(s.hi), 0.f);
    const dfv three_half(1.5f, 0.f);
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        dfv h = s * y * y;
        h.hi = __fmul_rn(h.hi, 0.5f);
        h.lo = __fmul_rn(h.lo, 0.5f);
        y = y * (three_half - h);
    }
    return y;
}

// First table index with rvf[i] >= d from the uniform-spacing guess (float).
__device__ __forceinline__ int64_t df_search(const float *__restrict__ rvf, int64_t n, float d, float inv_dr) {
    int64_t g = (int64_t)(d * inv_dr);
    g = g < 0 ? 0 : (g > n - 1 ? n - 1 : g);
    for (int it = 0; it < 8; ++it) {
        if (g < n && rvf[g] < d) {
            ++g;
            continue;
        }
        if (g > 0 && rvf[g - 1] >= d) {
            --g;
            continue;
        }
        return g;
    }
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (rvf[mid] < d)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void store_pair_df(PairData<dfv> &pd, PairData<float> &pf, int64_t w, int32_t b, dfv A,
                                              dfv B, const dfv rh[3], dfv d) {
    const dfv BA = B - A;
    pd.nbr[w] = b;
    pd.A[w] = A;
    pd.BA[w] = BA;
    pd.rx[w] = rh[0];
    pd.ry[w] = rh[1];
    pd.rz[w] = rh[2];
    pd.dist[w] = d;
    pf.A[w] = A.hi;
    pf.BA[w] = BA.hi;
    pf.rx[w] = rh[0].hi;
    pf.ry[w] = rh[1].hi;
    pf.rz[w] = rh[2].hi;
}

// Double-float couplings of one kept pair from its (minimum-image) separation r.
__device__ __forceinline__ void df_pair_out(const DfTab &tab, PairData<dfv> &pdf, PairData<float> &p32, int64_t wp,
                                            int32_t b, const dfv r[3], int *__restrict__ err) {
    const dfv s2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    const dfv y = df_rsqrt(s2);
    const dfv d = s2 * y;
    const dfv rh[3] = {r[0] * y, r[1] * y, r[2] * y};
    dfv A(0.f, 0.f), B(0.f, 0.f);
    int64_t i = df_search(tab.rvf, tab.ntab, d.hi, tab.inv_dr);
    // The float search can land one segment off when d lies within a float rounding of a node;
    // settle the bracket r_{i-1} < d <= r_i (the reference's searchsorted 'left') in double-float,
    // so the coupling is interpolated inside its segment instead of extrapolated across the node.
    if (i > 1 && i < tab.ntab) {
        const dfv lo = d - df_lo(tab.seg_r[i]);
        if (lo.hi < 0.f || (lo.hi == 0.f && lo.lo <= 0.f)) --i;
    }
    if (i > 0 && i + 1 < tab.ntab) {
        const dfv hi = d - df_lo(tab.seg_r[i + 1]);
        if (hi.hi > 0.f || (hi.hi == 0.f && hi.lo > 0.f)) ++i;
    }
    if (i <= 0 || i >= tab.ntab) {
        atomicExch(err, 1);
    } else {
        const float4 sr = tab.seg_r[i], sp = tab.seg_perp[i], sq = tab.seg_para[i];
        const dfv tt = (d - df_lo(sr)) * df_hi(sr);
        A = df_lo(sp) + tt * df_hi(sp);
        B = df_lo(sq) + tt * df_hi(sq);
    }
    store_pair_df(pdf, p32, wp, b, A, B, rh, d);
}

// Double-float pair list of the dipole operator, as k_csr_fill.  The keep decision is that of the float64 form (inside
// the screen's inner margin the float64 distance is below rc too), and so is the separation (double-float difference,
// float64 for a far-wrapped pair).
__global__ void __launch_bounds__(kFillWarps * 32) k_csr_fill_df(const double *__restrict__ x,
                                                                 const float4 *__restrict__ xs,
                                                                 const float2 *__restrict__ xdf, PairScreen ps,
                                                                 const int32_t *__restrict__ lin,
                                                                 const int32_t *__restrict__ counts,
                                                                 const int64_t *__restrict__ starts, int64_t n,
                                                                 int64_t ncx, int64_t ncy, int64_t ncz,
                                                                 const int64_t *__restrict__ off27, DfTab tab,
                                                                 PairData<dfv> pdf, PairData<float> p32,
                                                                 int *__restrict__ err) {
    __shared__ int32_t q_b[kFillWarps][128];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    dfv L[3], halfL[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        L[k] = dfv(ps.L[k]);
        halfL[k] = dfv(0.5 * ps.L[k]);
    }
    // queue entries [0, cnt) of particle a -> pairs w .. w + cnt - 1, one per lane (cnt <= 32)
    auto drain = [&](int32_t a, int cnt, int64_t w) {
        if (lane >= cnt) return;
        const int32_t b = q_b[wid][lane];
        dfv r[3];
        bool big = false;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float2 pa = xdf[3 * a + k], pb = xdf[3 * b + k];
            dfv v = dfv_two_diff(pa.x, pb.x) + dfv_two_diff(pa.y, pb.y);
            big = big || !(fabsf(v.hi) < ps.Lf[k] * 0.999f);
            // minimum image with the float64 path's rule: v >= L/2 -> v - L, v <= -L/2 -> v + L
            const dfv up = v - halfL[k], dn = v + halfL[k];
            if (up.hi > 0.f || (up.hi == 0.f && up.lo >= 0.f))
                v = v - L[k];
            else if (dn.hi < 0.f || (dn.hi == 0.f && dn.lo <= 0.f))
                v = v + L[k];
            r[k] = v;
        }
        if (big) {   // far-wrapped: float64 supplies the vector
            double r64[3];
            pair_exact(x, a, b, ps, r64);
            for (int k = 0; k < 3; ++k) r[k] = dfv(r64[k]);
        }
        df_pair_out(tab, pdf, p32, w + lane, b, r, err);
    };
    for (int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; s < n; s += nw) {
        const float4 pa = xs[s];
        const int32_t a = __float_as_int(pa.w);
        const CellWalk cw = cell_walk(lin[a], lane, counts, starts, ncx, ncy, ncz);
        csr_row_walk(x, xs, ps, cw, pa, lane, off27[(int64_t)a * 27], q_b[wid],
                     [&](int cnt, int64_t w) { drain(a, cnt, w); });
    }
}

__global__ void k_pairs_df_to_f64(PairData<dfv> pd, int64_t np, PairData<double> p64) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < np; e += (int64_t)gridDim.x * blockDim.x) {
        p64.A[e] = (double)pd.A[e];
        p64.BA[e] = (double)pd.BA[e];
        p64.rx[e] = (double)pd.rx[e];
        p64.ry[e] = (double)pd.ry[e];
        p64.rz[e] = (double)pd.rz[e];
        p64.dist[e] = (double)pd.dist[e];
    }
}

static PairScreen make_screen(const double *box, double rc, double maxabs) {
    PairScreen ps;
    double Lmax = 0.0;
    for (int k = 0; k < 3; ++k) {
        ps.L[k] = box[k];
        ps.Lf[k] = (float)box[k];
        Lmax = box[k] > Lmax ? box[k] : Lmax;
    }
    ps.rc = rc;
    // per-component error of the float32 difference and wrap: rounding of both
    // positions (<= 2^-24 |x| each), of the box and of the result
    const double eps = 4.0 * 5.9604644775390625e-08 * (maxabs + Lmax);
    const double m = 4.0 * 1.7320508075688772 * eps + 1e-6 * rc;
    const double lo = rc > m ? rc - m : 0.0;
    ps.rc2_lo = (float)(lo * lo * (1.0 - 1e-5));
    ps.rc2_hi = (float)((rc + m) * (rc + m) * (1.0 + 1e-5));
    return ps;
}

// float32 copy of the positions and the largest |coordinate| (as ordered float bits).
// xs[k] = float position and id of particle sorted[k]; the largest |coordinate| to maxbits.
__global__ void k_positions_f32(const double *__restrict__ x, const int32_t *__restrict__ sorted, int64_t n,
                                float4 *__restrict__ xs, unsigned *__restrict__ maxbits) {
    unsigned local = 0u;   // (a NaN coordinate's bits are above every number's)
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const int32_t a = sorted[k];
        const float4 v = make_float4((float)x[3 * (int64_t)a], (float)x[3 * (int64_t)a + 1], (float)x[3 * (int64_t)a + 2],
                                     __int_as_float(a));
        xs[k] = v;
        local = max(local, max(__float_as_uint(fabsf(v.x)), max(__float_as_uint(fabsf(v.y)), __float_as_uint(fabsf(v.z)))));
    }
    for (int o = 16; o > 0; o >>= 1) local = max(local, __shfl_xor_sync(0xffffffffu, local, o));
    if ((threadIdx.x & 31) == 0) atomicMax(maxbits, local);
}

__global__ void k_row_ptr(const int64_t *__restrict__ off27, const int64_t *__restrict__ cnt27, int64_t n,
                          int64_t *__restrict__ row_ptr) {
    for (int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; a <= n; a += (int64_t)gridDim.x * blockDim.x) {
        row_ptr[a] = a < n ? off27[a * 27] : off27[n * 27 - 1] + cnt27[n * 27 - 1];
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
void compute_ncell(const double *box, double rmax, int64_t *ncell) {
    for (int d = 0; d < 3; ++d) {
        int64_t v = (int64_t)floor(box[d] / rmax);
        ncell[d] = v < 3 ? 3 : v;
    }
}

bool cells_fit(const int64_t *ncell) {
    int64_t ncells = 1;
    for (int d = 0; d < 3; ++d) {
        if (ncell[d] > INT32_MAX / ncells) return false;
        ncells *= ncell[d];
    }
    return true;
}

size_t cell_bins_bytes(int64_t n, int64_t ncells) {
    size_t b = 0;
    b += 256 + (size_t)n * 4;         // lin
    b += 256 + (size_t)ncells * 4;    // counts
    b += 256 + (size_t)ncells * 8;    // starts
    b += 256 + (size_t)ncells * 4;    // cursor
    b += 256 + (size_t)n * 4;         // sorted
    b += 256 + (size_t)n * 4;         // unsorted
    b += 256 + scan_workspace(ncells);
    return b;
}

static void *carve(char *&p, size_t bytes) {
    uintptr_t u = ((uintptr_t)p + 255) & ~(uintptr_t)255;
    p = (char *)(u + bytes);
    return (void *)u;
}

int cell_bins_build(const int64_t *cell3, int64_t n, const int64_t *ncell, void *ws, CellBins &cb, cudaStream_t s) {
    int64_t ncells = ncell[0] * ncell[1] * ncell[2];
    char *p = (char *)ws;
    cb.ncell[0] = ncell[0];
    cb.ncell[1] = ncell[1];
    cb.ncell[2] = ncell[2];
    cb.ncells = ncells;
    cb.n = n;
    cb.lin = (int32_t *)carve(p, (size_t)n * 4);
    cb.counts = (int32_t *)carve(p, (size_t)ncells * 4);
    cb.starts = (int64_t *)carve(p, (size_t)ncells * 8);
    cb.cursor = (int32_t *)carve(p, (size_t)ncells * 4);
    cb.sorted = (int32_t *)carve(p, (size_t)n * 4);
    cb.unsorted = (int32_t *)carve(p, (size_t)n * 4);
    void *scan_tmp = carve(p, scan_workspace(ncells));
    if (n == 0) return MPS_OK;
    MPS_CUDA_TRY(cudaMemsetAsync(cb.counts, 0, (size_t)ncells * 4, s));
    MPS_CUDA_TRY(cudaMemsetAsync(cb.cursor, 0, (size_t)ncells * 4, s));
    k_cell_lin<<<grid_for(n, 256), 256, 0, s>>>(cell3, n, ncell[0], ncell[1], ncell[2], cb.lin, cb.counts);
    MPS_LAUNCH_CHECK();
    int rc = exclusive_scan_i32_to_i64(cb.counts, cb.starts, ncells, scan_tmp, s);
    if (rc) return rc;
    k_cell_scatter<<<grid_for(n, 256), 256, 0, s>>>(cb.lin, n, cb.starts, cb.cursor, cb.unsorted);
    MPS_LAUNCH_CHECK();
    k_cell_rank<<<grid_for(ncells * 32, 256), 256, 0, s>>>(cb.unsorted, cb.counts, cb.starts, ncells, cb.sorted);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int cell_assign(const double *x, int64_t n, const double *box, const int64_t *ncell, int64_t *cell3, cudaStream_t s) {
    if (n == 0) return MPS_OK;
    k_cell_assign<<<grid_for(n, 256), 256, 0, s>>>(x, n, box[0], box[1], box[2], ncell[0], ncell[1], ncell[2], cell3);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int positions_f32(const double *x, const int32_t *sorted, int64_t n, float4 *xs, unsigned *maxbits, double *maxabs,
                  cudaStream_t s) {
    MPS_CUDA_TRY(cudaMemsetAsync(maxbits, 0, sizeof(unsigned), s));
    k_positions_f32<<<grid_for(n, 256), 256, 0, s>>>(x, sorted, n, xs, maxbits);
    MPS_LAUNCH_CHECK();
    unsigned hb = 0;
    MPS_CUDA_TRY(cudaMemcpyAsync(&hb, maxbits, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    MPS_CUDA_TRY(cudaStreamSynchronize(s));
    float f;
    memcpy(&f, &hb, sizeof(f));
    *maxabs = (double)f * (1.0 + 1e-6);
    return MPS_OK;
}

int csr_pairs_count(const double *x, const float4 *xs, double maxabs, const double *box, double rc, const CellBins &cb,
                    int64_t *cnt27, int64_t *off27, void *scan_tmp, int64_t *last2, cudaStream_t s) {
    int64_t n = cb.n;
    k_csr_count<<<grid_for(n * 32, 256, 152 * 64), 256, 0, s>>>(x, xs, make_screen(box, rc, maxabs), cb.lin, cb.counts,
                                                                cb.starts, n, cb.ncell[0], cb.ncell[1], cb.ncell[2], cnt27);
    MPS_LAUNCH_CHECK();
    int r = exclusive_scan_i64(cnt27, off27, 27 * n, scan_tmp, s);
    if (r) return r;
    MPS_CUDA_TRY(cudaMemcpyAsync(&last2[0], off27 + 27 * n - 1, 8, cudaMemcpyDeviceToHost, s));
    MPS_CUDA_TRY(cudaMemcpyAsync(&last2[1], cnt27 + 27 * n - 1, 8, cudaMemcpyDeviceToHost, s));
    return MPS_OK;
}

int csr_pairs_fill(const double *x, const float4 *xs, double maxabs, const double *box, double rc, const CellBins &cb,
                   const int64_t *cnt27,
                   const int64_t *off27, const double *perp, const double *para, const double *rv, int64_t ntab,
                   int64_t *row_ptr, PairData<double> p64, PairData<float> p32, int *err, cudaStream_t s) {
    int64_t n = cb.n;
    k_row_ptr<<<grid_for(n + 1, 256), 256, 0, s>>>(off27, cnt27, n, row_ptr);
    MPS_LAUNCH_CHECK();
    double rv_last = 0.0;
    if (ntab > 0) {
        MPS_CUDA_TRY(cudaMemcpyAsync(&rv_last, rv + ntab - 1, sizeof(double), cudaMemcpyDeviceToHost, s));
        MPS_CUDA_TRY(cudaStreamSynchronize(s));
    }
    const double inv_dr = rv_last > 0 ? (double)(ntab - 1) / rv_last : 0.0;
    k_csr_fill<<<grid_for(n * 32, kFillWarps * 32, 152 * 64), kFillWarps * 32, 0, s>>>(
        x, xs, make_screen(box, rc, maxabs), cb.lin, cb.counts, cb.starts, n, cb.ncell[0], cb.ncell[1], cb.ncell[2], off27,
        perp, para, rv, ntab, inv_dr, p64, p32, err);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

size_t df_tab_bytes(int64_t ntab) { return 256 * 4 + (size_t)ntab * (sizeof(float) + 3 * sizeof(float4)); }

int df_tab_build(const double *perp, const double *para, const double *rv, int64_t ntab, void *buf, DfTab &t,
                 cudaStream_t s) {
    char *p = (char *)buf;
    auto carve = [&](size_t bytes) {
        uintptr_t u = ((uintptr_t)p + 255) & ~(uintptr_t)255;
        p = (char *)(u + bytes);
        return (void *)u;
    };
    float *rvf = (float *)carve(sizeof(float) * ntab);
    float4 *sr = (float4 *)carve(sizeof(float4) * ntab);
    float4 *sp = (float4 *)carve(sizeof(float4) * ntab);
    float4 *sq = (float4 *)carve(sizeof(float4) * ntab);
    k_df_tab<<<grid_for(ntab, 256), 256, 0, s>>>(perp, para, rv, ntab, rvf, sr, sp, sq);
    MPS_LAUNCH_CHECK();
    double rv_last = 0.0;
    MPS_CUDA_TRY(cudaMemcpyAsync(&rv_last, rv + ntab - 1, sizeof(double), cudaMemcpyDeviceToHost, s));
    MPS_CUDA_TRY(cudaStreamSynchronize(s));
    t.rvf = rvf;
    t.seg_r = sr;
    t.seg_perp = sp;
    t.seg_para = sq;
    t.ntab = ntab;
    t.inv_dr = rv_last > 0 ? (float)((double)(ntab - 1) / rv_last) : 0.f;
    return MPS_OK;
}

int positions_df(const double *x, int64_t n, float2 *xdf, cudaStream_t s) {
    k_positions_df<<<grid_for(3 * n, 256), 256, 0, s>>>(x, 3 * n, xdf);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int csr_pairs_fill_df(const double *x, const float4 *xs, const float2 *xdf, double maxabs, const double *box, double rc,
                      const CellBins &cb, const int64_t *cnt27, const int64_t *off27, const DfTab &tab,
                      int64_t *row_ptr, PairData<dfv> pdf, PairData<float> p32, int *err, cudaStream_t s) {
    const int64_t n = cb.n;
    k_row_ptr<<<grid_for(n + 1, 256), 256, 0, s>>>(off27, cnt27, n, row_ptr);
    MPS_LAUNCH_CHECK();
    k_csr_fill_df<<<grid_for(n * 32, kFillWarps * 32, 152 * 64), kFillWarps * 32, 0, s>>>(
        x, xs, xdf, make_screen(box, rc, maxabs), cb.lin, cb.counts, cb.starts, n, cb.ncell[0],
        cb.ncell[1], cb.ncell[2], off27, tab, pdf, p32, err);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int pairs_df_to_f64(const PairData<dfv> &pdf, int64_t np, PairData<double> p64, cudaStream_t s) {
    if (np == 0) return MPS_OK;
    k_pairs_df_to_f64<<<grid_for(np, 256), 256, 0, s>>>(pdf, np, p64);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}


int near_positions(const double *x, const int32_t *sorted, int64_t n, const Box3 &box, const NearBox &nb, float4 *xs,
                   cudaStream_t s) {
    if (n == 0) return MPS_OK;
    k_near_positions<<<grid_for(n, 256), 256, 0, s>>>(x, sorted, n, nullptr, 0, box, nb, xs, nullptr);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

// What the walks around the probes read: the sources' cells, the probes' cell coordinates and the screen positions of
// both, in one allocation (six of them, and a second launch for the positions, had been 4 % of a map of one probe).
struct ProbeCells {
    int64_t ncell[3];
    Box3 box;
    NearBox nb;
    CellBins cb;
    int64_t *cell_e;
    float4 *xs, *es;
    int *err;
    void *mem = nullptr;
};

static int probe_cells_build(const double *xe, int64_t ne, const double *xp, int64_t np, const double *box, double rc,
                             ProbeCells &pc, cudaStream_t s) {
    compute_ncell(box, rc, pc.ncell);
    if (!cells_fit(pc.ncell)) return MPS_BAD_ARG;
    const int64_t ncells = pc.ncell[0] * pc.ncell[1] * pc.ncell[2];
    const size_t bins = cell_bins_bytes(np, ncells);
    const size_t bytes = 256 * 6 + bins + (sizeof(int64_t) * 3 + sizeof(float4)) * (size_t)(np + ne) + sizeof(int);
    if (cudaMallocAsync(&pc.mem, bytes, s) != cudaSuccess) {
        pc.mem = nullptr;
        cudaGetLastError();
        return MPS_NO_MEMORY;
    }
    char *p = (char *)pc.mem;
    int64_t *cell_p = (int64_t *)carve(p, sizeof(int64_t) * 3 * (size_t)np);
    pc.cell_e = (int64_t *)carve(p, sizeof(int64_t) * 3 * (size_t)ne);
    pc.xs = (float4 *)carve(p, sizeof(float4) * (size_t)np);
    pc.es = (float4 *)carve(p, sizeof(float4) * (size_t)ne);
    pc.err = (int *)carve(p, sizeof(int));
    void *ws = carve(p, bins);
    const bool periodic[3] = {true, true, true};
    pc.box = Box3{{box[0], box[1], box[2]}};
    pc.nb = make_near_box(box, rc, periodic);
    if (cudaMemsetAsync(pc.err, 0, sizeof(int), s) != cudaSuccess) return MPS_CUDA_ERR;
    int r = cell_assign(xp, np, box, pc.ncell, cell_p, s);
    if (!r) r = cell_bins_build(cell_p, np, pc.ncell, ws, pc.cb, s);
    if (!r) r = cell_assign(xe, ne, box, pc.ncell, pc.cell_e, s);
    if (r) return r;
    k_near_positions<<<grid_for(np + ne, 256), 256, 0, s>>>(xp, pc.cb.sorted, np, xe, ne, pc.box, pc.nb, pc.xs, pc.es);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

// Status of a probe sum whose kernel has been launched (r: status so far): waits for it.
static int probe_cells_end(ProbeCells &pc, int r, cudaStream_t s) {
    int herr = 0;
    if (!r && cudaGetLastError() != cudaSuccess) r = MPS_CUDA_ERR;
    if (!r && (cudaMemcpyAsync(&herr, pc.err, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
               cudaStreamSynchronize(s) != cudaSuccess))
        r = MPS_CUDA_ERR;
    if (pc.mem) cudaFreeAsync(pc.mem, s);
    return !r && herr ? MPS_TABLE_RANGE : r;
}

int probe_real_space(const double *xe, int64_t ne, const double *xp, const double *p, int64_t np, const double *box,
                     double rc, const double *perp, const double *para, const double *rv, int64_t ntab, double *out,
                     cudaStream_t s) {
    if (ne == 0) return MPS_OK;
    if (ntab < 2) return MPS_BAD_ARG;
    ProbeCells pc;
    const int r = probe_cells_build(xe, ne, xp, np, box, rc, pc, s);
    if (!r)
        k_probe_real<<<grid_for(ne * 32, 128, 152 * 128), 128, 0, s>>>(
            xe, ne, pc.cell_e, pc.es, xp, pc.xs, p, pc.cb.counts, pc.cb.starts, pc.ncell[0], pc.ncell[1], pc.ncell[2],
            pc.box, pc.nb, rc, perp, para, rv, ntab, out, pc.err);
    return probe_cells_end(pc, r, s);
}

int probe_real_space_quad(const double *xe, int64_t ne, const double *xp, const double *sq, int64_t np,
                          const double *box, double rc, const double *tab9, const double *rv, int64_t ntab,
                          double *out, cudaStream_t s) {
    if (ne == 0) return MPS_OK;
    if (ntab < 2) return MPS_BAD_ARG;
    ProbeCells pc;
    const int r = probe_cells_build(xe, ne, xp, np, box, rc, pc, s);
    if (!r)
        k_probe_real_quad<<<grid_for(ne * 32, 128, 152 * 128), 128, 0, s>>>(
            xe, ne, pc.cell_e, pc.es, xp, pc.xs, sq, pc.cb.counts, pc.cb.starts, pc.ncell[0], pc.ncell[1], pc.ncell[2],
            pc.box, pc.nb, rc, tab9, rv, ntab, out, pc.err);
    return probe_cells_end(pc, r, s);
}

int probe_real_space_cs(const double *xe, int64_t ne, const double *xp, const double *p, const int32_t *cls,
                        int32_t cmin, int32_t M, int64_t np, const double *box, double rc, const double *perp,
                        const double *para, const double *rv, int64_t ntab, double *out, cudaStream_t s) {
    if (ne == 0) return MPS_OK;
    if (ntab < 2 || M < 1 || cmin < 0 || cmin >= M) return MPS_BAD_ARG;
    ProbeCells pc;
    const int r = probe_cells_build(xe, ne, xp, np, box, rc, pc, s);
    if (!r)
        k_probe_real_cs<<<grid_for(ne * 32, 128, 152 * 128), 128, 0, s>>>(
            xe, ne, pc.cell_e, pc.es, xp, pc.xs, p, cls, cmin, M, pc.cb.counts, pc.cb.starts, pc.ncell[0], pc.ncell[1],
            pc.ncell[2], pc.box, pc.nb, rc, perp, para, rv, ntab, out, pc.err);
    return probe_cells_end(pc, r, s);
}

}  // namespace mps

using namespace mps;

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" int mps_cell_list(const double *x, int64_t n, const double *box, double rmax, int64_t *cell,
                             int64_t *ncell, mps_stream_t stream) {
    if (n < 0 || !box || !ncell || !(rmax > 0) || (n > 0 && (!x || !cell))) return MPS_BAD_ARG;
    for (int d = 0; d < 3; ++d)
        if (!(box[d] > 0)) return MPS_BAD_ARG;
    compute_ncell(box, rmax, ncell);
    return cell_assign(x, n, box, ncell, cell, (cudaStream_t)stream);
}

// The kernels index particles and cells with int32 (cell linear index, sorted ids) and the slot
// arrays with 27 n entries: reject sizes whose products would wrap before anything is sized from them.
static bool nl_sizes_ok(int64_t n, const int64_t *ncell) {
    if (n < 0 || n > INT32_MAX / 27) return false;
    int64_t ncells = 1;
    for (int d = 0; d < 3; ++d) {
        if (ncell[d] < 1 || ncell[d] > INT32_MAX) return false;
        if (__builtin_mul_overflow(ncells, ncell[d], &ncells)) return false;
    }
    return ncells <= INT32_MAX;
}

static size_t nl_layout(int64_t n, const int64_t *ncell, size_t *bins_bytes) {
    int64_t ncells = ncell[0] * ncell[1] * ncell[2];
    size_t b = cell_bins_bytes(n, ncells);
    *bins_bytes = b;
    b += 256 + (size_t)27 * n * 8;         // slot counts
    b += 256 + (size_t)27 * n * 8;         // slot offsets
    b += 256 + scan_workspace(27 * n);
    return b;
}

extern "C" size_t mps_neighbor_list_workspace(int64_t n, const int64_t *ncell) {
    if (!ncell || !nl_sizes_ok(n, ncell)) return SIZE_MAX;
    size_t bb;
    return nl_layout(n, ncell, &bb) + 256;
}

static int nl_common(const int64_t *cell, int64_t n, const int64_t *ncell, void *ws, size_t ws_bytes, CellBins &cb,
                     int64_t *&slot_cnt, int64_t *&slot_off, void *&scan_tmp, cudaStream_t s) {
    if (n < 0 || !ncell || !ws) return MPS_BAD_ARG;
    if (!nl_sizes_ok(n, ncell)) return MPS_BAD_ARG;
    size_t bb;
    if (ws_bytes < nl_layout(n, ncell, &bb)) return MPS_BAD_ARG;
    int r = cell_bins_build(cell, n, ncell, ws, cb, s);
    if (r) return r;
    char *p = (char *)ws + bb;
    slot_cnt = (int64_t *)carve(p, (size_t)27 * n * 8);
    slot_off = (int64_t *)carve(p, (size_t)27 * n * 8);
    scan_tmp = carve(p, scan_workspace(27 * n));
    return MPS_OK;
}

extern "C" int mps_neighbor_list_count(const int64_t *cell, int64_t n, const int64_t *ncell, void *workspace,
                                       size_t workspace_bytes, int64_t *n_pairs, mps_stream_t stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (!n_pairs) return MPS_BAD_ARG;
    *n_pairs = 0;
    if (n == 0) return MPS_OK;
    CellBins cb;
    int64_t *sc, *so;
    void *st;
    int r = nl_common(cell, n, ncell, workspace, workspace_bytes, cb, sc, so, st, s);
    if (r) return r;
    k_candidate_slots<<<grid_for(27 * n, 256), 256, 0, s>>>(cb.sorted, cb.lin, cb.counts, cb.starts, n, ncell[0],
                                                            ncell[1], ncell[2], sc);
    MPS_LAUNCH_CHECK();
    r = exclusive_scan_i64(sc, so, 27 * n, st, s);
    if (r) return r;
    int64_t last[2];
    MPS_CUDA_TRY(cudaMemcpyAsync(&last[0], so + 27 * n - 1, 8, cudaMemcpyDeviceToHost, s));
    MPS_CUDA_TRY(cudaMemcpyAsync(&last[1], sc + 27 * n - 1, 8, cudaMemcpyDeviceToHost, s));
    MPS_CUDA_TRY(cudaStreamSynchronize(s));
    *n_pairs = last[0] + last[1];
    return MPS_OK;
}

extern "C" int mps_neighbor_list_fill(const int64_t *cell, int64_t n, const int64_t *ncell, void *workspace,
                                      size_t workspace_bytes, int64_t *p1, int64_t *p2, mps_stream_t stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (n == 0) return MPS_OK;
    CellBins cb;
    int64_t *sc, *so;
    void *st;
    int r = nl_common(cell, n, ncell, workspace, workspace_bytes, cb, sc, so, st, s);
    if (r) return r;
    k_candidate_slots<<<grid_for(27 * n, 256), 256, 0, s>>>(cb.sorted, cb.lin, cb.counts, cb.starts, n, ncell[0],
                                                            ncell[1], ncell[2], sc);
    MPS_LAUNCH_CHECK();
    r = exclusive_scan_i64(sc, so, 27 * n, st, s);
    if (r) return r;
    k_candidate_fill<<<grid_for(27 * n, 256), 256, 0, s>>>(cb.sorted, cb.lin, cb.counts, cb.starts, n, ncell[0],
                                                           ncell[1], ncell[2], so, p1, p2);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

extern "C" size_t mps_real_space_pairs_workspace(int64_t n_cand) {
    return 256 * 4 + (size_t)n_cand * 4 + (size_t)n_cand * 8 + scan_workspace(n_cand) + 16;
}

static int pairs_layout(int64_t n_cand, void *ws, size_t ws_bytes, int32_t *&flag, int64_t *&off, void *&tmp,
                        int *&err) {
    if (ws_bytes < mps_real_space_pairs_workspace(n_cand) || !ws) return MPS_BAD_ARG;
    char *p = (char *)ws;
    flag = (int32_t *)carve(p, (size_t)n_cand * 4);
    off = (int64_t *)carve(p, (size_t)n_cand * 8);
    err = (int *)carve(p, 16);
    tmp = carve(p, scan_workspace(n_cand));
    return MPS_OK;
}

extern "C" int mps_real_space_pairs_count(const double *x, int64_t n, const double *box, const int64_t *p1,
                                          const int64_t *p2, int64_t n_cand, double rc, void *workspace,
                                          size_t workspace_bytes, int64_t *n_kept, mps_stream_t stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (!n_kept || !box || n_cand < 0) return MPS_BAD_ARG;
    *n_kept = 0;
    if (n_cand == 0) return MPS_OK;
    int32_t *flag;
    int64_t *off;
    void *tmp;
    int *err;
    int r = pairs_layout(n_cand, workspace, workspace_bytes, flag, off, tmp, err);
    if (r) return r;
    k_pair_flag<<<grid_for(n_cand, 256), 256, 0, s>>>(x, box[0], box[1], box[2], p1, p2, n_cand, rc, flag);
    MPS_LAUNCH_CHECK();
    r = exclusive_scan_i32_to_i64(flag, off, n_cand, tmp, s);
    if (r) return r;
    int64_t lo;
    int32_t lf;
    MPS_CUDA_TRY(cudaMemcpyAsync(&lo, off + n_cand - 1, 8, cudaMemcpyDeviceToHost, s));
    MPS_CUDA_TRY(cudaMemcpyAsync(&lf, flag + n_cand - 1, 4, cudaMemcpyDeviceToHost, s));
    MPS_CUDA_TRY(cudaStreamSynchronize(s));
    *n_kept = lo + lf;
    return MPS_OK;
}

extern "C" int mps_real_space_pairs_fill(const double *x, int64_t n, const double *box, const int64_t *p1,
                                         const int64_t *p2, int64_t n_cand, double rc, const double *perp,
                                         const double *para, const double *rvals, int64_t n_tab, void *workspace,
                                         size_t workspace_bytes, int64_t *p1f, int64_t *p2f, double *rhat, double *A,
                                         double *B, mps_stream_t stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (n_cand == 0) return MPS_OK;
    if (!box || n_tab < 2) return MPS_BAD_ARG;
    int32_t *flag;
    int64_t *off;
    void *tmp;
    int *err;
    int r = pairs_layout(n_cand, workspace, workspace_bytes, flag, off, tmp, err);
    if (r) return r;
    // flags and offsets were produced by _count on the same workspace
    MPS_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), s));
    k_pair_fill<<<grid_for(n_cand, 256), 256, 0, s>>>(x, box[0], box[1], box[2], p1, p2, n_cand, flag, off, perp,
                                                      para, rvals, n_tab, p1f, p2f, rhat, A, B, err);
    MPS_LAUNCH_CHECK();
    int herr = 0;
    MPS_CUDA_TRY(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s));
    MPS_CUDA_TRY(cudaStreamSynchronize(s));
    return herr ? MPS_TABLE_RANGE : MPS_OK;
}