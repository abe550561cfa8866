// Gradient form of the float32 wave-space operator (inner operator of the
// mixed-precision solve).
//
// The reference operator spreads the three moment components onto three grids
// and scales their spectra by H k k^T / |k|^2.  Since k k^T = (ik)(ik)^*, the same
// operator (up to the sampling error of the Gaussian's derivative) is
//   rho(n) = sum_a m_a . grad_r w_a(n)              one scalar grid per vector
//   phi    = IFFT( H / |k|^2 FFT(rho) )
//   E_a    = h^3 sum_n grad_r w_a(n) phi(n)
// with r = node - x_a and grad_r w = -(4 xi^2 / eta_d) r_d w per axis (separable:
// the per-axis factors w_d and g_d = dw_d/dr_d).  One FFT pair per vector instead
// of three, a third of the grid traffic.  It differs from the reference operator
// by the discretisation error of the derivative (about 1e-5 relative at the
// configurations measured), which the float64-accurate refinement residual
// removes: the mixed solve still converges to the reference operator's solution.
//
// The kernels follow the tiled spread / contract of tiles.cu (one CTA per
// 16 x 16 x TZ tile, deterministic, no atomics).
#include "gradop.cuh"

#include <cstdlib>
#include <cstring>

namespace mps {


// g[a][d][j] = dw_d/dr at stencil node j of axis d (float32).
__global__ void k_grad_factors(const double *__restrict__ x, int64_t n, GridParams gp, const double *__restrict__ w64,
                               float *__restrict__ g32) {
    const int P = gp.P;
    const int lo = (P - 1) / 2;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n * 3; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = t / 3;
        const int d = (int)(t % 3);
        const double h = gp.h[d];
        const double xv = x[3 * a + d];
        const double v = __ddiv_rn(xv, h);
        const double af = floor(fabs(v) + 0.5);
        const double node0 = v > 0 ? af : (v < 0 ? -af : 0.0 * af);
        const double base = __dsub_rn(__dmul_rn(node0, h), xv);
        const double c = -4.0 * gp.xi * gp.xi / gp.eta[d];
        for (int j = 0; j < P; ++j) {
            const double r = base + (double)(j - lo) * h;
            g32[(a * 3 + d) * P + j] = (float)(c * r * w64[(a * 3 + d) * P + j]);
        }
    }
}

// H / |k|^2 on the half spectrum (float32), H including 1/G; zero at k = 0.  One
// thread per point of the spectrum's quarter, written to its mirrored points (same
// |k|^2 and H there).
__global__ void k_grad_scale_coef(GridParams gp, const double *__restrict__ H, float *__restrict__ hs) {
    const HalfQuarter q(gp.N);
    const int64_t Gq = q.size();
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < Gq; t += (int64_t)gridDim.x * blockDim.x) {
        int ix, iy, iz;
        q.point(t, &ix, &iy, &iz);
        const double kx = fft_freq(ix, gp.N[0]) * gp.kfac[0];
        const double ky = fft_freq(iy, gp.N[1]) * gp.kfac[1];
        const double kz = fft_freq(iz, gp.N[2]) * gp.kfac[2];
        const double k2 = kx * kx + ky * ky + kz * kz;
        const float v = k2 > 0 ? (float)(H[((int64_t)iz * q.Ny + iy) * q.Nxh + ix] / k2) : 0.f;
        mirror_points(q, ix, iy, iz, [&](int64_t i, int, int) { hs[i] = v; });
    }
}

// Owner-computes spread: thread (tx, ty) of the CTA owns the column (X0+tx,
// Y0+ty, Z0..Z0+TZ-1) of the tile and accumulates it in registers over the
// tile's particle list (fixed order: deterministic, no atomics).  Particles are
// staged in chunks with their per-axis factors already aligned to the tile --
// w and dw/dr at every tile column, row and plane, zero where the stencil does
// not reach -- plus masks of the tile columns, rows and planes they cover, so a
// warp (an 8 x 4 patch of the tile's columns: the particle's 10-wide stencil
// often misses one half of the tile in x, which a warp of two full 16-wide rows
// could not skip) skips a particle with one uniform test and otherwise runs a branch-free
// update: value(x,y,z) = (mx gx wy + my wx gy) wz + mz wx wy gz, over the groups
// of 4 tile planes the particle reaches (a plane mask staged with the factors).
// Staging: a lane aligns one particle's factors to half of one axis and keeps the mask of the positions covered (no
// divisions, no shared-memory atomics); the warps then walk only the particles that reach their patch, from ballots.
// Alone, at depth 12: 0.288 -> 0.217 ms a launch for three vectors of N = 1e5 on 144^3, 0.387 -> 0.241 for one of
// N = 2e5 on 192^3.
// An update of two multiply-adds (not a product, a multiply-add and an addition): 0.223 -> 0.200 ms for the three
// vectors beside the pair sum, 0.244 -> 0.241 for the one.
// particles staged per barrier interval: 96 measured 0.300 ms per launch at the bench workload against 0.323
// for 32 (fewer barriers, and the warps' uneven shares of a chunk even out), 0.306 for 64 and 0.301 for 128
constexpr int kGChunk = 96;

// Bounds of 5 blocks per SM (48 registers, 36.5 KB of shared memory each): 0.293 ms per launch at the bench
// workload against 0.299 at 4 blocks (64 registers), 0.300 at 6 (spills) and 0.342 unbounded.
// Depth 12 (36 accumulators for 3 vectors, 64 registers) at 4 blocks per SM, depth 16 (48) at 3.
template <int TZ, int NR>
__global__ void __launch_bounds__(256, TZ > 12 ? 3 : (TZ > 8 ? 4 : 5))
    k_spread_grad_tiled(const double *__restrict__ m, int64_t n, int r0,
                        const int32_t *__restrict__ start,
                        const float *__restrict__ w, const float *__restrict__ g,
                        GridParams gp, const int64_t *__restrict__ tstart,
                        const int32_t *__restrict__ entries, int ntx, int nty,
                        float *__restrict__ grid) {
    constexpr int kPos = kTileX + kTileY + TZ + 1 - TZ % 2;   // aligned positions per particle (odd: no bank conflicts)
    constexpr int kMS = (3 * NR + 3) & ~3;       // moments, padded to a float4 multiple
    __shared__ float2 s_f[kGChunk][kPos];        // (w, dw/dr) at tile columns, rows, planes
    __shared__ __align__(16) float s_m[kGChunk][kMS];
    __shared__ unsigned s_mask[6][kGChunk];      // positions covered: halves of the columns, rows, planes
    const int64_t t = blockIdx.x;
    const int bx = (int)(t % ntx), by = (int)((t / ntx) % nty), bz = (int)(t / ((int64_t)ntx * nty));
    const int X0 = bx * kTileX, Y0 = by * kTileY, Z0 = bz * TZ;
    // warp wid owns the 8 x 4 patch (columns 8 (wid & 1) .. +8, rows 4 (wid >> 1) .. +4) of the 16 x 16 tile
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int px = wid & 1, py = wid >> 1;
    const int tx = 8 * px + (lane & 7), ty = 4 * py + (lane >> 3);
    const int P = gp.P;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    float acc[TZ][NR];
#pragma unroll
    for (int z = 0; z < TZ; ++z)
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[z][r] = 0.f;
    const int64_t e0 = tstart[t], e1 = tstart[t + 1];
    for (int64_t cb = e0; cb < e1; cb += kGChunk) {
        const int cnt = (int)min((int64_t)kGChunk, e1 - cb);
        if (threadIdx.x < cnt) {
            const int32_t a = entries[cb + threadIdx.x];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const double *ma = m + ((int64_t)(r0 + r) * n + a) * 3;
                s_m[threadIdx.x][3 * r + 0] = (float)ma[0];
                s_m[threadIdx.x][3 * r + 1] = (float)ma[1];
                s_m[threadIdx.x][3 * r + 2] = (float)ma[2];
            }
        }
        // a warp aligns the factors of 32 particles (one per lane) to half of one of the tile's axes, and each lane
        // keeps the mask of the positions its particle covers
        for (int task = wid; task < 6 * (kGChunk / 32); task += 8) {
            const int pp = 32 * (task / 6) + lane, d = (task % 6) >> 1, half = task & 1;
            if (pp >= cnt) continue;
            const int len = d == 2 ? TZ : kTileX, k0 = half ? len / 2 : 0, k1 = half ? len : len / 2;
            const int origin = d == 0 ? X0 : (d == 1 ? Y0 : Z0), Nd = d == 0 ? Nx : (d == 1 ? Ny : Nz);
            const int64_t a = entries[cb + pp];
            int j = origin + k0 - start[3 * a + d];   // stencil index of the first position, in [-N, 2 N)
            if (j < 0) j += Nd;
            if (j >= Nd) j -= Nd;
            const float *wa = w + (a * 3 + d) * P, *ga = g + (a * 3 + d) * P;
            const int base = d * kTileX;
            unsigned mask = 0u;
#pragma unroll 4
            for (int k = k0; k < k1; ++k) {
                const bool hit = j < P && origin + k < Nd;
                s_f[pp][base + k] = hit ? make_float2(wa[j], ga[j]) : make_float2(0.f, 0.f);
                mask |= hit ? 1u << k : 0u;
                if (++j >= Nd) j = 0;
            }
            s_mask[2 * d + half][pp] = mask;
        }
        __syncthreads();
        for (int word = 0; word < cnt; word += 32) {
            // the particles that reach this warp's patch: some of its 4 rows and some of its 8 columns are covered
            bool reach = false;
            if (word + lane < cnt)
                reach = ((s_mask[px][word + lane] >> (8 * px)) & 0xFFu) != 0u &&
                        ((s_mask[2 + (py >> 1)][word + lane] >> (4 * py)) & 0xFu) != 0u;
            for (unsigned list = __ballot_sync(0xffffffffu, reach); list; list &= list - 1) {
                const int pp = word + __ffs(list) - 1;
                const float2 fx = s_f[pp][tx], fy = s_f[pp][kTileX + ty];
                const float gxwy = fx.y * fy.x, wxgy = fx.x * fy.y, wxwy = fx.x * fy.x;
                float cA[NR], cB[NR];
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    cA[r] = s_m[pp][3 * r] * gxwy + s_m[pp][3 * r + 1] * wxgy;
                    cB[r] = s_m[pp][3 * r + 2] * wxwy;
                }
                // planes in groups of 4; a group the particle does not reach is skipped (uniform over the CTA)
                const unsigned planes = s_mask[4][pp] | s_mask[5][pp];
#pragma unroll
                for (int z0 = 0; z0 < TZ; z0 += 4) {
                    if (TZ > 4 && ((planes >> z0) & 0xFu) == 0u) continue;
#pragma unroll
                    for (int z = z0; z < z0 + 4 && z < TZ; ++z) {
                        const float2 fz = s_f[pp][kTileX + kTileY + z];
#pragma unroll
                        for (int r = 0; r < NR; ++r) {   // (one sum a + b on the right is three instructions, this two)
                            acc[z][r] += cA[r] * fz.x;
                            acc[z][r] += cB[r] * fz.y;
                        }
                    }
                }
            }
        }
        __syncthreads();
    }
    const int gxn = X0 + tx, gyn = Y0 + ty;
    if (gxn < Nx && gyn < Ny) {
        const int64_t G = gp.G;
#pragma unroll
        for (int z = 0; z < TZ; ++z) {
            const int gz = Z0 + z;
            if (gz < Nz) {
                const int64_t node = ((int64_t)gz * Ny + gyn) * Nx + gxn;
#pragma unroll
                for (int r = 0; r < NR; ++r) grid[(int64_t)(r0 + r) * G + node] = acc[z][r];
            }
        }
    }
}


constexpr int kGRowPad = kTileX + 1;

template <int TZ, int NR>
__global__ void __launch_bounds__(256) k_contract_grad_tiled(const float *__restrict__ grid, int r0,
                                                             const int32_t *__restrict__ start,
                                                             const float *__restrict__ w, const float *__restrict__ g,
                                                             GridParams gp, const int64_t *__restrict__ tstart,
                                                             const int32_t *__restrict__ entries, int ntx, int nty,
                                                             float *__restrict__ partial) {
    constexpr int kPlane = kTileY * kGRowPad;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *tile = (float *)smem_raw;                        // [NR][TZ][16][17]
    float *wbuf = tile + NR * TZ * kPlane;                  // [8 warps][2][3*kMaxP]
    const int64_t t = blockIdx.x;
    const int bx = (int)(t % ntx), by = (int)((t / ntx) % nty), bz = (int)(t / ((int64_t)ntx * nty));
    const int X0 = bx * kTileX, Y0 = by * kTileY, Z0 = bz * TZ;
    const int tx = threadIdx.x & (kTileX - 1), ty = threadIdx.x >> 4;
    const int P = gp.P;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const int64_t G = gp.G;
    const int64_t e0 = tstart[t], e1 = tstart[t + 1];
    if (e0 == e1) return;
    {
        const int gxn = X0 + tx, gyn = Y0 + ty;
        const bool in = gxn < Nx && gyn < Ny;
#pragma unroll
        for (int z = 0; z < TZ; ++z) {
            const int gz = Z0 + z;
            const int64_t node = ((int64_t)gz * Ny + gyn) * Nx + gxn;
#pragma unroll
            for (int r = 0; r < NR; ++r)
                tile[(r * TZ + z) * kPlane + ty * kGRowPad + tx] =
                    (in && gz < Nz) ? grid[(int64_t)(r0 + r) * G + node] : 0.f;
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float *wb = wbuf + wid * 2 * 3 * kMaxP;
    float *gb = wb + 3 * kMaxP;
    for (int64_t e = e0 + wid; e < e1; e += 8) {
        const int32_t a = entries[e];
        int ox = X0 - start[3 * a], oy = Y0 - start[3 * a + 1], oz = Z0 - start[3 * a + 2];
        if (ox < 0) ox += Nx;
        if (oy < 0) oy += Ny;
        if (oz < 0) oz += Nz;
        for (int k = lane; k < 3 * P; k += 32) {
            wb[(k / P) * kMaxP + (k % P)] = w[(int64_t)a * 3 * P + k];
            gb[(k / P) * kMaxP + (k % P)] = g[(int64_t)a * 3 * P + k];
        }
        int xr = lane - ox, yr = lane - oy, zr = lane - oz;
        if (xr < 0) xr += Nx;
        if (yr < 0) yr += Ny;
        if (zr < 0) zr += Nz;
        const unsigned mx = __ballot_sync(0xffffffffu, lane < P && xr < kTileX && X0 + xr < Nx);
        const unsigned my = __ballot_sync(0xffffffffu, lane < P && yr < kTileY && Y0 + yr < Ny);
        const unsigned mz = __ballot_sync(0xffffffffu, lane < P && zr < TZ && Z0 + zr < Nz);
        __syncwarp();
        const int nx = __popc(mx), ny = __popc(my);
        float acc[3 * NR];
#pragma unroll
        for (int c = 0; c < 3 * NR; ++c) acc[c] = 0.f;
        for (int q = lane; q < nx * ny; q += 32) {
            const int jx = (int)__fns(mx, 0, q % nx + 1), jy = (int)__fns(my, 0, q / nx + 1);
            int xx = jx - ox, yy = jy - oy;
            if (xx < 0) xx += Nx;
            if (yy < 0) yy += Ny;
            float s0[NR], s1[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) s0[r] = s1[r] = 0.f;
            unsigned mzz = mz;
            while (mzz) {
                const int jz = __ffs(mzz) - 1;
                mzz &= mzz - 1;
                int zz = jz - oz;
                if (zz < 0) zz += Nz;
                const float wz = wb[2 * kMaxP + jz], gz = gb[2 * kMaxP + jz];
                const float *tp = tile + zz * kPlane + yy * kGRowPad + xx;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const float v = tp[r * TZ * kPlane];
                    s0[r] += v * wz;
                    s1[r] += v * gz;
                }
            }
            const float wx = wb[jx], wy = wb[kMaxP + jy], gx = gb[jx], gy = gb[kMaxP + jy];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                acc[3 * r + 0] += gx * wy * s0[r];
                acc[3 * r + 1] += wx * gy * s0[r];
                acc[3 * r + 2] += wx * wy * s1[r];
            }
        }
#pragma unroll
        for (int c = 0; c < 3 * NR; ++c) acc[c] = warp_sum(acc[c]);
        if (lane == 0) {
#pragma unroll
            for (int c = 0; c < 3 * NR; ++c) partial[e * 3 * NR + c] = acc[c];
        }
        __syncwarp();
    }
}

// Each particle's partials summed in its fixed tile order (float64 accumulation).
template <int NR>
__global__ void k_contract_grad_gather(const float *__restrict__ partial, int64_t n, int r0,
                                       const int64_t *__restrict__ pstart, const int32_t *__restrict__ pentry,
                                       double hprod, double *__restrict__ out) {
    constexpr int C = 3 * NR;
    for (int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; a < n; a += (int64_t)gridDim.x * blockDim.x) {
        double acc[C];
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c] = 0.0;
        for (int64_t k = pstart[a]; k < pstart[a + 1]; ++k) {
            const float *pp = partial + (int64_t)pentry[k] * C;
#pragma unroll
            for (int c = 0; c < C; ++c) acc[c] += (double)pp[c];
        }
#pragma unroll
        for (int r = 0; r < NR; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) out[((int64_t)(r0 + r) * n + a) * 3 + c] = acc[3 * r + c] * hprod;
    }
}

// The columns of a stencil by rounds of a warp, for the contractions below: lane's column (jx, jy) of a round, the
// planes sub, sub + lpp, ... of it; false: none.  For the supports of the staged contraction (8 and 10) the columns
// that a round reads together lie in different banks of its region, whose rows are 20 floats apart: 8 x 4 columns of
// every other row, then the edge of 10 x 10, 24 columns and 12 with two lanes each.  Elsewhere 32 consecutive columns a
// round.
__host__ __device__ constexpr int grad_rounds(int P) { return P == 8 ? 2 : (P == 10 ? 4 : (P * P + 31) / 32); }

__device__ __forceinline__ bool grad_column(int P, int round, int lane, int *jx, int *jy, int *sub, int *lpp) {
    *sub = 0;
    *lpp = 1;
    if (P != 8 && P != 10) {
        int idx;
        if (!stencil_row(32 * round, P, lane, &idx, sub, lpp)) return false;
        *jx = idx % P;
        *jy = idx / P;
        return true;
    }
    if (round < 2) {
        *jx = lane & 7;
        *jy = 2 * (lane >> 3) + round;
        return true;
    }
    if (round == 2) {
        const int e = lane - 16;   // columns 8 and 9 of rows 0, 1, 2, 5
        *jx = e < 0 ? lane & 7 : 8 + (e & 1);
        *jy = e < 0 ? 8 + (lane >> 3) : (e < 6 ? e >> 1 : 5);
        return lane < 24;
    }
    const int c = lane < 12 ? lane : lane - 12, q = c >> 1;   // columns 8 and 9 of rows 3, 4, 6, 7, 8, 9
    *jx = 8 + (c & 1);
    *jy = q < 2 ? 3 + q : 4 + q;
    *sub = lane < 12 ? 0 : 1;
    *lpp = 2;
    return lane < 24;
}

// Contraction as a warp-per-particle gather: the grids of the gradient form (one
// per vector) are small enough to be read mostly from L2.  Lanes take the (x, y)
// columns of the stencil, each runs its z column; fixed summation order.  Warps
// visit particles in `order` (spatially sorted: the warps of one CTA read
// overlapping stencils, so much of it comes from L1); null = input order.
// 3 blocks per SM (79 registers for 3 vectors, no spills): 0.283 ms per launch at the bench workload against 0.293
// with the 64-register cap of 4 blocks (which spills) and 0.338 with 2 blocks
template <int NR>
__global__ void __launch_bounds__(256, 3) k_contract_grad_warp(const float *__restrict__ grid, int64_t n, int r0,
                                                            const int32_t *__restrict__ order,
                                                            const int32_t *__restrict__ start,
                                                            const float *__restrict__ w, const float *__restrict__ g,
                                                            GridParams gp, double *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int oc = warp_sums_index<3 * NR>(lane);   // the output component this lane writes
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int P = gp.P;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const int64_t G = gp.G;
    for (int64_t i = warp; i < n; i += nw) {
        const int64_t a = order ? order[i] : i;
        const int sx = start[3 * a], sy = start[3 * a + 1], sz = start[3 * a + 2];
        const float *wa = w + a * 3 * P, *ga = g + a * 3 * P;
        float acc[3 * NR];
#pragma unroll
        for (int c = 0; c < 3 * NR; ++c) acc[c] = 0.f;
        for (int round = 0; round < grad_rounds(P); ++round) {
            int jx, jy, sub, lpp;
            if (!grad_column(P, round, lane, &jx, &jy, &sub, &lpp)) continue;
            int ix = sx + jx;
            if (ix >= Nx) ix -= Nx;
            int iy = sy + jy;
            if (iy >= Ny) iy -= Ny;
            const int64_t rowb = (int64_t)ix + (int64_t)Nx * iy;
            float s0[NR], s1[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) s0[r] = s1[r] = 0.f;
            // unrolled over the whole z run of P = 10 (10 x NR loads in flight per lane; 5 and 2 measured slower)
#pragma unroll 10
            for (int jz = sub; jz < P; jz += lpp) {
                int iz = sz + jz;
                if (iz >= Nz) iz -= Nz;
                const int64_t node = rowb + (int64_t)Nx * Ny * iz;
                const float wz = wa[2 * P + jz], gz = ga[2 * P + jz];
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const float v = __ldg(grid + (int64_t)(r0 + r) * G + node);
                    s0[r] += v * wz;
                    s1[r] += v * gz;
                }
            }
            const float wx = wa[jx], wy = wa[P + jy], gx = ga[jx], gy = ga[P + jy];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                acc[3 * r + 0] += gx * wy * s0[r];
                acc[3 * r + 1] += wx * gy * s0[r];
                acc[3 * r + 2] += wx * wy * s1[r];
            }
        }
        const float v = warp_sums(acc, lane);
        if (oc >= 0) out[((int64_t)(r0 + oc / 3) * n + a) * 3 + oc % 3] = float_to_double(v) * gp.hprod;
    }
}

// Contraction by home blocks (the default where the support is 8 or 10): one CTA per kHomeBlock^3 block of grid nodes
// stages every node its particles' stencils can reach -- the block grown by P - 1 nodes per axis, one plane of nodes
// per vector -- in shared memory, and its particles' offsets and per-axis factors (kHomeChunk particles at a time).
// One warp per particle then runs the sums of k_contract_grad_warp in the same order, from shared memory and registers
// instead of L2: the results are bit-identical.  P is a template parameter, so the z runs unroll completely with the z
// factors in registers and the shared-memory offsets are immediates.  A node is staged by about (1 + (P - 1) / 8)^3
// blocks (9.6 at P = 10), all from L2; with one vector a CTA takes three home blocks along y (6.2).  Shared memory
// bounds it (a node's read and its staging), so the rows lie 20 floats apart: the columns that a round of the warp
// reads together then hit different banks (grad_column), and a row is staged by five 16-byte copies.  The sums end one
// to a lane, converted and scaled together: lane 0's 3 NR conversions and multiplications had cost a warp 6 NR float64
// instructions a particle.  Three vectors of N = 1e5 on 144^3 / one of N = 2e5 on 192^3: 0.209 / 0.155 ms with two-way
// bank conflicts, staging by single floats and lane 0's epilogue; 0.168 / 0.136 with the sums one to a lane and
// asynchronous copies; 0.118 / 0.109 so.  78 KB of shared memory at P = 10 and 3 vectors, 3 blocks per SM (80
// registers); float4 nodes (the 3 vectors interleaved, 2 blocks per SM) were slower.
constexpr int kHomeChunk = 24;
constexpr int kHomeRow = 20;   // floats from one row of the region to the next (grad_column), whole 16-byte pieces

// A CTA covers BY home blocks along y: the margin of P - 1 nodes is staged once for all of them.
template <int NR, int P, int BY>
struct HomeTile {
    static constexpr int RX = kHomeBlock + P - 1, RY = BY * kHomeBlock + P - 1, RZ = kHomeBlock + P - 1;
    static constexpr int VOL = kHomeRow * RY * RZ;
    static_assert(RX <= kHomeRow, "a row holds the region's columns");
    static constexpr size_t smem =
        sizeof(float) * ((size_t)NR * VOL + 2 * kHomeChunk * 3 * P) + sizeof(int) * 4 * kHomeChunk;
};

template <int NR, int P, int BY>
__global__ void __launch_bounds__(256, NR == 1 ? 4 : 3) k_contract_grad_home(
    const float *__restrict__ grid, int64_t n, int r0, const int64_t *__restrict__ hstart,
    const int32_t *__restrict__ hentries, int nbx, int nby, const int32_t *__restrict__ start,
    const float *__restrict__ w, const float *__restrict__ g, GridParams gp, double *__restrict__ out) {
    using HT = HomeTile<NR, P, BY>;
    constexpr int RX = HT::RX, RY = HT::RY, RZ = HT::RZ, VOL = HT::VOL, RS = kHomeRow, RR = RS * RY;
    constexpr int F = 3 * P;                        // per-axis factors of one particle
    extern __shared__ __align__(16) float s_reg[];  // [NR][VOL] nodes, x fastest
    float *s_w = s_reg + NR * VOL;                  // [kHomeChunk][F]
    float *s_g = s_w + kHomeChunk * F;              // [kHomeChunk][F]
    int *s_p = (int *)(s_g + kHomeChunk * F);       // [kHomeChunk][4]: offsets in the block, particle id
    const int tby = (nby + BY - 1) / BY;
    const int64_t b = blockIdx.x;
    const int bx = (int)(b % nbx), by0 = (int)((b / nbx) % tby) * BY, bz = (int)(b / ((int64_t)nbx * tby));
    // the home blocks' particle lists, one after the other
    int64_t first[BY];
    int upto[BY], total = 0;
#pragma unroll
    for (int k = 0; k < BY; ++k) {
        first[k] = 0;
        if (by0 + k < nby) {
            const int64_t hb = ((int64_t)bz * nby + by0 + k) * nbx + bx;
            first[k] = hstart[hb] - total;
            total += (int)(hstart[hb + 1] - hstart[hb]);
        }
        upto[k] = total;
    }
    if (total == 0) return;   // the whole CTA leaves: no barrier is left waiting
    auto entry = [&](int q) {
        int64_t e = first[0];
#pragma unroll
        for (int k = 1; k < BY; ++k) e = q >= upto[k - 1] ? first[k] : e;
        return (int64_t)hentries[e + q];
    };
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2];
    const int64_t G = gp.G;
    const int X0 = bx * kHomeBlock, Y0 = by0 * kHomeBlock, Z0 = bz * kHomeBlock;
    const float *g0 = grid + (int64_t)r0 * G;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int oc = warp_sums_index<3 * NR>(lane);   // the output component this lane writes
    // origin + offset < 3 N (the host requires it): at most two wraps
    auto wrap2 = [](int i, int N) {
        i -= i >= N ? N : 0;
        return i - (i >= N ? N : 0);
    };
    if (Nx % 4 == 0) {   // rows by 16-byte pieces: X0 is a multiple of 8, so no piece wraps within
        constexpr int PC = RS / 4;
        for (int i = threadIdx.x; i < RY * RZ * PC; i += 256) {
            const int row = i / PC, c = i - row * PC, z = row / RY, y = row - z * RY;
            const float *src = g0 + ((int64_t)wrap2(Z0 + z, Nz) * Ny + wrap2(Y0 + y, Ny)) * Nx + wrap2(X0 + 4 * c, Nx);
#pragma unroll
            for (int r = 0; r < NR; ++r)
                copy_async((float4 *)(s_reg + r * VOL + row * RS + 4 * c), (const float4 *)(src + r * G));
        }
    } else {
        for (int i = threadIdx.x; i < RY * RZ * RX; i += 256) {
            const int row = i / RX, x = i - row * RX, z = row / RY, y = row - z * RY;
            const float *src = g0 + ((int64_t)wrap2(Z0 + z, Nz) * Ny + wrap2(Y0 + y, Ny)) * Nx + wrap2(X0 + x, Nx);
#pragma unroll
            for (int r = 0; r < NR; ++r) copy_async(s_reg + r * VOL + row * RS + x, src + r * G);
        }
    }
    for (int c0 = 0; c0 < total; c0 += kHomeChunk) {
        const int cnt = min(kHomeChunk, total - c0);
        for (int q = threadIdx.x; q < cnt * F; q += 256) {
            const int p = q / F, k = q - p * F;
            const int64_t a = entry(c0 + p);
            s_w[q] = w[a * F + k];
            s_g[q] = g[a * F + k];
        }
        if (threadIdx.x < cnt) {
            const int64_t a = entry(c0 + threadIdx.x);
            // a home block holds the stencil's first node: offsets in [0, kHomeBlock), in y [0, BY kHomeBlock)
            s_p[4 * threadIdx.x + 0] = start[3 * a] - X0;
            s_p[4 * threadIdx.x + 1] = start[3 * a + 1] - Y0;
            s_p[4 * threadIdx.x + 2] = start[3 * a + 2] - Z0;
            s_p[4 * threadIdx.x + 3] = (int)a;
        }
        copy_async_wait();
        __syncthreads();   // the region (first pass) and this chunk's particle data are in place
        for (int pp = wid; pp < cnt; pp += 8) {
            const int ox = s_p[4 * pp], oy = s_p[4 * pp + 1], oz = s_p[4 * pp + 2];
            const int64_t a = s_p[4 * pp + 3];
            const float *wa = s_w + pp * F, *ga = s_g + pp * F;
            float wz[P], gz[P];
#pragma unroll
            for (int j = 0; j < P; ++j) {
                wz[j] = wa[2 * P + j];
                gz[j] = ga[2 * P + j];
            }
            float acc[3 * NR];
#pragma unroll
            for (int c = 0; c < 3 * NR; ++c) acc[c] = 0.f;
#pragma unroll
            for (int round = 0; round < grad_rounds(P); ++round) {
                int jx, jy, sub, lpp;   // lpp is a constant of each unrolled round
                if (!grad_column(P, round, lane, &jx, &jy, &sub, &lpp)) continue;
                const float *col = s_reg + (oz * RY + oy + jy) * RS + ox + jx;
                float s0[NR], s1[NR];
#pragma unroll
                for (int r = 0; r < NR; ++r) s0[r] = s1[r] = 0.f;
                if (lpp == 1) {
#pragma unroll
                    for (int jz = 0; jz < P; ++jz) {
#pragma unroll
                        for (int r = 0; r < NR; ++r) {
                            const float v = col[r * VOL + jz * RR];
                            s0[r] += v * wz[jz];
                            s1[r] += v * gz[jz];
                        }
                    }
                } else {
                    for (int jz = sub; jz < P; jz += lpp) {
                        const float wzj = wa[2 * P + jz], gzj = ga[2 * P + jz];
#pragma unroll
                        for (int r = 0; r < NR; ++r) {
                            const float v = col[r * VOL + jz * RR];
                            s0[r] += v * wzj;
                            s1[r] += v * gzj;
                        }
                    }
                }
                const float wx = wa[jx], wy = wa[P + jy], gx = ga[jx], gy = ga[P + jy];
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    acc[3 * r + 0] += gx * wy * s0[r];
                    acc[3 * r + 1] += wx * gy * s0[r];
                    acc[3 * r + 2] += wx * wy * s1[r];
                }
            }
            const float v = warp_sums(acc, lane);
            if (oc >= 0) out[((int64_t)(r0 + oc / 3) * n + a) * 3 + oc % 3] = float_to_double(v) * gp.hprod;
        }
        __syncthreads();   // this chunk's particle data is read before the next chunk overwrites it
    }
}

bool contract_grad_home_supported(const GridParams &gp) {
    if (gp.P != 8 && gp.P != 10) return false;
    for (int d = 0; d < 3; ++d)
        if (gp.N[d] < kHomeBlock || gp.N[d] < gp.P) return false;
    return true;
}

template <int NR, int P, int BY>
static int home_launch(const float *grid, int64_t n, int r0, const int32_t *start, const float *w, const float *g,
                       const GridParams &gp, const TileBins &tb, double *out, cudaStream_t s) {
    constexpr size_t smem = HomeTile<NR, P, BY>::smem;
    if (smem > 48 * 1024)
        MPS_CUDA_TRY(cudaFuncSetAttribute(k_contract_grad_home<NR, P, BY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
    const unsigned blocks = (unsigned)tb.nhb[0] * (unsigned)((tb.nhb[1] + BY - 1) / BY) * (unsigned)tb.nhb[2];
    k_contract_grad_home<NR, P, BY><<<blocks, 256, smem, s>>>(grid, n, r0, tb.hstart, tb.hentries, tb.nhb[0],
                                                                  tb.nhb[1], start, w, g, gp, out);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

// One vector leaves room for three home blocks to a CTA: taken where every SM still gets four CTAs and the longer
// region wraps at most twice.
template <int P>
static int home_dispatch(const float *grid, int64_t n, int nrhs, const int32_t *start, const float *w, const float *g,
                         const GridParams &gp, const TileBins &tb, double *out, cudaStream_t s) {
    const bool wide = tb.nhome >= 3 * 4 * 152 && gp.N[1] >= 16;
    for (int r0 = 0; r0 < nrhs; r0 += 3) {
        const int nr = min(3, nrhs - r0);
        const int rc = nr == 3   ? home_launch<3, P, 1>(grid, n, r0, start, w, g, gp, tb, out, s)
                       : nr == 2 ? home_launch<2, P, 1>(grid, n, r0, start, w, g, gp, tb, out, s)
                       : wide    ? home_launch<1, P, 3>(grid, n, r0, start, w, g, gp, tb, out, s)
                                 : home_launch<1, P, 1>(grid, n, r0, start, w, g, gp, tb, out, s);
        if (rc) return rc;
    }
    return MPS_OK;
}

int contract_grad_home(const float *grid, int64_t n, int nrhs, const int32_t *start, const float *w, const float *g,
                       const GridParams &gp, const TileBins &tb, double *out, cudaStream_t s) {
    if (!tb.has_home || !contract_grad_home_supported(gp)) return MPS_BAD_ARG;
    if (gp.P == 10) return home_dispatch<10>(grid, n, nrhs, start, w, g, gp, tb, out, s);
    return home_dispatch<8>(grid, n, nrhs, start, w, g, gp, tb, out, s);
}

int contract_grad_warp(const float *grid, int64_t n, int nrhs, const int32_t *order, const int32_t *start,
                       const float *w, const float *g, const GridParams &gp, double *out, cudaStream_t s) {
    const unsigned blocks = grid_for(n * 32, 256, 152 * 64);
    for (int r0 = 0; r0 < nrhs; r0 += 3) {
        const int nr = min(3, nrhs - r0);
        if (nr == 3)
            k_contract_grad_warp<3><<<blocks, 256, 0, s>>>(grid, n, r0, order, start, w, g, gp, out);
        else if (nr == 2)
            k_contract_grad_warp<2><<<blocks, 256, 0, s>>>(grid, n, r0, order, start, w, g, gp, out);
        else
            k_contract_grad_warp<1><<<blocks, 256, 0, s>>>(grid, n, r0, order, start, w, g, gp, out);
        MPS_LAUNCH_CHECK();
    }
    return MPS_OK;
}

int grad_factors(const double *x, int64_t n, const GridParams &gp, const double *w64, float *g32, cudaStream_t s) {
    k_grad_factors<<<grid_for(3 * n, 256), 256, 0, s>>>(x, n, gp, w64, g32);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int grad_scale_coef(const GridParams &gp, const double *H, float *hs, cudaStream_t s) {
    k_grad_scale_coef<<<grid_for(HalfQuarter(gp.N).size(), 256), 256, 0, s>>>(gp, H, hs);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template <int TZ, int NR>
static int grad_launch(const double *m, int64_t n, int r0, const int32_t *start, const float *w, const float *g,
                       const GridParams &gp, const TileBins &tb, float *grid, float *partial, double *out,
                       bool spread_phase, cudaStream_t s) {
    if (spread_phase) {
        k_spread_grad_tiled<TZ, NR><<<(unsigned)tb.ntiles, 256, 0, s>>>(m, n, r0, start, w, g, gp, tb.tile_start,
                                                                         tb.entries, tb.ntx, tb.nty, grid);
        MPS_LAUNCH_CHECK();
        return MPS_OK;
    }
    const size_t smem = sizeof(float) * ((size_t)NR * TZ * kTileY * kGRowPad + 8 * 2 * 3 * kMaxP);
    if (smem > 48 * 1024)
        MPS_CUDA_TRY(cudaFuncSetAttribute(k_contract_grad_tiled<TZ, NR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
    k_contract_grad_tiled<TZ, NR><<<(unsigned)tb.ntiles, 256, smem, s>>>(grid, r0, start, w, g, gp, tb.tile_start,
                                                                          tb.entries, tb.ntx, tb.nty, partial);
    MPS_LAUNCH_CHECK();
    k_contract_grad_gather<NR><<<grid_for(n, 256), 256, 0, s>>>(partial, n, r0, tb.pstart, tb.pentry, gp.hprod, out);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template <int TZ>
static int grad_dispatch(const double *m, int64_t n, int nrhs, const int32_t *start, const float *w, const float *g,
                         const GridParams &gp, const TileBins &tb, float *grid, float *partial, double *out,
                         bool spread_phase, cudaStream_t s) {
    for (int r0 = 0; r0 < nrhs; r0 += 3) {
        const int nr = min(3, nrhs - r0);
        int rc = nr == 3   ? grad_launch<TZ, 3>(m, n, r0, start, w, g, gp, tb, grid, partial, out, spread_phase, s)
                 : nr == 2 ? grad_launch<TZ, 2>(m, n, r0, start, w, g, gp, tb, grid, partial, out, spread_phase, s)
                           : grad_launch<TZ, 1>(m, n, r0, start, w, g, gp, tb, grid, partial, out, spread_phase, s);
        if (rc) return rc;
    }
    return MPS_OK;
}

template <int TZ>
static int spread_grad_deep(const double *m, int64_t n, int nrhs, const int32_t *start, const float *w,
                            const float *g, const GridParams &gp, const TileBins &tb, float *grid, cudaStream_t s) {
    for (int r0 = 0; r0 < nrhs; r0 += 3) {
        const int nr = min(3, nrhs - r0);
        const unsigned blocks = (unsigned)tb.ntiles;
        if (nr == 3)
            k_spread_grad_tiled<TZ, 3><<<blocks, 256, 0, s>>>(m, n, r0, start, w, g, gp, tb.tile_start, tb.entries,
                                                              tb.ntx, tb.nty, grid);
        else if (nr == 2)
            k_spread_grad_tiled<TZ, 2><<<blocks, 256, 0, s>>>(m, n, r0, start, w, g, gp, tb.tile_start, tb.entries,
                                                              tb.ntx, tb.nty, grid);
        else
            k_spread_grad_tiled<TZ, 1><<<blocks, 256, 0, s>>>(m, n, r0, start, w, g, gp, tb.tile_start, tb.entries,
                                                              tb.ntx, tb.nty, grid);
        MPS_LAUNCH_CHECK();
    }
    return MPS_OK;
}

int spread_grad_tiled(const double *m, int64_t n, int nrhs, const int32_t *start, const float *w, const float *g,
                      const GridParams &gp, const TileBins &tb, float *grid, cudaStream_t s) {
    if (tb.tz == 16) return spread_grad_deep<16>(m, n, nrhs, start, w, g, gp, tb, grid, s);
    if (tb.tz == 12) return spread_grad_deep<12>(m, n, nrhs, start, w, g, gp, tb, grid, s);
    if (tb.tz == 8) return grad_dispatch<8>(m, n, nrhs, start, w, g, gp, tb, grid, nullptr, nullptr, true, s);
    if (tb.tz == 4) return grad_dispatch<4>(m, n, nrhs, start, w, g, gp, tb, grid, nullptr, nullptr, true, s);
    return MPS_BAD_ARG;
}

int contract_grad_tiled(const float *grid, int64_t n, int nrhs, const int32_t *start, const float *w, const float *g,
                        const GridParams &gp, const TileBins &tb, float *partial, double *out, cudaStream_t s) {
    float *gr = const_cast<float *>(grid);
    if (tb.tz == 8) return grad_dispatch<8>(nullptr, n, nrhs, start, w, g, gp, tb, gr, partial, out, false, s);
    if (tb.tz == 4) return grad_dispatch<4>(nullptr, n, nrhs, start, w, g, gp, tb, gr, partial, out, false, s);
    return MPS_BAD_ARG;
}

}  // namespace mps
