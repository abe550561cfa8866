// Point-dipole pair forces and energies for fixed dipoles
// (CPU - HOOMD simulation test/dipole_forces_ext/_dipole_forces_ext.cpp:119-452).
//
// One warp per particle walks the 27 surrounding cells (cell edge >= r_cut, at
// least 3 cells per axis): every pair is evaluated from both ends, so
// forces and energies need no atomics and the summation order is fixed.  The
// pair terms are the reference's: minimum image d - L rint(d/L) (z only when
// periodic), 1e-24 <= r^2 <= r_cut^2,
//   U = pref [(mi.mj)/r^3 - 3 (mi.r)(mj.r)/r^5], half to each particle,
//   F_i = 3 pref / r^5 [(mi.mj) r + (mj.r) mi + (mi.r) mj - 5 (mi.r)(mj.r) r / r^2].
#include "cellwalk.cuh"

namespace mps {

// About one candidate in six lies inside r_cut.  The walk screens candidates in float32 and the float64 pair terms run
// on 32 kept pairs at a time: they are what GB300's float64 rate bounds (20,000 dipoles, 69 neighbours of 442
// candidates each: the whole call from host arrays takes 0.46 ms; with one thread a particle and every candidate in
// float64 this kernel alone took 3.27 ms of 3.56).
__global__ void __launch_bounds__(128) k_dipole_forces(const double *__restrict__ pos, const double *__restrict__ dip,
                                                       int64_t n, Box3 box, Box3 inv_box, int periodic_z, double rc2,
                                                       double pref, const int32_t *__restrict__ lin,
                                                       const int32_t *__restrict__ counts,
                                                       const int64_t *__restrict__ starts,
                                                       const float4 *__restrict__ xs, NearBox nb, int64_t ncx,
                                                       int64_t ncy, int64_t ncz, double *__restrict__ F,
                                                       double *__restrict__ pe) {
    __shared__ int32_t q[4][kNearQueue];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; s < n; s += nw) {
        const float4 pa = xs[s];
        const int64_t i = __float_as_int(pa.w);
        const double xi = pos[3 * i], yi = pos[3 * i + 1], zi = pos[3 * i + 2];
        const double mxi = dip[3 * i], myi = dip[3 * i + 1], mzi = dip[3 * i + 2];
        const CellWalk cw = cell_walk(lin[i], lane, counts, starts, ncx, ncy, ncz);
        double fx = 0.0, fy = 0.0, fz = 0.0, e = 0.0;
        near_walk(cw, lane, xs, pa, (int32_t)i, nb, q[wid], [&](int32_t j) {
            double dx = xi - pos[3 * (int64_t)j], dy = yi - pos[3 * (int64_t)j + 1], dz = zi - pos[3 * (int64_t)j + 2];
            // a quotient that rounds to the other side of a half belongs to a separation of half a box, beyond r_cut
            dx -= box.L[0] * rint(dx * inv_box.L[0]);
            dy -= box.L[1] * rint(dy * inv_box.L[1]);
            if (periodic_z) dz -= box.L[2] * rint(dz * inv_box.L[2]);
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (r2 > rc2 || r2 < 1e-24) return;
            const double inv_r = rsqrt(r2);
            double inv_r2 = inv_r * inv_r;
            inv_r2 = fma(inv_r2, fma(-r2, inv_r2, 1.0), inv_r2);   // the rounding of the square taken out
            const double inv_r3 = inv_r2 * inv_r;
            const double inv_r5 = inv_r3 * inv_r2;
            const double *mj = dip + 3 * (int64_t)j;
            const double mxj = mj[0], myj = mj[1], mzj = mj[2];
            const double mimj = mxi * mxj + myi * myj + mzi * mzj;
            const double mir = mxi * dx + myi * dy + mzi * dz;
            const double mjr = mxj * dx + myj * dy + mzj * dz;
            const double mm = mir * mjr;
            const double coef = pref * 3.0 * inv_r5;
            const double sd = mimj - 5.0 * mm * inv_r2;
            fx += coef * (sd * dx + mjr * mxi + mir * mxj);
            fy += coef * (sd * dy + mjr * myi + mir * myj);
            fz += coef * (sd * dz + mjr * mzi + mir * mzj);
            e += 0.5 * (pref * (mimj * inv_r3 - 3.0 * mm * inv_r5));
        });
        const double v = warp_sum4(fx, fy, fz, e, lane);
        if ((lane & 7) == 0) *(lane < 24 ? F + 3 * i + lane / 8 : pe + i) = v;
    }
}

}  // namespace mps

using namespace mps;

extern "C" int mps_dipole_forces(const double *pos, const double *dip, int64_t n, const double *box, double r_cut,
                                 double prefactor, int32_t periodic_z, double *forces, double *pe,
                                 mps_stream_t stream) {
    if (n < 0 || !box || (n > 0 && (!pos || !dip || !forces || !pe))) return MPS_BAD_ARG;
    for (int d = 0; d < 3; ++d)
        if (!(box[d] > 0)) return MPS_BAD_ARG;
    if (!(r_cut > 0)) return MPS_BAD_ARG;
    if (r_cut >= 0.5 * fmin(box[0], box[1])) return MPS_RC_GT_HALF_BOX;
    if (periodic_z && r_cut >= 0.5 * box[2]) return MPS_RC_GT_HALF_BOX;
    if (n == 0) return MPS_OK;
    cudaStream_t s = (cudaStream_t)stream;
    int64_t ncell[3];
    compute_ncell(box, r_cut, ncell);
    if (!cells_fit(ncell)) return MPS_BAD_ARG;
    const int64_t ncells = ncell[0] * ncell[1] * ncell[2];
    int64_t *cell3 = nullptr;
    void *bins = nullptr;
    float4 *xs = nullptr;
    MPS_CUDA_TRY(cudaMallocAsync((void **)&cell3, sizeof(int64_t) * 3 * n, s));
    if (cudaMallocAsync(&bins, cell_bins_bytes(n, ncells), s) != cudaSuccess ||
        cudaMallocAsync((void **)&xs, sizeof(float4) * n, s) != cudaSuccess) {
        set_last_error(cudaGetLastError(), "cudaMallocAsync", __FILE__, __LINE__);
        cudaFreeAsync(cell3, s);
        if (bins) cudaFreeAsync(bins, s);
        return MPS_CUDA_ERR;
    }
    const bool per[3] = {true, true, periodic_z != 0};
    const Box3 b3{{box[0], box[1], box[2]}}, inv3{{1.0 / box[0], 1.0 / box[1], 1.0 / box[2]}};
    const NearBox nb = make_near_box(box, r_cut, per);
    CellBins cb;
    int rc = cell_assign(pos, n, box, ncell, cell3, s);
    if (!rc) rc = cell_bins_build(cell3, n, ncell, bins, cb, s);
    if (!rc) rc = near_positions(pos, cb.sorted, n, b3, nb, xs, s);
    if (!rc) {
        k_dipole_forces<<<grid_for(n * 32, 128, 152 * 128), 128, 0, s>>>(
            pos, dip, n, b3, inv3, periodic_z, r_cut * r_cut, prefactor, cb.lin, cb.counts, cb.starts, xs, nb, ncell[0],
            ncell[1], ncell[2], forces, pe);
        count_launch();
        if (cudaGetLastError() != cudaSuccess) rc = MPS_CUDA_ERR;
    }
    cudaFreeAsync(cell3, s);
    cudaFreeAsync(bins, s);
    cudaFreeAsync(xs, s);
    return rc;
}
