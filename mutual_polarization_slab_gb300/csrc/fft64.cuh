// Float64 3-D real transforms of the dipole operator's wave-space stages (see fft64.cu).
#pragma once

#include "grid.cuh"

namespace mps {

constexpr int kF64MaxStages = 10;
constexpr int kF64MaxN = 1024;
// Largest prime factor of an axis that fft64.cu takes; a prime radix p costs p - 1 multiply-adds a point.
// Up to 127 that beats cuFFT (measured on p^3 and (2p)^3, every prime from 53: 1.02 .. 1.53 times; p = 127, one vector:
// 4.82 -> 3.75 ms); above it cuFFT transforms by convolution and keeps the axis.
constexpr int kF64MaxPrime = 127;

// Mixed-radix plan of one axis: stage s has radix R[s], Ns[s] = R[0] ... R[s-1].  tw holds each stage's twiddles
// exp(-2 pi i jm r / (Ns R)) at twoff[s] + jm R + r, and, for a prime radix above 5, its R roots at rtoff[s] or, where
// third[s] = q > 0, the permutation and coefficients of the split into thirds (stage64_thirds).
struct F64Axis {
    int N = 0, nst = 0;
    int R[kF64MaxStages], Ns[kF64MaxStages], twoff[kF64MaxStages], rtoff[kF64MaxStages], third[kF64MaxStages];
    const double2 *tw = nullptr;
};

struct F64Plan3 {
    bool ok = false;
    F64Axis ax[3];
};

// Builds (once per device and axis length) the tables of a grid's axes; ok = false where an axis is not supported.
int f64_plan(const GridParams &gp, F64Plan3 *out);

// Whether the transforms are the faster ones on a grid that they support; cuFFT keeps the others.  A pass deals the
// butterflies of at most eight lines to a block, and short lines leave it few of them.  fused: f64_z_scale_dipole,
// which saves a third of the z transforms and the scale's own pass; without it (f64_z) the axes have to be long enough
// or the grids few.
bool f64_pays(const GridParams &gp, bool fused, int ngrids);

// 0.5 H / |k|^2 on the half spectrum (H includes 1/G; zero at k = 0): the factor 1/2 belongs to f64_forward_xy.
int f64_scale_coef(const GridParams &gp, const double *H, double *hs, cudaStream_t s);

// spec = twice the x and y transforms of ncomp real grids (half spectrum, x fastest, as R2C lays it out).
int f64_forward_xy(const double *grid, void *spec, int ncomp, const GridParams &gp, const F64Plan3 &pl,
                   cudaStream_t s);
// z transform, the dipole operator's scale H k k^T / |k|^2 (Nyquist rule) and the inverse z transform.
int f64_z_scale_dipole(void *spec, int nrhs, const GridParams &gp, const F64Plan3 &pl, const double *hs,
                       cudaStream_t s);
// The z transform by itself, of ncomp spectra (forward, or inverse and unnormalised), for scales of other operators.
int f64_z(void *spec, int ncomp, const GridParams &gp, const F64Plan3 &pl, int inverse, cudaStream_t s);
int f64_inverse_yx(void *spec, double *grid, int ncomp, const GridParams &gp, const F64Plan3 &pl, cudaStream_t s);

}  // namespace mps
