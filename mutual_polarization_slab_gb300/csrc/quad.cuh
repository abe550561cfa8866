#pragma once

#include "grid.cuh"
#include "tiles.cuh"

namespace mps {

template <typename T>
int spread_gen(const double *m, int64_t n, int nrhs, int ncomp, const int32_t *start, const T *w,
               const GridParams &gp, T *grid, cudaStream_t s);
template <typename T>
int contract_gen(const T *grid, int64_t n, int nrhs, int ncomp, const int32_t *start, const T *w,
                 const GridParams &gp, double *out, cudaStream_t s);
// The same for the eight float32 grids of each vector with the home bins (tile_bins_home).
bool contract_home8_pays(const GridParams &gp, int64_t n);
int contract_home8(const float *grid, int64_t n, int nrhs, const int32_t *start, const float *w, const GridParams &gp,
                   const TileBins &tb, double *out, cudaStream_t s);
int quad_diag(const double *lam, int64_t total, const double *gq2, double *diag, cudaStream_t s);
// c64: half spectrum x 4, c32 (optional): half spectrum x 8 (the same and the unit wave vector).
int quad_kcoef(const GridParams &gp, double *c64, float *c32, cudaStream_t s);
// factor: a power of two that the scale takes on (1/2 for spectra of twice the transform).
template <typename T>
int scale_quad(void *spec, int nrhs, const GridParams &gp, const T *coef, cudaStream_t s, double factor = 1.0);
int quad_pair_coefs(const double *dist, int64_t np, const double *perp, const double *para, const double *qt,
                    const double *rv, int64_t ntab, double *c64, float *c32, int *err, cudaStream_t s);
// m32: scratch of 8 n nrhs floats (T = float only).
template <typename T>
int real_space_quad(const double *m, float *m32, double *out, int64_t n, int nrhs, const int64_t *row_ptr, int64_t np,
                    const int32_t *nbr, const T *rx, const T *ry, const T *rz, const T *coef, const double *diagS,
                    const double *diagQ, const int32_t *diag_of_rhs, cudaStream_t s);

}  // namespace mps
