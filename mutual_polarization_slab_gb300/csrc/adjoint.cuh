#pragma once

#include "cells.cuh"
#include "grid.cuh"

namespace mps {

// slopes: scratch of ntab entries; order: visiting order of the particles or null.
template <typename T>
int rs_force(const double *m, int64_t n, const int64_t *row_ptr, const PairData<T> &pd, const double *perp,
             const double *para, const double *rv, int64_t ntab, double2 *slopes, const int32_t *order, double *F,
             int *err, cudaStream_t s);
// Adds the wave-space part to F; g: scratch of 3 n P values.
int wave_force(const double *phi, const double *x, const double *m, int64_t n, const int32_t *start, const double *w,
               double *g, const GridParams &gp, double *F, cudaStream_t s);
int eps_grad(const double *m, const double *diag, double self, int64_t n, double *dE, cudaStream_t s);

}  // namespace mps
