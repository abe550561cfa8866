#pragma once

#include "cells.cuh"
#include "grid.cuh"
#include "tiles.cuh"

namespace mps {

int cs_pair_coefs(const int64_t *row_ptr, const int32_t *nbr, const double *dist, int64_t n, int64_t np,
                  const double *radius, const int32_t *cls, int64_t M, const double *tab, const double *rv,
                  int64_t ntab, double xi, PairData<double> p64, PairData<float> p32, int *err, cudaStream_t s);
int cs_diag(const double *lam, int64_t n, int64_t nsets, const double *radius, const int32_t *cls, int64_t M,
            const double *tab, int64_t ntab, double xi, double *diag, cudaStream_t s);
int cs_geometry(const double *x, int64_t n, const GridParams &gp, const double *radius, double xi, double eta,
                int32_t *start, double *base, double *g64, float *g32, cudaStream_t s);
int cs_green(const GridParams &gp, double eta, double xi, double *c64, float *c32, cudaStream_t s);
template <typename T>
int spread_cs(const double *m, int64_t n, int nrhs, const int32_t *start, const double *base, const T *g,
              const GridParams &gp, T *grid, cudaStream_t s);
template <typename T>
int scale_cs(void *spec, int nrhs, const GridParams &gp, const T *coef, cudaStream_t s, double factor = 1.0);
template <typename T>
int contract_cs(const T *grid, int64_t n, int nrhs, const int32_t *start, const double *base, const T *g,
                const GridParams &gp, double *out, cudaStream_t s);
// The float32 spread and contraction of many vectors (scratch of cs_many_floats, 16-byte aligned; tb from
// cs_bins_build), each where it is the faster one.
bool cs_many_spread(const GridParams &gp, int64_t n, int nrhs);
bool cs_many_contract(const GridParams &gp, int64_t n, int nrhs);
size_t cs_many_floats(int nrhs, int64_t G);
int cs_bins_build(const int32_t *start, int64_t n, const GridParams &gp, TileBins &tb, cudaStream_t s);
int spread_cs_many(const double *m, int64_t n, int nrhs, const int32_t *start, const double *base, const float *g,
                   const GridParams &gp, const TileBins &tb, float *scratch, float *grid, cudaStream_t s);
int contract_cs_many(const float *grid, int64_t n, int nrhs, const int32_t *start, const double *base, const float *g,
                     const GridParams &gp, float *scratch, double *out, cudaStream_t s);

}  // namespace mps
