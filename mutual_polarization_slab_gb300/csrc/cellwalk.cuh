// Warp walks over the 27 cells around a point, shared by the pair-list, probe and
// point-dipole force kernels.
#pragma once

#include "cells.cuh"

namespace mps {

// Neighbour cell o (0..26) of cell c: offsets (o / 9 - 1, o / 3 % 3 - 1, o % 3 - 1), the x offset
// outermost as in the reference's loop.  Computed, not read from a __constant__ table, so the kernels
// need no per-device upload and give the same offsets on every GPU of the process.
__device__ __forceinline__ int32_t nb_cell(int32_t c, int o, int64_t ncx, int64_t ncy, int64_t ncz) {
    int64_t cx = c % ncx, cy = (c / ncx) % ncy, cz = c / (ncx * ncy);
    cx = wrap_index(cx + (o / 9 - 1), ncx);
    cy = wrap_index(cy + ((o / 3) % 3 - 1), ncy);
    cz = wrap_index(cz + (o % 3 - 1), ncz);
    return (int32_t)(cx + ncx * (cy + ncy * cz));
}

// Warp-per-particle walk over the candidates of the 27 neighbour cells in (cell
// offset, position in the cell) order.  Lane o < 27 holds neighbour cell o's first
// sorted position and the exclusive prefix of the cell counts; candidate j is
// located by a binary search over those lanes.  One warp per particle keeps the
// dependent loads (particle, cells, candidates) to a few per particle instead of a
// few per (particle, cell).
struct CellWalk {
    int64_t cstart;   // lane o < 27: sorted position of neighbour cell o's first particle
    int pre;          // lane o < 27: candidates in cells 0..o-1
    int total;        // candidates of all 27 cells (warp-uniform)
};

__device__ __forceinline__ CellWalk cell_walk(int32_t c, int lane, const int32_t *__restrict__ counts,
                                              const int64_t *__restrict__ starts, int64_t ncx, int64_t ncy,
                                              int64_t ncz) {
    CellWalk cw;
    cw.cstart = 0;
    int cnt = 0;
    if (lane < 27) {
        const int32_t nb = nb_cell(c, lane, ncx, ncy, ncz);
        cw.cstart = starts[nb];
        cnt = counts[nb];
    }
    int v = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += u;
    }
    cw.pre = v - cnt;
    cw.total = __shfl_sync(0xffffffffu, v, 31);
    return cw;
}

// Cell offset o and sorted position of candidate j (0 <= j < total); all lanes call it.
__device__ __forceinline__ void walk_at(const CellWalk &cw, int j, int &o, int64_t &pos) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const int mid = lo + step;
        const int p = __shfl_sync(0xffffffffu, cw.pre, mid < 27 ? mid : 26);
        if (mid < 27 && p <= j) lo = mid;
    }
    o = lo;
    pos = __shfl_sync(0xffffffffu, cw.cstart, lo) + (j - __shfl_sync(0xffffffffu, cw.pre, lo));
}

// Float32 screen of a walk's candidates.  GB300 issues float64 at a sixty-fourth of its float32 rate and only one
// candidate in six or seven of the 27 cells lies inside the cutoff, so candidates are sorted out in float32 and the
// float64 pair terms run on the rest.  The screen never drops a pair whose float64 separation is inside the cutoff:
// each coordinate difference is shrunk by a bound of its float32 rounding (positions wrapped into the box along the
// periodic axes, so that bound is a constant there; 2^-22 (|a| + |b|) elsewhere), and the minimum image of a
// difference is never longer than the image the pair terms take.  A NaN passes, and the pair terms see it.
struct NearBox {
    float L[3], half[3];   // 0 and infinity: no minimum image along this axis
    float err[3];          // rounding bound of a wrapped difference
    float rc2;             // squared cutoff, rounded up
};

inline NearBox make_near_box(const double *box, double rc, const bool *periodic) {
    NearBox nb;
    for (int k = 0; k < 3; ++k) {
        nb.L[k] = periodic[k] ? (float)box[k] : 0.f;
        nb.half[k] = periodic[k] ? 0.5f * (float)box[k] : INFINITY;
        nb.err[k] = periodic[k] ? (float)(box[k] * 9.5367431640625e-07) : 0.f;   // 2^-20 L: 8 half-ulps of L
    }
    nb.rc2 = (float)(rc * rc * (1.0 + 1e-5));
    return nb;
}

// Float32 position of a point for the screen (periodic axes wrapped into the box); w = id.
__device__ __forceinline__ float4 near_position(const double *__restrict__ x, int64_t i, const Box3 &box,
                                                const NearBox &nb) {
    float v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double u = x[3 * i + k];
        // beyond 1e9 box lengths the wrapped value is not accurate enough for the screen: NaN, always kept
        const double w = fabs(u) < 1e9 * box.L[k] ? u - box.L[k] * floor(u / box.L[k]) : (double)NAN;
        v[k] = (float)(nb.L[k] != 0.f ? w : u);
    }
    return make_float4(v[0], v[1], v[2], __int_as_float((int)i));
}

// xs[k] = near_position of point sorted[k].
int near_positions(const double *x, const int32_t *sorted, int64_t n, const Box3 &box, const NearBox &nb, float4 *xs,
                   cudaStream_t s);

__device__ __forceinline__ bool near_screen(const float4 &a, const float4 &b, const NearBox &nb) {
    const float pa[3] = {a.x, a.y, a.z}, pb[3] = {b.x, b.y, b.z};
    float s2 = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float v = fabsf(pa[k] - pb[k]);
        if (v > nb.half[k]) v = fabsf(v - nb.L[k]);
        const float e = nb.L[k] != 0.f ? nb.err[k] : 2.4e-7f * (fabsf(pa[k]) + fabsf(pb[k]));
        v = fmaxf(v - e, 0.f);   // a NaN difference becomes 0: kept
        s2 = fmaf(v, v, s2);
    }
    return !(s2 > nb.rc2);
}

constexpr int kNearQueue = 96;   // ids a warp's queue holds: fewer than 32 waiting, 64 candidates a round

// Walks the candidates of cw in order, queues the ids (other than skip) that pass the screen against point pa in
// the warp's shared-memory queue q, and calls drain(id) for 32 of them at a time, one per lane, so that the float64
// pair terms run on full warps.  The lane of a pair depends on the particles alone: sums over lanes keep one order.
template <class F>
__device__ __forceinline__ void near_walk(const CellWalk &cw, int lane, const float4 *__restrict__ xs,
                                          const float4 &pa, int32_t skip, const NearBox &nb, int32_t *q, F &&drain) {
    int qn = 0;
    for (int j0 = 0; j0 < cw.total; j0 += 64) {
        float4 c[2];
        // both candidates of a lane are loaded before either is tested: their latencies overlap
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = j0 + 32 * h + lane;
            int o;
            int64_t pos;
            walk_at(cw, j < cw.total ? j : cw.total - 1, o, pos);
            c[h] = xs[pos];
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int32_t id = __float_as_int(c[h].w);
            const bool keep = j0 + 32 * h + lane < cw.total && id != skip && near_screen(pa, c[h], nb);
            const unsigned mask = __ballot_sync(0xffffffffu, keep);
            if (keep) q[qn + __popc(mask & ((1u << lane) - 1u))] = id;
            qn += __popc(mask);
        }
        __syncwarp();
        int done = 0;
        for (; qn - done >= 32; done += 32) drain(q[done + lane]);
        if (done) {
            const int rest = qn - done;
            const int32_t v = lane < rest ? q[done + lane] : 0;
            __syncwarp();
            if (lane < rest) q[lane] = v;
            qn = rest;
        }
        __syncwarp();
    }
    if (lane < qn) drain(q[lane]);
    __syncwarp();
}

}  // namespace mps
