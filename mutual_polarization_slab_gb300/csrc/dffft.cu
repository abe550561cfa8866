// Double-float 3-D real FFT pipeline (see dffft.cuh).
//
// Arithmetic: a value is hi + lo (two floats).  Sums use the two-sum error-free
// transformation, products the FMA-based two-product; every step is written
// with __fadd_rn/__fmul_rn/__fmaf_rn so the compiler cannot contract or reorder
// it.  A complex value is a float4 (re.hi, re.lo, im.hi, im.lo).
//
// Transforms: a block holds a few 1-D lines in shared memory and runs a mixed-radix (2 .. 8) Stockham FFT on all of
// them (stage s reads in[j + r N/R], multiplies by the twiddle w^(r (j mod Ns)) of the Ns R-point DFT and writes
// out[(j / Ns) Ns R + j mod Ns + r Ns]; the output is in natural order); the butterflies of all lines are numbered
// through and dealt to the threads, so no lane idles for a line length that is no multiple of 32.  A line's points lie
// with one element of padding to every 128 bytes: the first stage's stores, R apart, would otherwise share a bank.
// Inverse transforms are the forward ones with the output read backwards.
//   x pass   two real rows form one complex line; the half spectra are separated as Z[k] + conj Z[N-k] and
//            -i (Z[k] - conj Z[N-k]), twice the rows' (the scale holds the factor 1/2)
//   y pass   tiles of consecutive kx columns, coalesced along kx
//   z pass   forward FFT, the dipole Green's scale k (k . f) H / |k|^2 and the inverse FFT in one kernel; as the scale
//            is of rank one, x and y enter only as kx fx + ky fy: two transforms each way instead of three
// The float32 issue rate bounds it (some 220 instructions a point and transform in double-float).  Against one warp to
// a line, radices up to 5, three z transforms and the six-entry scale tensor, three vectors on 192^3: x 0.52 and 0.46
// -> 0.39 and 0.45 ms, y 0.61 -> 0.38, z 1.29 -> 0.61 (with the x and y passes twice 3.49 -> 2.20); one vector on 240^3
// 2.17 -> 1.65 ms, on 60 x 72 x 160 156 -> 102 us.
#include <math.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "dffft.cuh"

namespace mps {

#define MPS_TRY_STATUS(expr)          \
    do {                              \
        int _r = (expr);              \
        if (_r != MPS_OK) return _r;  \
    } while (0)

struct dfr {
    float hi, lo;
};
struct dfc {
    dfr re, im;
};

__device__ __forceinline__ dfr fts(float a, float b) {
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
// Sums and products inside a butterfly leave their result unnormalised: (s, e)
// with s the rounded leading sum (product) and e its exact rounding error plus
// the companion terms, |e| a few ulp of s.  The two-sum and the FMA residual are
// exact for any leading parts, so an unnormalised operand costs at most a couple
// of bits of the ~2^-48 accuracy; values are normalised once when a stage stores
// them (st4), not after every operation.
__device__ __forceinline__ dfr dadd(dfr a, dfr b) {
    const float s = __fadd_rn(a.hi, b.hi);
    const float bb = __fsub_rn(s, a.hi);
    float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
    e = __fadd_rn(e, __fadd_rn(a.lo, b.lo));
    return {s, e};
}
__device__ __forceinline__ dfr dneg(dfr a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ dfr dsub(dfr a, dfr b) { return dadd(a, dneg(b)); }
__device__ __forceinline__ dfr dmul(dfr a, dfr b) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    return {p, e};
}
__device__ __forceinline__ dfr dnorm(dfr a) { return fts(a.hi, a.lo); }
__device__ __forceinline__ dfr dhalf(dfr a) { return {__fmul_rn(a.hi, 0.5f), __fmul_rn(a.lo, 0.5f)}; }
__device__ __forceinline__ dfr dfrom(double v) {
    const float h = __double2float_rn(v);
    return {h, __double2float_rn(v - (double)h)};
}
// A constant split at compile time (no conversions at run time).
__host__ __device__ constexpr dfr dfk(double c) { return {(float)c, (float)(c - (double)(float)c)}; }

__device__ __forceinline__ dfc cadd(dfc a, dfc b) { return {dadd(a.re, b.re), dadd(a.im, b.im)}; }
__device__ __forceinline__ dfc csub(dfc a, dfc b) { return {dsub(a.re, b.re), dsub(a.im, b.im)}; }
__device__ __forceinline__ dfc cmul(dfc a, dfc w) {
    return {dsub(dmul(a.re, w.re), dmul(a.im, w.im)), dadd(dmul(a.re, w.im), dmul(a.im, w.re))};
}
__device__ __forceinline__ dfc cscale(dfc a, dfr c) { return {dmul(a.re, c), dmul(a.im, c)}; }
__device__ __forceinline__ dfc chalf(dfc a) { return {dhalf(a.re), dhalf(a.im)}; }
__device__ __forceinline__ dfc mul_i(dfc a) { return {dneg(a.im), a.re}; }
__device__ __forceinline__ dfc mul_mi(dfc a) { return {a.im, dneg(a.re)}; }
__device__ __forceinline__ dfc cconj(dfc a) { return {a.re, dneg(a.im)}; }
__device__ __forceinline__ dfc ld4(float4 v) { return {{v.x, v.y}, {v.z, v.w}}; }
__device__ __forceinline__ float4 st4(dfc a) {
    const dfr r = dnorm(a.re), i = dnorm(a.im);
    return make_float4(r.hi, r.lo, i.hi, i.lo);
}
__device__ __forceinline__ dfc czero() { return {{0.f, 0.f}, {0.f, 0.f}}; }

// Arithmetic policies: the storage type S of a complex value in memory and its
// register form V, with the operations the transforms use.
struct ArithDF {
    using S = float4;
    using V = dfc;
    __device__ static __forceinline__ V ld(S v) { return ld4(v); }
    __device__ static __forceinline__ S st(V v) { return st4(v); }
    __device__ static __forceinline__ V tw(float4 t) { return ld4(t); }
    __device__ static __forceinline__ V add(V a, V b) { return cadd(a, b); }
    __device__ static __forceinline__ V sub(V a, V b) { return csub(a, b); }
    __device__ static __forceinline__ V mul(V a, V b) { return cmul(a, b); }
    __device__ static __forceinline__ V scl(V a, dfr c) { return cscale(a, c); }
    // times exp(-i pi / 4), times exp(-3 i pi / 4)
    __device__ static __forceinline__ V w8(V a) {
        constexpr dfr c = dfk(0.70710678118654752440084436210485);
        return {dmul(dadd(a.re, a.im), c), dmul(dsub(a.im, a.re), c)};
    }
    __device__ static __forceinline__ V w83(V a) {
        constexpr dfr c = dfk(0.70710678118654752440084436210485);
        return {dmul(dsub(a.im, a.re), c), dneg(dmul(dadd(a.re, a.im), c))};
    }
    __device__ static __forceinline__ V half(V a) { return chalf(a); }
    __device__ static __forceinline__ V pi(V a) { return mul_i(a); }
    __device__ static __forceinline__ V mi(V a) { return mul_mi(a); }
    __device__ static __forceinline__ V conj(V a) { return cconj(a); }
    __device__ static __forceinline__ V zero() { return czero(); }
    __device__ static __forceinline__ V zero_im(V a) { return {a.re, {0.f, 0.f}}; }
    // real factors: an integer frequency times the wave-number step, products, the scale's table entry
    using R = dfr;
    using Coef = float2;
    static constexpr int kPad = 3;   // one element of padding to every 2^kPad
    __device__ static __forceinline__ R freq(int m, float hi, float lo) {
        const float f = (float)m, p = __fmul_rn(f, hi);
        return {p, __fmaf_rn(f, lo, __fmaf_rn(f, hi, -p))};
    }
    __device__ static __forceinline__ R rmul(R a, R b) { return dmul(a, b); }
    __device__ static __forceinline__ V mulr(V a, R c) { return cscale(a, c); }
    __device__ static __forceinline__ R coef(Coef h, R, R, R) { return {h.x, h.y}; }
};

struct ArithF32 {
    using S = float2;
    using V = float2;
    __device__ static __forceinline__ V ld(S v) { return v; }
    __device__ static __forceinline__ S st(V v) { return v; }
    __device__ static __forceinline__ V tw(float4 t) { return make_float2(t.x, t.z); }
    __device__ static __forceinline__ V add(V a, V b) { return make_float2(a.x + b.x, a.y + b.y); }
    __device__ static __forceinline__ V sub(V a, V b) { return make_float2(a.x - b.x, a.y - b.y); }
    __device__ static __forceinline__ V mul(V a, V b) {
        return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
    }
    __device__ static __forceinline__ V scl(V a, dfr c) { return make_float2(a.x * c.hi, a.y * c.hi); }
    __device__ static __forceinline__ V w8(V a) {
        const float c = 0.70710678f;
        return make_float2(c * (a.x + a.y), c * (a.y - a.x));
    }
    __device__ static __forceinline__ V w83(V a) {
        const float c = 0.70710678f;
        return make_float2(c * (a.y - a.x), -c * (a.x + a.y));
    }
    __device__ static __forceinline__ V half(V a) { return make_float2(0.5f * a.x, 0.5f * a.y); }
    __device__ static __forceinline__ V pi(V a) { return make_float2(-a.y, a.x); }
    __device__ static __forceinline__ V mi(V a) { return make_float2(a.y, -a.x); }
    __device__ static __forceinline__ V conj(V a) { return make_float2(a.x, -a.y); }
    __device__ static __forceinline__ V zero() { return make_float2(0.f, 0.f); }
    __device__ static __forceinline__ V zero_im(V a) { return make_float2(a.x, 0.f); }
    using R = float;
    using Coef = float;
    static constexpr int kPad = 4;
    __device__ static __forceinline__ R freq(int m, float hi, float) { return (float)m * hi; }
    __device__ static __forceinline__ R rmul(R a, R b) { return a * b; }
    __device__ static __forceinline__ V mulr(V a, R c) { return make_float2(a.x * c, a.y * c); }
    // H of the component form: 0.5 H / |k|^2
    __device__ static __forceinline__ R coef(Coef h, R x, R y, R z) {
        const float k2 = x * x + y * y + z * z;
        return k2 > 0.f ? 0.5f * h / k2 : 0.f;
    }
};

// Small DFTs, forward sign (w = exp(-2 pi i / R)).
template <class A, int R>
struct Dft;

template <class A>
struct Dft<A, 2> {
    __device__ static __forceinline__ void run(typename A::V *v) {
        const auto a = v[0], b = v[1];
        v[0] = A::add(a, b);
        v[1] = A::sub(a, b);
    }
};

template <class A>
struct Dft<A, 3> {
    __device__ static __forceinline__ void run(typename A::V *v) {
        const auto a = A::add(v[1], v[2]), b = A::sub(v[1], v[2]);
        const auto m = A::sub(v[0], A::half(a));
        constexpr dfr c = dfk(0.86602540378443864676372317075294);   // sqrt(3) / 2
        const auto tb = A::scl(b, c);
        v[0] = A::add(v[0], a);
        v[1] = A::add(m, A::mi(tb));
        v[2] = A::add(m, A::pi(tb));
    }
};

template <class A>
__device__ __forceinline__ void dft4(typename A::V &v0, typename A::V &v1, typename A::V &v2, typename A::V &v3) {
    const auto a = A::add(v0, v2), b = A::sub(v0, v2), c = A::add(v1, v3), d = A::sub(v1, v3);
    v0 = A::add(a, c);
    v2 = A::sub(a, c);
    v1 = A::add(b, A::mi(d));
    v3 = A::add(b, A::pi(d));
}

template <class A>
struct Dft<A, 4> {
    __device__ static __forceinline__ void run(typename A::V *v) { dft4<A>(v[0], v[1], v[2], v[3]); }
};

template <class A>
struct Dft<A, 8> {
    __device__ static __forceinline__ void run(typename A::V *v) {
        dft4<A>(v[0], v[2], v[4], v[6]);
        dft4<A>(v[1], v[3], v[5], v[7]);
        const auto o1 = A::w8(v[3]), o2 = A::mi(v[5]), o3 = A::w83(v[7]);
        const auto e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
        v[0] = A::add(e0, o0);
        v[4] = A::sub(e0, o0);
        v[1] = A::add(e1, o1);
        v[5] = A::sub(e1, o1);
        v[2] = A::add(e2, o2);
        v[6] = A::sub(e2, o2);
        v[3] = A::add(e3, o3);
        v[7] = A::sub(e3, o3);
    }
};

// 3 x 2 without twiddles (Good's index maps): input (2 a + 3 b) mod 6, output (4 a + 3 b) mod 6.
template <class A>
struct Dft<A, 6> {
    __device__ static __forceinline__ void run(typename A::V *v) {
        typename A::V e[3] = {v[0], v[2], v[4]}, o[3] = {v[3], v[5], v[1]};
        Dft<A, 3>::run(e);
        Dft<A, 3>::run(o);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v[4 * k % 6] = A::add(e[k], o[k]);
            v[(4 * k + 3) % 6] = A::sub(e[k], o[k]);
        }
    }
};

template <class A>
struct Dft<A, 5> {
    __device__ static __forceinline__ void run(typename A::V *v) {
        constexpr dfr c1 = dfk(0.30901699437494742410229341718282), c2 = dfk(-0.80901699437494742410229341718282);
        constexpr dfr s1 = dfk(0.95105651629515357211643933337938), s2 = dfk(0.58778525229247312916870595463907);
        const auto a1 = A::add(v[1], v[4]), b1 = A::sub(v[1], v[4]), a2 = A::add(v[2], v[3]),
                   b2 = A::sub(v[2], v[3]);
        const auto m1 = A::add(v[0], A::add(A::scl(a1, c1), A::scl(a2, c2)));
        const auto m2 = A::add(v[0], A::add(A::scl(a1, c2), A::scl(a2, c1)));
        const auto t1 = A::add(A::scl(b1, s1), A::scl(b2, s2));
        const auto t2 = A::sub(A::scl(b1, s2), A::scl(b2, s1));
        v[0] = A::add(v[0], A::add(a1, a2));
        v[1] = A::add(m1, A::mi(t1));
        v[2] = A::add(m2, A::mi(t2));
        v[3] = A::add(m2, A::pi(t2));
        v[4] = A::add(m1, A::pi(t1));
    }
};

// ---------------------------------------------------------------------------
// Stages on the nl lines of a block (p.N points each, line stride ld)
// ---------------------------------------------------------------------------
// Six blocks an SM (80 registers, 36 KB of shared memory each), the sums over both passes in x and y and the z pass: on
// 192^3, 240^3, 60 x 72 x 160 2.26 ms, 1.65 ms, 105 us; five blocks of 44 KB 2.36, 1.64, 103; eight of 27 KB 2.24,
// 1.91, 97 (32-byte rows in z); four of 54 KB with radices 10 and 12 2.52, 1.95, 124; six of 36 KB with them 2.31,
// 1.85, 112.
constexpr int kDfThreads = 128, kDfBlocks = 6;
constexpr size_t kDfSmem = 36 * 1024;

// Position of point i of a line.
template <class A>
__host__ __device__ __forceinline__ unsigned at(unsigned i) {
    return i + (i >> A::kPad);
}
// x / d for x < 2^16 by the multiplier ceil(2^32 / d) (0 stands for d = 1).
__device__ __forceinline__ unsigned div16(unsigned x, unsigned mul) { return mul ? __umulhi(x, mul) : x; }

template <class A, int R>
__device__ __forceinline__ void df_stage(const typename A::S *in, typename A::S *out, int nl, int ld, const DfAxisPlan &p,
                                         const float4 *tws, int s) {
    const unsigned NR = p.N / R, Ns = p.Ns[s];
    const float4 *tw = tws + p.twoff[s];
    for (unsigned w = threadIdx.x; w < nl * NR; w += kDfThreads) {
        const unsigned line = div16(w, p.mNR[s]), j = w - line * NR, jq = div16(j, p.mNs[s]), jm = j - jq * Ns;
        const typename A::S *a = in + line * ld;
        typename A::V v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = A::ld(a[at<A>(j + r * NR)]);
        if (Ns > 1) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = A::mul(v[r], A::tw(tw[(r - 1) * Ns + jm]));
        }
        Dft<A, R>::run(v);
        typename A::S *o = out + line * ld;
        const unsigned d = jq * Ns * R + jm;
#pragma unroll
        for (int r = 0; r < R; ++r) o[at<A>(d + r * Ns)] = A::st(v[r]);
    }
}

// Forward transform of the nl lines in a (b: scratch of the same size); returns the buffer with the result.  All
// threads of the block call it; the lines are complete in a, and the result is complete on return.
template <class A>
__device__ typename A::S *fft_lines(typename A::S *a, typename A::S *b, int nl, int ld, const DfAxisPlan &p,
                                    const float4 *tws) {
    for (int s = 0; s < p.nst; ++s) {
        switch (p.R[s]) {
            case 2: df_stage<A, 2>(a, b, nl, ld, p, tws, s); break;
            case 3: df_stage<A, 3>(a, b, nl, ld, p, tws, s); break;
            case 4: df_stage<A, 4>(a, b, nl, ld, p, tws, s); break;
            case 5: df_stage<A, 5>(a, b, nl, ld, p, tws, s); break;
            case 6: df_stage<A, 6>(a, b, nl, ld, p, tws, s); break;
            default: df_stage<A, 8>(a, b, nl, ld, p, tws, s); break;
        }
        __syncthreads();
        typename A::S *x = a;
        a = b;
        b = x;
    }
    return a;
}

// The twiddles go to the front of shared memory, the lines behind them.  (From global memory they missed L1, which the
// lines' shared memory leaves small: with them and the lines' loads waited for one by one, the y pass on 192^3 took
// 0.58 ms for three vectors.)
template <class A>
__device__ __forceinline__ typename A::S *lines_after_twiddles(float4 *sm, const DfAxisPlan &p) {
    for (int i = threadIdx.x; i < p.ntw; i += kDfThreads) copy_async(sm + i, p.tw + i);
    return reinterpret_cast<typename A::S *>(sm + p.ntw);
}

// ---------------------------------------------------------------------------
// x pass (Rl: real type of the grids): two rows of Nx of a grid are one line (npairs lines over all the stacked grids)
// ---------------------------------------------------------------------------
template <class A, typename Rl>
__global__ void __launch_bounds__(kDfThreads, kDfBlocks)
    k_fft_x_fwd(const Rl *__restrict__ grid, typename A::S *__restrict__ spec,
                int64_t npairs, RowPairs rp, DfAxisPlan px, int L, int ld) {
    extern __shared__ float4 sm[];
    typename A::S *buf = lines_after_twiddles<A>(sm, px);
    const int Nx = px.N, Nxh = Nx / 2 + 1;
    const int64_t ntiles = (npairs + L - 1) / L;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t p0 = tile * L;
        const int nl = (int)min((int64_t)L, npairs - p0);
        const RowPairs::Lines ln = rp.from(p0);
        const Rl *rows = grid + ln.row0 * Nx;
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nx); i += kDfThreads) {
            const unsigned line = div16(i, px.mN), n = i - line * Nx;
            Rl *d = reinterpret_cast<Rl *>(buf + line * ld + at<A>(n));   // (re, im)
            bool two;
            const Rl *row = rows + (int64_t)ln.row(line, &two) * Nx + n;
            copy_async(d, row);
            if (two)
                copy_async(d + 1, row + Nx);
            else
                d[1] = Rl{};
        }
        copy_async_wait();
        __syncthreads();
        const typename A::S *Z = fft_lines<A>(buf, buf + L * ld, nl, ld, px, sm);
        typename A::S *out = spec + ln.row0 * Nxh;
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nxh); i += kDfThreads) {
            const unsigned line = div16(i, px.mNh), k = i - line * Nxh;
            const auto zk = A::ld(Z[line * ld + at<A>(k)]), zc = A::conj(A::ld(Z[line * ld + at<A>(k ? Nx - k : 0)]));
            bool two;
            typename A::S *o = out + (int64_t)ln.row(line, &two) * Nxh + k;
            o[0] = A::st(A::add(zk, zc));
            if (two) o[Nxh] = A::st(A::mi(A::sub(zk, zc)));
        }
        __syncthreads();
    }
}

template <class A, typename Rl>
__global__ void __launch_bounds__(kDfThreads, kDfBlocks)
    k_fft_x_inv(const typename A::S *__restrict__ spec, Rl *__restrict__ grid,
                int64_t npairs, RowPairs rp, DfAxisPlan px, int L, int ld) {
    extern __shared__ float4 sm[];
    typename A::S *buf = lines_after_twiddles<A>(sm, px);
    const int Nx = px.N, Nxh = Nx / 2 + 1;
    const int64_t ntiles = (npairs + L - 1) / L;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t p0 = tile * L;
        const int nl = (int)min((int64_t)L, npairs - p0);
        const RowPairs::Lines ln = rp.from(p0);
        const typename A::S *in = spec + ln.row0 * Nxh;
        // X0 + i X1 at k and, from the Hermitian halves, at N - k; the real bins' imaginary parts are dropped
#pragma unroll 4
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nxh); i += kDfThreads) {
            const unsigned line = div16(i, px.mNh), k = i - line * Nxh;
            bool two;
            const typename A::S *row = in + (int64_t)ln.row(line, &two) * Nxh + k;
            auto x0 = A::ld(row[0]), x1 = two ? A::ld(row[Nxh]) : A::zero();
            const bool real_bin = k == 0 || 2 * k == (unsigned)Nx;
            if (real_bin) {
                x0 = A::zero_im(x0);
                x1 = A::zero_im(x1);
            }
            buf[line * ld + at<A>(k)] = A::st(A::add(x0, A::pi(x1)));
            if (!real_bin) buf[line * ld + at<A>(Nx - k)] = A::st(A::conj(A::add(x0, A::mi(x1))));
        }
        copy_async_wait();
        __syncthreads();
        const typename A::S *Z = fft_lines<A>(buf, buf + L * ld, nl, ld, px, sm);
        Rl *rows = grid + ln.row0 * Nx;
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nx); i += kDfThreads) {
            const unsigned line = div16(i, px.mN), n = i - line * Nx;
            const Rl *z = reinterpret_cast<const Rl *>(Z + line * ld + at<A>(n ? Nx - n : 0));
            bool two;
            Rl *row = rows + (int64_t)ln.row(line, &two) * Nx + n;
            row[0] = z[0];
            if (two) row[Nx] = z[1];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// y pass: L (a power of two) consecutive kx columns of one (component, z) plane
// ---------------------------------------------------------------------------
template <class A>
__global__ void __launch_bounds__(kDfThreads, kDfBlocks)
    k_fft_y(typename A::S *__restrict__ spec, int64_t nplanes, int Nxh,
            DfAxisPlan py, int L, int ld, int inverse) {
    extern __shared__ float4 sm[];
    typename A::S *buf = lines_after_twiddles<A>(sm, py);
    const int Ny = py.N, nblk = (Nxh + L - 1) / L;
    const unsigned t = threadIdx.x & (L - 1), y0 = threadIdx.x / L, ys = kDfThreads / L;
    for (int64_t tile = blockIdx.x; tile < nplanes * nblk; tile += gridDim.x) {
        const int64_t plane = tile / nblk;
        const int kx0 = (int)(tile % nblk) * L, nl = min(L, Nxh - kx0);
        typename A::S *base = spec + plane * Ny * (int64_t)Nxh + kx0 + t;
        if ((int)t < nl)
            for (unsigned y = y0; y < (unsigned)Ny; y += ys) copy_async(buf + t * ld + at<A>(y), base + (int64_t)y * Nxh);
        copy_async_wait();
        __syncthreads();
        const typename A::S *Z = fft_lines<A>(buf, buf + L * ld, nl, ld, py, sm);
        if ((int)t < nl)
            for (unsigned y = y0; y < (unsigned)Ny; y += ys)
                base[(int64_t)y * Nxh] = Z[t * ld + at<A>(inverse && y ? Ny - y : y)];
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// z pass with the dipole scale: L consecutive kx columns at one ky, the 3 components of one vector.
// out = k (k . f) h, the sum over the components whose axis is on its Nyquist bin apart from the others' (the real part
// of the complex pipeline's coupling).  Columns with both or neither of kx, ky on the Nyquist bin need two lines,
// a = kx fx + ky fy and b = fz:  out_x = kx t, out_y = ky t, out_z = u with t, u the inverse transforms of h (a + kz b)
// and h kz (a + kz b); where z is on the other side of the rule than x and y, of h a and h kz^2 b.  A tile that holds
// one of the few other columns takes three lines a column, fewer columns at a time.
// ---------------------------------------------------------------------------
template <class A>
__global__ void __launch_bounds__(kDfThreads, kDfBlocks)
    k_fft_z_scale(typename A::S *__restrict__ spec, int nrhs, GridParams gp,
                  DfAxisPlan pz, DfStep q, const typename A::Coef *__restrict__ h,
                  int L, int ld) {
    using V = typename A::V;
    using Rr = typename A::R;
    extern __shared__ float4 sm[];
    typename A::S *const buf = lines_after_twiddles<A>(sm, pz), *const other = buf + max(2 * L, 3) * ld;
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2], Nxh = Nx / 2 + 1, nblk = (Nxh + L - 1) / L;
    const int64_t zs = (int64_t)Ny * Nxh, Gc = zs * Nz;
    const int64_t ntiles = (int64_t)nrhs * Ny * nblk;
    const unsigned t = threadIdx.x & (L - 1), z0 = threadIdx.x / L, zstep = kDfThreads / L;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int kx0 = (int)(tile % nblk) * L, nl = min(L, Nxh - kx0);
        const int ky = (int)((tile / nblk) % Ny), r = (int)(tile / ((int64_t)nblk * Ny));
        const bool nyy = 2 * ky == Ny, has_nyx = 2 * (kx0 + nl - 1) == Nx;   // the last column may be x's Nyquist bin
        const bool two = nyy ? (nl == 1 && has_nyx) : !has_nyx;
        const int batch = two ? L : max(1, 2 * L / 3);
        const Rr qy = A::freq(fft_freq(ky, Ny), q.hi[1], q.lo[1]);
        for (int c0 = 0; c0 < nl; c0 += batch) {
            const int cols = min(batch, nl - c0), bs = cols * ld, kx = kx0 + c0 + (int)t;
            const bool mine = (int)t < cols;
            const Rr qx = A::freq(fft_freq(mine ? kx : 0, Nx), q.hi[0], q.lo[0]);
            const int64_t col = (int64_t)ky * Nxh + kx;
            typename A::S *base = spec + (int64_t)(3 * r) * Gc + col;
            if (mine && two) {
#pragma unroll 4
                for (unsigned z = z0; z < (unsigned)Nz; z += zstep) {
                    const typename A::S *f = base + z * zs, fx = f[0], fy = f[Gc];
                    typename A::S *o = buf + t * ld + at<A>(z);
                    copy_async(o + bs, f + 2 * Gc);
                    o[0] = A::st(A::add(A::mulr(A::ld(fx), qx), A::mulr(A::ld(fy), qy)));
                }
            } else if (mine) {
                for (unsigned z = z0; z < (unsigned)Nz; z += zstep)
                    for (int c = 0; c < 3; ++c) copy_async(buf + t * ld + at<A>(z) + c * bs, base + z * zs + c * Gc);
            }
            copy_async_wait();
            __syncthreads();
            // both transforms from one call: two copies of the stages overflow the instruction cache (three vectors on
            // 192^3 0.65 -> 0.61 ms)
            typename A::S *Z = buf;
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass) {
                Z = fft_lines<A>(Z, Z == buf ? other : buf, (two ? 2 : 3) * cols, ld, pz, sm);
                if (pass) break;
                if (mine) {
#pragma unroll 2
                    for (unsigned z = z0; z < (unsigned)Nz; z += zstep) {
                        const Rr qz = A::freq(fft_freq(z, Nz), q.hi[2], q.lo[2]);
                        const bool nyz = 2 * (int)z == Nz;
                        const Rr hc = A::coef(h[z * zs + col], qx, qy, qz);
                        typename A::S *o = Z + t * ld + at<A>(z);
                        if (two) {
                            const V a = A::ld(o[0]), b = A::mulr(A::ld(o[bs]), qz);
                            const bool same = nyz == nyy;   // nyy == nyx here
                            const V s = A::add(a, b);
                            o[0] = A::st(A::mulr(same ? s : a, hc));
                            o[bs] = A::st(A::mulr(same ? s : b, A::rmul(hc, qz)));
                        } else {
                            const bool ny[3] = {2 * kx == Nx, nyy, nyz};
                            const Rr qc[3] = {qx, qy, qz};
                            V s0 = A::zero(), s1 = A::zero();   // off and on the Nyquist bins
#pragma unroll
                            for (int c = 0; c < 3; ++c) {
                                const V v = A::mulr(A::ld(o[c * bs]), qc[c]);
                                if (ny[c])
                                    s1 = A::add(s1, v);
                                else
                                    s0 = A::add(s0, v);
                            }
#pragma unroll
                            for (int c = 0; c < 3; ++c)
                                o[c * bs] = A::st(A::mulr(ny[c] ? s1 : s0, A::rmul(hc, qc[c])));
                        }
                    }
                }
                __syncthreads();
            }
            if (mine)
                for (unsigned z = z0; z < (unsigned)Nz; z += zstep) {
                    typename A::S *f = base + z * zs;
                    const typename A::S *o = Z + t * ld + at<A>(z ? Nz - z : 0);
                    if (two) {
                        const V v = A::ld(o[0]);
                        f[0] = A::st(A::mulr(v, qx));
                        f[Gc] = A::st(A::mulr(v, qy));
                        f[2 * Gc] = o[bs];
                    } else {
                        f[0] = o[0];
                        f[Gc] = o[bs];
                        f[2 * Gc] = o[2 * bs];
                    }
                }
            __syncthreads();
        }
    }
}

// 0.5 H / |k|^2 per half-spectrum point as a double-float number, in float64 once per grid; one thread per point of the
// spectrum's quarter.
__global__ void k_df_scale(GridParams gp, const double *__restrict__ H, float2 *__restrict__ hs) {
    const HalfQuarter hq(gp.N);
    const int64_t Gq = hq.size();
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < Gq; t += (int64_t)gridDim.x * blockDim.x) {
        int kx, ky, kz;
        hq.point(t, &kx, &ky, &kz);
        const double qx = fft_freq(kx, gp.N[0]) * gp.kfac[0];
        const double qy = fft_freq(ky, gp.N[1]) * gp.kfac[1];
        const double qz = fft_freq(kz, gp.N[2]) * gp.kfac[2];
        const double k2 = qx * qx + qy * qy + qz * qz;
        const dfr d = dfrom(k2 > 0.0 ? 0.5 * H[((int64_t)kz * hq.Ny + ky) * hq.Nxh + kx] / k2 : 0.0);
        mirror_points(hq, kx, ky, kz, [&](int64_t i, int, int) { hs[i] = make_float2(d.hi, d.lo); });
    }
}

int df_scale_table(const GridParams &gp, const double *H, float2 *hs, cudaStream_t s) {
    k_df_scale<<<grid_for(HalfQuarter(gp.N).size(), 256), 256, 0, s>>>(gp, H, hs);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

// ---------------------------------------------------------------------------
// Plans
// ---------------------------------------------------------------------------
static std::map<std::pair<int, int>, DfAxisPlan> g_df_axes;   // per (device, length)
static std::mutex g_df_mu;

// Radices of a 2-3-5 length with the fewest double-float instructions a point: the butterfly, the twiddles (32 each,
// none in the first stage), the stores' normalisation and a charge for a stage's passes over shared memory.
static std::vector<int> df_radices(int n) {
    static const struct { int R; double ops; } kR[] = {{2, 32}, {3, 108}, {4, 128}, {5, 320}, {6, 312}, {8, 432}};
    std::vector<int> best, cur;
    double cost = 1e30;
    auto search = [&](auto &self, int left, double c) -> void {
        if (c >= cost) return;
        if (left == 1) {
            cost = c;
            best = cur;
            return;
        }
        for (const auto &r : kR)
            if (left % r.R == 0 && cur.size() < (size_t)kDfMaxStages) {
                const double tw = cur.empty() ? 0.0 : 32.0 * (r.R - 1);
                cur.push_back(r.R);
                self(self, left / r.R, c + (r.ops + tw + 6.0 * r.R) / r.R + 16.0);
                cur.pop_back();
            }
    };
    search(search, n, 0.0);
    return best;
}

static unsigned div16_mul(unsigned d) { return d == 1 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d); }

// MPS_OK with supported = false for a length that the transforms do not take; other status codes are failures that say
// nothing about the length.
static int df_axis(int N, int dev, DfAxisPlan *out, bool *supported) {
    *supported = false;
    if (N < 2 || N > 1024) return MPS_OK;
    std::lock_guard<std::mutex> lk(g_df_mu);
    auto it = g_df_axes.find({dev, N});
    if (it != g_df_axes.end()) {
        *out = it->second;
        *supported = true;
        return MPS_OK;
    }
    int m = N;
    for (int f : {2, 3, 5})
        while (m % f == 0) m /= f;
    if (m != 1) return MPS_OK;
    DfAxisPlan p;
    p.N = N;
    p.mN = div16_mul(N);
    p.mNh = div16_mul(N / 2 + 1);
    std::vector<float4> tw;
    int ns = 1;
    for (int R : df_radices(N)) {
        const int s = p.nst++;
        p.R[s] = R;
        p.Ns[s] = ns;
        p.mNR[s] = div16_mul(N / R);
        p.mNs[s] = div16_mul(ns);
        p.twoff[s] = (int)tw.size();
        if (ns > 1)
            for (int r = 1; r < R; ++r)
                for (int jm = 0; jm < ns; ++jm) {
                    const double ang = -2.0 * M_PI * (double)(jm * r) / (double)(ns * R);
                    const double c = cos(ang), sn = sin(ang);
                    const float ch = (float)c, sh = (float)sn;
                    tw.push_back(make_float4(ch, (float)(c - (double)ch), sh, (float)(sn - (double)sh)));
                }
        ns *= R;
    }
    if (tw.empty()) tw.push_back(make_float4(1.f, 0.f, 0.f, 0.f));
    float4 *d = nullptr;
    // before another thread can find the plan
    const int rc = upload_table(tw.data(), sizeof(float4) * tw.size(), (void **)&d);
    if (rc) return rc;
    p.tw = d;
    p.ntw = (int)tw.size();
    g_df_axes[{dev, N}] = p;
    *out = p;
    *supported = true;
    return MPS_OK;
}

int df_plan(const GridParams &gp, DfPlan3 *out) {
    out->ok = false;
    if (gp.N[0] % 2 != 0) return MPS_OK;
    int dev = 0;
    MPS_CUDA_TRY(cudaGetDevice(&dev));
    for (int d = 0; d < 3; ++d) {
        bool supported;
        const int rc = df_axis(gp.N[d], dev, &out->ax[d], &supported);
        if (rc || !supported) return rc;
    }
    out->ok = true;
    return MPS_OK;
}

// ---------------------------------------------------------------------------
// Launches
// ---------------------------------------------------------------------------
// Padded length of a line, odd (lines side by side then start in different banks).
template <class A>
static int line_stride(int N) {
    return (int)at<A>(N - 1) + 1 | 1;
}

// Lines (columns) to a block: up to 8 (whole 128-byte rows of the strided passes) within kDfSmem, fewer where the grid
// has too few lines to give every SM two blocks.
static int lines_per_block(size_t column, int64_t columns) {
    int L = 8;
    while (L > 1 && (column * L > kDfSmem || columns / L < 304)) L /= 2;
    return L;
}

// One value for every launch of a kernel (three lines of the longest axis, their scratch, its twiddles): calls from
// several threads agree.
template <class A, typename K>
static int set_smem(K kernel, size_t bytes) {
    const size_t most = sizeof(typename A::S) * 6 * (size_t)line_stride<A>(1024) + sizeof(float4) * 1024;
    if (bytes > most) return MPS_BAD_ARG;
    if (bytes > 48 * 1024)
        MPS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    return MPS_OK;
}

template <class A, typename Rl>
static int launch_x(bool fwd, const Rl *gin, Rl *gout, typename A::S *spec, int ncomp, const GridParams &gp,
                    const DfAxisPlan &px, cudaStream_t s) {
    const RowPairs rp((int64_t)gp.N[2] * gp.N[1]);
    const int64_t npairs = (int64_t)ncomp * rp.pairs;
    const int ld = line_stride<A>(px.N);
    const size_t column = sizeof(typename A::S) * 2 * (size_t)ld;
    const int L = lines_per_block(column, npairs);
    const unsigned blocks = grid_for((npairs + L - 1) / L, 1, INT32_MAX);
    const size_t smem = sizeof(float4) * px.ntw + column * L;
    if (fwd) {
        MPS_TRY_STATUS((set_smem<A>(k_fft_x_fwd<A, Rl>, smem)));
        k_fft_x_fwd<A, Rl><<<blocks, kDfThreads, smem, s>>>(gin, spec, npairs, rp, px, L, ld);
    } else {
        MPS_TRY_STATUS((set_smem<A>(k_fft_x_inv<A, Rl>, smem)));
        k_fft_x_inv<A, Rl><<<blocks, kDfThreads, smem, s>>>(spec, gout, npairs, rp, px, L, ld);
    }
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template <class A>
static int launch_y(typename A::S *spec, int ncomp, const GridParams &gp, const DfAxisPlan &py, int inverse,
                    cudaStream_t s) {
    const int64_t nplanes = (int64_t)ncomp * gp.N[2];
    const int Nxh = gp.N[0] / 2 + 1, ld = line_stride<A>(py.N);
    const size_t column = sizeof(typename A::S) * 2 * (size_t)ld;
    const int L = lines_per_block(column, nplanes * Nxh), nblk = (Nxh + L - 1) / L;
    const size_t smem = sizeof(float4) * py.ntw + column * L;
    MPS_TRY_STATUS((set_smem<A>(k_fft_y<A>, smem)));
    k_fft_y<A><<<grid_for(nplanes * nblk, 1, INT32_MAX), kDfThreads, smem, s>>>(spec, nplanes, Nxh, py, L, ld, inverse);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

template <class A>
static int launch_z_scale(typename A::S *spec, int nrhs, const GridParams &gp, const DfAxisPlan &pz,
                          const typename A::Coef *h, cudaStream_t s) {
    const int Nxh = gp.N[0] / 2 + 1, ld = line_stride<A>(gp.N[2]);
    const size_t column = sizeof(typename A::S) * 4 * (size_t)ld;
    const int L = lines_per_block(column, (int64_t)nrhs * gp.N[1] * Nxh), nblk = (Nxh + L - 1) / L;
    const size_t smem = sizeof(float4) * pz.ntw + column / 2 * std::max(2 * L, 3);   // (three lines where L = 1)
    MPS_TRY_STATUS((set_smem<A>(k_fft_z_scale<A>, smem)));
    DfStep q;
    for (int d = 0; d < 3; ++d) {
        q.hi[d] = (float)gp.kfac[d];
        q.lo[d] = (float)(gp.kfac[d] - (double)q.hi[d]);
    }
    k_fft_z_scale<A><<<grid_for((int64_t)nrhs * gp.N[1] * nblk, 1, INT32_MAX), kDfThreads, smem, s>>>(spec, nrhs, gp, pz, q,
                                                                                                     h, L, ld);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int df_forward_xy(const float2 *grid, float4 *spec, int ncomp, const GridParams &gp, const DfPlan3 &pl,
                  cudaStream_t s) {
    if (!pl.ok) return MPS_BAD_ARG;
    MPS_TRY_STATUS((launch_x<ArithDF, float2>(true, grid, nullptr, spec, ncomp, gp, pl.ax[0], s)));
    return launch_y<ArithDF>(spec, ncomp, gp, pl.ax[1], 0, s);
}

int df_inverse_yx(float4 *spec, float2 *grid, int ncomp, const GridParams &gp, const DfPlan3 &pl, cudaStream_t s) {
    if (!pl.ok) return MPS_BAD_ARG;
    MPS_TRY_STATUS(launch_y<ArithDF>(spec, ncomp, gp, pl.ax[1], 1, s));
    return launch_x<ArithDF, float2>(false, nullptr, grid, spec, ncomp, gp, pl.ax[0], s);
}

int df_z_scale_dipole(float4 *spec, int nrhs, const GridParams &gp, const DfPlan3 &pl, const float2 *hs,
                      cudaStream_t s) {
    if (!pl.ok) return MPS_BAD_ARG;
    return launch_z_scale<ArithDF>(spec, nrhs, gp, pl.ax[2], hs, s);
}

int f32_forward_xy(const float *grid, float2 *spec, int ncomp, const GridParams &gp, const DfPlan3 &pl,
                   cudaStream_t s) {
    if (!pl.ok) return MPS_BAD_ARG;
    MPS_TRY_STATUS((launch_x<ArithF32, float>(true, grid, nullptr, spec, ncomp, gp, pl.ax[0], s)));
    return launch_y<ArithF32>(spec, ncomp, gp, pl.ax[1], 0, s);
}

int f32_inverse_yx(float2 *spec, float *grid, int ncomp, const GridParams &gp, const DfPlan3 &pl, cudaStream_t s) {
    if (!pl.ok) return MPS_BAD_ARG;
    MPS_TRY_STATUS(launch_y<ArithF32>(spec, ncomp, gp, pl.ax[1], 1, s));
    return launch_x<ArithF32, float>(false, nullptr, grid, spec, ncomp, gp, pl.ax[0], s);
}

int f32_z_scale_dipole(float2 *spec, int nrhs, const GridParams &gp, const DfPlan3 &pl, const float *H,
                       cudaStream_t s) {
    if (!pl.ok) return MPS_BAD_ARG;
    return launch_z_scale<ArithF32>(spec, nrhs, gp, pl.ax[2], H, s);
}

}  // namespace mps
