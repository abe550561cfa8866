// Float64 3-D real transforms of the dipole operator.
//
// GB300 issues two float64 multiply-adds a clock on an SM, so one float64 warp instruction holds its scheduler's
// float64 pipe for some 64 cycles: everything else in these kernels (shared-memory passes, index arithmetic, twiddle
// loads) hides behind the arithmetic, and the float64 operations per point are what there is to save.
//   x pass    two real rows of a grid make one complex line (half the work of a complex transform a row), separated
//             without the factor 1/2, which the scale holds
//   z pass    forward transform, scale and inverse transform in one kernel.  Because the scale is k (k . f) H / |k|^2,
//             the x and y components enter only as a = kx fx + ky fy: two transforms each way instead of three
//   butterflies  of all lines of a block are numbered through and dealt to its threads, so no lane idles for a line
//             length that is no multiple of 32; radices up to 12 run in registers
//   primes    a radix p above 5 runs as p - 1 multiply-adds a point on the sums and differences x_r +- x_{p-r}; where
//             (p - 1) / 2 = 3 q with q prime to 3, five for every nine of them (stage64_thirds)
// The passes run at the float64 rate (x and y on 192^3: 24 operations a point in 97 % of the time that the measured
// 5.0e11 multiply-adds a second would take).  Against cuFFT's D2Z / Z2D with the scale as a pass of its own, both ways,
// float64: three vectors on 192^3 14.96 -> 8.33 ms, on 64^3 0.40 -> 0.30; one vector on 86^3 1.22 -> 0.46, on 240^3
// 12.6 -> 6.3, on 96^3 0.65 -> 0.36 ms; twelve on 25^3 0.147 -> 0.135, on 43^3 0.93 -> 0.79 ms.
#include "fft64.cuh"

#include <math.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

namespace mps {

// ---------------------------------------------------------------------------
// Complex arithmetic and small transforms (forward sign)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 zmul(double2 a, double2 w) {
    return make_double2(fma(a.x, w.x, -a.y * w.y), fma(a.x, w.y, a.y * w.x));
}
__device__ __forceinline__ double2 zmi(double2 a) { return make_double2(a.y, -a.x); }   // -i a
__device__ __forceinline__ double2 zpi(double2 a) { return make_double2(-a.y, a.x); }   // i a

template <int R>
struct Dft64;

template <>
struct Dft64<2> {
    __device__ static __forceinline__ void run(double2 *v) {
        const double2 a = v[0], b = v[1];
        v[0] = zadd(a, b);
        v[1] = zsub(a, b);
    }
};

template <>
struct Dft64<3> {
    __device__ static __forceinline__ void run(double2 *v) {
        const double c = 0.86602540378443864676372317075294;   // sqrt(3) / 2
        const double2 t = zadd(v[1], v[2]), d = zsub(v[1], v[2]);
        const double2 m = make_double2(fma(-0.5, t.x, v[0].x), fma(-0.5, t.y, v[0].y));
        v[0] = zadd(v[0], t);
        v[1] = make_double2(fma(c, d.y, m.x), fma(-c, d.x, m.y));
        v[2] = make_double2(fma(-c, d.y, m.x), fma(c, d.x, m.y));
    }
};

__device__ __forceinline__ void dft4(double2 &a0, double2 &a1, double2 &a2, double2 &a3) {
    const double2 a = zadd(a0, a2), b = zsub(a0, a2), c = zadd(a1, a3), d = zsub(a1, a3);
    a0 = zadd(a, c);
    a2 = zsub(a, c);
    a1 = make_double2(b.x + d.y, b.y - d.x);
    a3 = make_double2(b.x - d.y, b.y + d.x);
}

template <>
struct Dft64<4> {
    __device__ static __forceinline__ void run(double2 *v) { dft4(v[0], v[1], v[2], v[3]); }
};

template <>
struct Dft64<5> {
    __device__ static __forceinline__ void run(double2 *v) {
        const double c1 = 0.30901699437494742410229341718282, c2 = -0.80901699437494742410229341718282;
        const double s1 = 0.95105651629515357211643933337938, s2 = 0.58778525229247312916870595463907;
        const double2 a1 = zadd(v[1], v[4]), b1 = zsub(v[1], v[4]), a2 = zadd(v[2], v[3]), b2 = zsub(v[2], v[3]);
        const double2 m1 = make_double2(fma(c1, a1.x, fma(c2, a2.x, v[0].x)), fma(c1, a1.y, fma(c2, a2.y, v[0].y)));
        const double2 m2 = make_double2(fma(c2, a1.x, fma(c1, a2.x, v[0].x)), fma(c2, a1.y, fma(c1, a2.y, v[0].y)));
        const double2 t1 = make_double2(fma(s1, b1.x, s2 * b2.x), fma(s1, b1.y, s2 * b2.y));
        const double2 t2 = make_double2(fma(s2, b1.x, -s1 * b2.x), fma(s2, b1.y, -s1 * b2.y));
        v[0] = zadd(v[0], zadd(a1, a2));
        v[1] = zadd(m1, zmi(t1));
        v[2] = zadd(m2, zmi(t2));
        v[3] = zadd(m2, zpi(t2));
        v[4] = zadd(m1, zpi(t1));
    }
};

constexpr double kSqrtHalf = 0.70710678118654752440084436210485;
// a times w8 = (1 - i) / sqrt 2, and times w8^3 = -(1 + i) / sqrt 2
__device__ __forceinline__ double2 zw8(double2 a) {
    return make_double2(kSqrtHalf * (a.x + a.y), kSqrtHalf * (a.y - a.x));
}
__device__ __forceinline__ double2 zw83(double2 a) {
    return make_double2(kSqrtHalf * (a.y - a.x), -kSqrtHalf * (a.x + a.y));
}

template <>
struct Dft64<8> {
    __device__ static __forceinline__ void run(double2 *v) {
        dft4(v[0], v[2], v[4], v[6]);
        dft4(v[1], v[3], v[5], v[7]);
        const double2 o1 = zw8(v[3]), o2 = zmi(v[5]), o3 = zw83(v[7]);
        const double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
        v[0] = zadd(e0, o0);
        v[4] = zsub(e0, o0);
        v[1] = zadd(e1, o1);
        v[5] = zsub(e1, o1);
        v[2] = zadd(e2, o2);
        v[6] = zsub(e2, o2);
        v[3] = zadd(e3, o3);
        v[7] = zsub(e3, o3);
    }
};

// Coprime factors A B in registers without twiddles (Good's index maps): input (B n1 + A n2) mod R, output
// (k1 B (1/B mod A) + k2 A (1/A mod B)) mod R.
template <int A, int B>
struct Coprime64 {
    static constexpr int R = A * B;
    static constexpr int inv(int x, int m) {
        for (int i = 1; i < m; ++i)
            if (x * i % m == 1) return i;
        return 1;
    }
    __device__ static __forceinline__ void run(double2 *v) {
        double2 u[R];
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) u[n2 * A + n1] = v[(B * n1 + A * n2) % R];
            Dft64<A>::run(u + n2 * A);
        }
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            double2 c[B];
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) c[n2] = u[n2 * A + k1];
            Dft64<B>::run(c);
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) v[(k1 * B * inv(B % A, A) + k2 * A * inv(A % B, B)) % R] = c[k2];
        }
    }
};
template <>
struct Dft64<6> : Coprime64<3, 2> {};
template <>
struct Dft64<10> : Coprime64<5, 2> {};
template <>
struct Dft64<12> : Coprime64<4, 3> {};

template <>
struct Dft64<9> {
    __device__ static __forceinline__ void run(double2 *v) {
        const double c1 = 0.76604444311897803520239265055542, s1 = 0.64278760968653932632264340990726;   // 2 pi / 9
        const double c2 = 0.17364817766693034885171662676931, s2 = 0.98480775301220805936674302458952;   // 4 pi / 9
        const double c4 = -0.93969262078590838405410927732473, s4 = 0.34202014332566873304409961468226;  // 8 pi / 9
        double2 u[9];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            u[3 * q] = v[q];
            u[3 * q + 1] = v[q + 3];
            u[3 * q + 2] = v[q + 6];
            Dft64<3>::run(u + 3 * q);
        }
        u[4] = zmul(u[4], make_double2(c1, -s1));
        u[5] = zmul(u[5], make_double2(c2, -s2));
        u[7] = zmul(u[7], make_double2(c2, -s2));
        u[8] = zmul(u[8], make_double2(c4, -s4));
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            double2 c[3] = {u[p], u[3 + p], u[6 + p]};
            Dft64<3>::run(c);
            v[p] = c[0];
            v[p + 3] = c[1];
            v[p + 6] = c[2];
        }
    }
};

// ---------------------------------------------------------------------------
// Stages on the lines of a block (nl lines of p.N points, line stride ld)
// ---------------------------------------------------------------------------
template <int R>
__device__ __forceinline__ void stage64(const double2 *in, double2 *out, int nl, int ld, int N, int Ns,
                                        const double2 *__restrict__ tw) {
    const unsigned NR = N / R;
    for (unsigned w = threadIdx.x; w < nl * NR; w += blockDim.x) {
        const unsigned line = w / NR, j = w - line * NR, jq = j / Ns, jm = j - jq * Ns;
        const double2 *a = in + line * ld + j;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = a[r * NR];
        if (Ns > 1) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = zmul(v[r], tw[jm * R + r]);
        }
        Dft64<R>::run(v);
        double2 *o = out + line * ld + jq * Ns * R + jm;
#pragma unroll
        for (int r = 0; r < R; ++r) o[r * Ns] = v[r];
    }
}

// Prime radix: x_r and x_{R-r} become their sum and difference in place, then each thread forms the output pair
// k, R - k of one butterfly: X_k = x_0 + sum_r (a_r cos - i b_r sin), X_{R-k} with + i.
__device__ __forceinline__ void stage64_prime(double2 *in, double2 *out, int nl, int ld, int N, int R, int Ns,
                                              const double2 *__restrict__ tw, const double2 *__restrict__ root) {
    const unsigned NR = N / R, h = (R - 1) / 2;
    for (unsigned w = threadIdx.x; w < nl * NR * h; w += blockDim.x) {
        const unsigned r = w / (nl * NR) + 1, lj = w % (nl * NR), line = lj / NR, j = lj - line * NR, jm = j % Ns;
        double2 *a = in + line * ld + j;
        double2 u = a[r * NR], v = a[(R - r) * NR];
        if (Ns > 1) {
            u = zmul(u, tw[jm * R + r]);
            v = zmul(v, tw[jm * R + R - r]);
        }
        a[r * NR] = zadd(u, v);
        a[(R - r) * NR] = zsub(u, v);
    }
    __syncthreads();
    for (unsigned w = threadIdx.x; w < nl * NR * (h + 1); w += blockDim.x) {
        const unsigned k = w / (nl * NR), lj = w % (nl * NR), line = lj / NR, j = lj - line * NR, jq = j / Ns,
                       jm = j - jq * Ns;
        const double2 *a = in + line * ld + j;
        double2 p = a[0], q = make_double2(0.0, 0.0);
        unsigned i = 0;
#pragma unroll 3
        for (unsigned r = 1; r <= h; ++r) {
            i += k;
            if (i >= (unsigned)R) i -= R;
            const double2 e = root[i], s = a[r * NR], d = a[(R - r) * NR];   // e = (cos, sin)
            p.x = fma(s.x, e.x, p.x);
            p.y = fma(s.y, e.x, p.y);
            q.x = fma(d.x, e.y, q.x);
            q.y = fma(d.y, e.y, q.y);
        }
        double2 *o = out + line * ld + jq * Ns * R + jm;
        o[k * Ns] = make_double2(p.x + q.y, p.y - q.x);
        if (k > 0) o[(R - k) * Ns] = make_double2(p.x - q.y, p.y + q.x);
    }
}

// Prime radix R with (R - 1) / 2 = 3 q, q prime to 3.  With r = g^T, k = g^S (g a generator), the sums over r of
// a_r cos(2 pi k r / R) and d_r sin(2 pi k r / R) are correlations over the exponents, Z_3 x Z_2q: the coefficient
// depends on (s1 + t1 mod 3, s2 + t2) only (and changes sign, the sine's, or not with s2 + t2 -> + q), t1 in Z_3, t2 <
// q standing for the pairs r, R - r.  In the direction of 3, with c_u = c' + c~_u, c' their mean,
//   y_s = c' (a_0 + a_1 + a_2) + z_s,
//   z_0 = alpha c~_0 + beta c~_1,  z_1 = alpha c~_1 + beta c~_2,  z_2 = -(z_0 + z_1),
// alpha = a_0 - a_2, beta = a_1 - a_2 (the c~ sum to zero): five multiplications instead of nine.
//   1  sums and differences of the pairs, then sum, alpha and beta of each triple of them, in place
//   2  a thread takes one part (cosine, sine), one component (re, im) and one s2 of a butterfly: three outputs
//   3  the outputs k and R - k from their two parts
// tab: q triples r (packed integers), then for the cosines and the sines 2 q entries (c', c~_0, c~_1, c~_2).
// Both ways, one vector on 86^3 (2 x 43) 0.58 -> 0.46 ms, 36 on 31^3 0.60 -> 0.54, one on 103^3 1.78 -> 1.15.
__device__ __forceinline__ void stage64_thirds(double2 *in, double2 *out, int nl, int ld, int N, int R, int q, int Ns,
                                               const double2 *__restrict__ tw, const double2 *__restrict__ tab) {
    const unsigned NR = N / R, nb = nl * NR;
    for (unsigned w = threadIdx.x; w < nb * q; w += blockDim.x) {
        const unsigned t = w / nb, lj = w - t * nb, line = lj / NR, j = lj - line * NR, jm = j % Ns;
        double2 *a = in + line * ld + j;
        const double2 pr = tab[t];
        const int r[3] = {__double2loint(pr.x), __double2hiint(pr.x), __double2loint(pr.y)};
        double2 s[3], d[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double2 u = a[r[c] * NR], v = a[(R - r[c]) * NR];
            if (Ns > 1) {
                u = zmul(u, tw[jm * R + r[c]]);
                v = zmul(v, tw[jm * R + R - r[c]]);
            }
            s[c] = zadd(u, v);
            d[c] = zsub(u, v);
        }
        a[r[0] * NR] = zadd(zadd(s[0], s[1]), s[2]);
        a[r[1] * NR] = zsub(s[0], s[2]);
        a[r[2] * NR] = zsub(s[1], s[2]);
        a[(R - r[0]) * NR] = zadd(zadd(d[0], d[1]), d[2]);
        a[(R - r[1]) * NR] = zsub(d[0], d[2]);
        a[(R - r[2]) * NR] = zsub(d[1], d[2]);
    }
    __syncthreads();
    for (unsigned w = threadIdx.x; w < nb * (4 * q + 2); w += blockDim.x) {
        const unsigned e = w / nb, lj = w - e * nb, line = lj / NR, j = lj - line * NR, jq = j / Ns, jm = j - jq * Ns;
        const unsigned comp = e & 1, s2 = e >> 2;
        const bool sine = e & 2;
        const double *a = (const double *)(in + line * ld + j) + comp;
        double *o = (double *)(out + line * ld + jq * Ns * R + jm) + comp;
        if (s2 == (unsigned)q) {   // X_0
            double m = a[0];
            for (int t = 0; t < q; ++t) m += a[2 * NR * __double2loint(tab[t].x)];
            o[0] = m;
            continue;
        }
        const double2 *c = tab + q + (sine ? 4 * q : 0) + 2 * s2;
        double m = sine ? 0.0 : a[0], z0 = 0.0, z1 = 0.0;
#pragma unroll 2
        for (int t = 0; t < q; ++t) {
            const double2 pr = tab[t], c0 = c[2 * t], c1 = c[2 * t + 1];   // (c', c~0), (c~1, c~2)
            const int r0 = __double2loint(pr.x), r1 = __double2hiint(pr.x), r2 = __double2loint(pr.y);
            const double sum = a[2 * NR * (sine ? R - r0 : r0)], al = a[2 * NR * (sine ? R - r1 : r1)],
                         be = a[2 * NR * (sine ? R - r2 : r2)];
            m = fma(sum, c0.x, m);
            z0 = fma(al, c0.y, fma(be, c1.x, z0));
            z1 = fma(al, c1.x, fma(be, c1.y, z1));
        }
        const double2 pk = tab[s2];
        const int k0 = __double2loint(pk.x), k1 = __double2hiint(pk.x), k2 = __double2loint(pk.y);
        o[2 * Ns * (sine ? R - k0 : k0)] = m + z0;
        o[2 * Ns * (sine ? R - k1 : k1)] = m + z1;
        o[2 * Ns * (sine ? R - k2 : k2)] = m - (z0 + z1);
    }
    __syncthreads();
    for (unsigned w = threadIdx.x; w < nb * 3 * q; w += blockDim.x) {
        const unsigned e = w / nb, lj = w - e * nb, line = lj / NR, j = lj - line * NR, jq = j / Ns, jm = j - jq * Ns;
        const unsigned t = e / 3, c = e - 3 * t;
        const double2 pr = tab[t];
        const int k = c == 0 ? __double2loint(pr.x) : (c == 1 ? __double2hiint(pr.x) : __double2loint(pr.y));
        double2 *o = out + line * ld + jq * Ns * R + jm;
        const double2 u = o[k * Ns], v = o[(R - k) * Ns];
        o[k * Ns] = make_double2(u.x + v.y, u.y - v.x);
        o[(R - k) * Ns] = make_double2(u.x - v.y, u.y + v.x);
    }
}

// Forward transform of the nl lines in a (b: scratch of the same size); returns the buffer with the result.  All
// threads of the block call it; the lines are complete in a, and the result is complete on return.
__device__ double2 *fft64_lines(double2 *a, double2 *b, int nl, int ld, const F64Axis &p) {
    for (int s = 0; s < p.nst; ++s) {
        const double2 *t = p.tw + p.twoff[s];
        switch (p.R[s]) {
#define F64_STAGE(R) case R: stage64<R>(a, b, nl, ld, p.N, p.Ns[s], t); break;
            F64_STAGE(2)
            F64_STAGE(3)
            F64_STAGE(4)
            F64_STAGE(5)
            F64_STAGE(6)
            F64_STAGE(8)
            F64_STAGE(9)
            F64_STAGE(10)
            F64_STAGE(12)
#undef F64_STAGE
            default:
                if (p.third[s])
                    stage64_thirds(a, b, nl, ld, p.N, p.R[s], p.third[s], p.Ns[s], t, p.tw + p.rtoff[s]);
                else
                    stage64_prime(a, b, nl, ld, p.N, p.R[s], p.Ns[s], t, p.tw + p.rtoff[s]);
                break;
        }
        __syncthreads();
        double2 *x = a;
        a = b;
        b = x;
    }
    return a;
}

// ---------------------------------------------------------------------------
// x pass: two rows of Nx of a grid are one complex line (npairs lines over all the stacked grids)
// ---------------------------------------------------------------------------
// 5 blocks an SM (96 registers): 8.33 ms for three vectors on 192^3 against 8.35 at 4 blocks; with radices 15 and 16 as
// well (128 registers, 4 blocks) 8.56, with none above 8 8.61.
constexpr int kF64Threads = 128, kF64Blocks = 5;

__global__ void __launch_bounds__(kF64Threads, kF64Blocks)
    k_f64_x_fwd(const double *__restrict__ grid,
                double2 *__restrict__ spec, int64_t npairs, RowPairs rp, F64Axis px,
                int L) {
    extern __shared__ double2 sm64[];
    const int Nx = px.N, Nxh = Nx / 2 + 1, ld = Nx | 1;
    const int64_t ntiles = (npairs + L - 1) / L;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t p0 = tile * L;
        const int nl = (int)min((int64_t)L, npairs - p0);
        const RowPairs::Lines ln = rp.from(p0);
        const double *rows = grid + ln.row0 * Nx;
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nx); i += blockDim.x) {
            const unsigned line = i / Nx, n = i - line * Nx;
            bool two;
            const double *row = rows + (int64_t)ln.row(line, &two) * Nx + n;
            sm64[line * ld + n] = make_double2(row[0], two ? row[Nx] : 0.0);
        }
        __syncthreads();
        const double2 *Z = fft64_lines(sm64, sm64 + L * ld, nl, ld, px);
        double2 *out = spec + ln.row0 * Nxh;
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nxh); i += blockDim.x) {
            const unsigned line = i / Nxh, k = i - line * Nxh;
            const double2 a = Z[line * ld + k], b = Z[line * ld + (k ? Nx - k : 0)];
            bool two;
            double2 *o = out + (int64_t)ln.row(line, &two) * Nxh + k;
            o[0] = make_double2(a.x + b.x, a.y - b.y);
            if (two) o[Nxh] = make_double2(a.y + b.y, b.x - a.x);
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kF64Threads, kF64Blocks)
    k_f64_x_inv(const double2 *__restrict__ spec, double *__restrict__ grid,
                int64_t npairs, RowPairs rp, F64Axis px, int L) {
    extern __shared__ double2 sm64[];
    const int Nx = px.N, Nxh = Nx / 2 + 1, ld = Nx | 1;
    const int64_t ntiles = (npairs + L - 1) / L;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t p0 = tile * L;
        const int nl = (int)min((int64_t)L, npairs - p0);
        const RowPairs::Lines ln = rp.from(p0);
        const double2 *in = spec + ln.row0 * Nxh;
        // conj(X0 + i X1) at k and, from the Hermitian halves, at N - k; the real bins' imaginary parts are dropped
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nxh); i += blockDim.x) {
            const unsigned line = i / Nxh, k = i - line * Nxh;
            bool two;
            const double2 *row = in + (int64_t)ln.row(line, &two) * Nxh + k;
            double2 a = row[0], b = two ? row[Nxh] : make_double2(0.0, 0.0);
            const bool real_bin = k == 0 || 2 * k == (unsigned)Nx;
            if (real_bin) a.y = b.y = 0.0;
            sm64[line * ld + k] = make_double2(a.x - b.y, -(a.y + b.x));
            if (!real_bin) sm64[line * ld + Nx - k] = make_double2(a.x + b.y, a.y - b.x);
        }
        __syncthreads();
        const double2 *Z = fft64_lines(sm64, sm64 + L * ld, nl, ld, px);
        double *rows = grid + ln.row0 * Nx;
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nx); i += blockDim.x) {
            const unsigned line = i / Nx, n = i - line * Nx;
            const double2 z = Z[line * ld + n];   // conj of the inverse transform
            bool two;
            double *row = rows + (int64_t)ln.row(line, &two) * Nx + n;
            row[0] = z.x;
            if (two) row[Nx] = -z.y;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// y pass: L consecutive columns of the (component, z) planes, numbered through all planes: a tile of the one column
// that 33 leave over beside four times eight would cost a warp's float64 instruction as much as a whole one (three
// vectors on 64^3 54.9 -> 50.9 us a pass)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kF64Threads, kF64Blocks)
    k_f64_y(double2 *__restrict__ spec, int64_t nplanes, int Nxh, F64Axis py,
            int L, int inverse) {
    extern __shared__ double2 sm64[];
    const int Ny = py.N, ld = Ny | 1;
    const double sg = inverse ? -1.0 : 1.0;
    const int64_t total = nplanes * Nxh, plane_len = (int64_t)Ny * Nxh;
    for (int64_t tile = blockIdx.x; tile * L < total; tile += gridDim.x) {
        const int64_t c0 = tile * L, p0 = c0 / Nxh;
        const unsigned k0 = (unsigned)(c0 - p0 * Nxh);
        const int nl = (int)min((int64_t)L, total - c0);
        double2 *base = spec + p0 * plane_len;
        auto column = [&](unsigned t) {   // offset of the tile's column t
            const unsigned k = k0 + t, w = k / (unsigned)Nxh;
            return (int64_t)w * plane_len + (k - w * (unsigned)Nxh);
        };
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Ny); i += blockDim.x) {
            const unsigned y = i / nl, t = i - y * nl;
            const double2 v = base[column(t) + (int64_t)y * Nxh];
            sm64[t * ld + y] = make_double2(v.x, sg * v.y);
        }
        __syncthreads();
        const double2 *Z = fft64_lines(sm64, sm64 + L * ld, nl, ld, py);
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Ny); i += blockDim.x) {
            const unsigned y = i / nl, t = i - y * nl;
            const double2 v = Z[t * ld + y];
            base[column(t) + (int64_t)y * Nxh] = make_double2(v.x, sg * v.y);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// z pass with the dipole scale: L consecutive kx columns at one ky, the 3 components of one vector.
// out = k (k . f) hs, the sum over the components whose axis is on its Nyquist bin apart from the others' (the real
// part of the complex pipeline's coupling).  Columns with both or neither of kx, ky on the Nyquist bin need two lines,
// a = kx fx + ky fy and b = fz:  out_x = kx t, out_y = ky t, out_z = u with t, u the inverse transforms of
// hs (a + kz b) and hs kz (a + kz b); where z is on the other side of the rule than x and y, of hs a and hs kz^2 b.
// A block that holds one of the few other columns takes three lines a column.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kF64Threads, kF64Blocks)
    k_f64_z_scale(double2 *__restrict__ spec, int nrhs, GridParams gp,
                  F64Axis pz, const double *__restrict__ hs, int L) {
    extern __shared__ double2 sm64[];
    const int Nx = gp.N[0], Ny = gp.N[1], Nz = gp.N[2], Nxh = Nx / 2 + 1, ld = Nz | 1, nblk = (Nxh + L - 1) / L;
    const int64_t zs = (int64_t)Ny * Nxh, Gc = zs * Nz;
    double2 *buf = sm64, *other = sm64 + 3 * L * ld;
    const int64_t ntiles = (int64_t)nrhs * Ny * nblk;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int kx0 = (int)(tile % nblk) * L, nl = min(L, Nxh - kx0);
        const int ky = (int)((tile / nblk) % Ny), r = (int)(tile / ((int64_t)nblk * Ny));
        double2 *base = spec + (int64_t)(3 * r) * Gc + (int64_t)ky * Nxh + kx0;
        const bool nyy = 2 * ky == Ny, has_nyx = 2 * (kx0 + nl - 1) == Nx;   // the last column may be x's Nyquist bin
        const double qy = fft_freq(ky, Ny) * gp.kfac[1];
        const bool two = nyy ? (nl == 1 && has_nyx) : !has_nyx;
        const int nlines = two ? 2 * nl : 3 * nl;
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nz); i += blockDim.x) {
            const unsigned z = i / nl, t = i - z * nl;
            const double2 *f = base + z * zs + t;
            const double2 fx = f[0], fy = f[Gc], fz = f[2 * Gc];
            double2 *o = buf + t * ld + z;
            if (two) {
                const double qx = fft_freq(kx0 + t, Nx) * gp.kfac[0];
                o[0] = make_double2(fma(qx, fx.x, qy * fy.x), fma(qx, fx.y, qy * fy.y));
                o[nl * ld] = fz;
            } else {
                o[0] = fx;
                o[nl * ld] = fy;
                o[2 * nl * ld] = fz;
            }
        }
        __syncthreads();
        double2 *Z = fft64_lines(buf, other, nlines, ld, pz);
        // the inverse transform runs on the conjugate
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nz); i += blockDim.x) {
            const unsigned z = i / nl, t = i - z * nl;
            const double qz = fft_freq(z, Nz) * gp.kfac[2];
            const bool nyz = 2 * (int)z == Nz;
            const double h = hs[z * zs + (int64_t)ky * Nxh + kx0 + t];
            double2 *o = Z + t * ld + z;
            if (two) {
                const double2 a = o[0], b = o[nl * ld];
                double2 s = a, u = make_double2(qz * b.x, qz * b.y);   // nyy == nyx here
                if (nyz == nyy) {
                    s = zadd(a, u);
                    u = s;
                }
                const double g = h * qz;
                o[0] = make_double2(h * s.x, -(h * s.y));
                o[nl * ld] = make_double2(g * u.x, -(g * u.y));
            } else {
                const bool ny[3] = {2 * (kx0 + (int)t) == Nx, nyy, nyz};
                const double q[3] = {fft_freq(kx0 + t, Nx) * gp.kfac[0], qy, qz};
                double2 s0 = make_double2(0.0, 0.0), s1 = s0;   // off and on the Nyquist bins
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const double2 f = o[c * nl * ld];
                    double2 &s = ny[c] ? s1 : s0;
                    s.x = fma(q[c], f.x, s.x);
                    s.y = fma(q[c], f.y, s.y);
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const double2 s = ny[c] ? s1 : s0;
                    o[c * nl * ld] = make_double2(h * q[c] * s.x, -(h * q[c] * s.y));
                }
            }
        }
        __syncthreads();
        Z = fft64_lines(Z, Z == buf ? other : buf, nlines, ld, pz);
        for (unsigned i = threadIdx.x; i < (unsigned)(nl * Nz); i += blockDim.x) {
            const unsigned z = i / nl, t = i - z * nl;
            double2 *f = base + z * zs + t;
            const double2 *o = Z + t * ld + z;
            if (two) {
                const double qx = fft_freq(kx0 + t, Nx) * gp.kfac[0];
                const double2 v = o[0], u = o[nl * ld];
                f[0] = make_double2(qx * v.x, -(qx * v.y));
                f[Gc] = make_double2(qy * v.x, -(qy * v.y));
                f[2 * Gc] = make_double2(u.x, -u.y);
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) f[c * Gc] = make_double2(o[c * nl * ld].x, -o[c * nl * ld].y);
            }
        }
        __syncthreads();
    }
}

__global__ void k_f64_scale_coef(GridParams gp, const double *__restrict__ H, double *__restrict__ hs) {
    const HalfQuarter q(gp.N);
    const int64_t Gq = q.size();
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < Gq; t += (int64_t)gridDim.x * blockDim.x) {
        int ix, iy, iz;
        q.point(t, &ix, &iy, &iz);
        const double kx = fft_freq(ix, gp.N[0]) * gp.kfac[0];
        const double ky = fft_freq(iy, gp.N[1]) * gp.kfac[1];
        const double kz = fft_freq(iz, gp.N[2]) * gp.kfac[2];
        const double k2 = kx * kx + ky * ky + kz * kz;
        const double v = k2 > 0 ? 0.5 * H[((int64_t)iz * q.Ny + iy) * q.Nxh + ix] / k2 : 0.0;
        mirror_points(q, ix, iy, iz, [&](int64_t i, int, int) { hs[i] = v; });
    }
}

int f64_scale_coef(const GridParams &gp, const double *H, double *hs, cudaStream_t s) {
    k_f64_scale_coef<<<grid_for(HalfQuarter(gp.N).size(), 256), 256, 0, s>>>(gp, H, hs);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

// ---------------------------------------------------------------------------
// Plans
// ---------------------------------------------------------------------------
constexpr double kF64StageCost = 1.0;
static std::map<std::pair<int, int>, F64Axis> g_f64_axes;   // per (device, length); at most kF64MaxN lengths
static std::mutex g_f64_mu;

// Radices of a 2-3-5 length with the fewest float64 operations (twiddles included; the first stage of a transform has
// none) plus a charge for each stage's passes over shared memory.
static std::vector<int> f64_radices(int n, bool first) {
    static const struct { int R; double ops; } kR[] = {{2, 4}, {3, 12}, {4, 16}, {5, 36}, {6, 36}, {8, 56},
        {9, 88}, {10, 92},
        {12, 96},
        };
    std::vector<int> best;
    double cost = 1e30;
    std::vector<int> cur;
    auto search = [&](auto &self, int left, double c) -> void {
        if (c >= cost) return;
        if (left == 1) {
            cost = c;
            best = cur;
            return;
        }
        for (const auto &r : kR)
            if (left % r.R == 0) {
                const bool tw = !(first && cur.empty());
                cur.push_back(r.R);
                self(self, left / r.R, c + (r.ops + (tw ? 4.0 * (r.R - 1) : 0.0)) / r.R + kF64StageCost);
                cur.pop_back();
            }
    };
    search(search, n, 0.0);
    return best;
}

// q of a prime whose (R - 1) / 2 = 3 q with q prime to 3; below q = 5 the split costs what it saves.
static int f64_third(int R) {
    const int q = (R - 1) / 6;
    return (R - 1) % 6 == 0 && q % 3 != 0 && q >= 5 ? q : 0;
}

// The table of stage64_thirds.
static void f64_thirds_table(int R, int q, std::vector<double2> &tw) {
    std::vector<int> power(R - 1);   // g^e mod R of the smallest generator g
    for (int g = 2;; ++g) {
        int x = 1, e = 0;
        do {
            power[e++] = x;
            x = x * g % R;
        } while (x != 1);
        if (e == R - 1) break;
    }
    auto at = [&](int u1, int u2) {   // the element whose exponent is u1 mod 3 and u2 mod 2 q
        int e = u2 % (2 * q);
        while (e % 3 != u1 % 3) e += 2 * q;
        return power[e];
    };
    auto pack = [](int lo, int hi) {
        const uint64_t b = (uint64_t)(uint32_t)lo | ((uint64_t)(uint32_t)hi << 32);
        double d;
        memcpy(&d, &b, sizeof d);
        return d;
    };
    for (int t = 0; t < q; ++t) tw.push_back(make_double2(pack(at(0, t), at(1, t)), pack(at(2, t), 0)));
    for (int sine = 0; sine < 2; ++sine)
        for (int u = 0; u < 2 * q; ++u) {
            double c[3];
            for (int k = 0; k < 3; ++k) {
                const double ang = 2.0 * M_PI * (double)at(k, u) / (double)R;
                c[k] = sine ? sin(ang) : cos(ang);
            }
            const double mean = (c[0] + c[1] + c[2]) / 3.0;
            tw.push_back(make_double2(mean, c[0] - mean));
            tw.push_back(make_double2(c[1] - mean, c[2] - mean));
        }
}

// MPS_OK with supported = false for a length that the transforms do not take; other status codes are failures that say
// nothing about the length.
static int f64_axis(int N, int dev, F64Axis *out, bool *supported) {
    *supported = false;
    if (N < 2 || N > kF64MaxN) return MPS_OK;
    std::lock_guard<std::mutex> lk(g_f64_mu);
    auto it = g_f64_axes.find({dev, N});
    if (it != g_f64_axes.end()) {
        *out = it->second;
        *supported = true;
        return MPS_OK;
    }
    F64Axis p;
    p.N = N;
    // primes above 5 first (their first stage has no twiddles), the rest by the cheapest sequence of radices
    std::vector<int> radices;
    int m = N;
    for (int f : {2, 3, 5})
        while (m % f == 0) m /= f;
    const int smooth = N / m;
    for (int f = 7; f <= m; f += 2)
        while (m % f == 0) {
            if (f > kF64MaxPrime) return MPS_OK;
            radices.push_back(f);
            m /= f;
        }
    const std::vector<int> rest = f64_radices(smooth, radices.empty());
    radices.insert(radices.end(), rest.begin(), rest.end());
    if (radices.size() > (size_t)kF64MaxStages) return MPS_OK;
    std::vector<double2> tw;
    int ns = 1;
    for (int R : radices) {
        const int s = p.nst++;
        p.R[s] = R;
        p.Ns[s] = ns;
        p.twoff[s] = (int)tw.size();
        for (int jm = 0; jm < ns; ++jm)
            for (int r = 0; r < R; ++r) {
                const double ang = -2.0 * M_PI * (double)((jm * r) % (ns * R)) / (double)(ns * R);
                tw.push_back(make_double2(cos(ang), sin(ang)));
            }
        p.rtoff[s] = (int)tw.size();
        const bool prime = s < (int)(radices.size() - rest.size());
        p.third[s] = prime ? f64_third(R) : 0;
        if (p.third[s])
            f64_thirds_table(R, p.third[s], tw);
        else if (prime)
            for (int r = 0; r < R; ++r) {
                const double ang = 2.0 * M_PI * (double)r / (double)R;
                tw.push_back(make_double2(cos(ang), sin(ang)));
            }
        ns *= R;
    }
    double2 *d = nullptr;
    // before another thread can find the plan
    const int rc = upload_table(tw.data(), sizeof(double2) * tw.size(), (void **)&d);
    if (rc) return rc;
    p.tw = d;
    g_f64_axes[{dev, N}] = p;
    *out = p;
    *supported = true;
    return MPS_OK;
}

int f64_plan(const GridParams &gp, F64Plan3 *out) {
    out->ok = false;
    int dev = 0;
    MPS_CUDA_TRY(cudaGetDevice(&dev));
    for (int d = 0; d < 3; ++d) {
        bool supported;
        const int rc = f64_axis(gp.N[d], dev, &out->ax[d], &supported);
        if (rc || !supported) return rc;
    }
    out->ok = true;
    return MPS_OK;
}

// Both ways, cuFFT against these, us.  Fused, with the scale: rods behind a short x lose (12 x 12 x 400, 12 and 24
// vectors 408 against 534 and 767 against 1012; 10 x 20 x 400, 3 vectors 177 against 221), wider ones and longer x do
// not (12 x 48 x 400, 3 vectors 458 against 438; 14 x 14 x 500, 24 vectors 1519 against 1280; 400 x 12 x 12 1118
// against 770).
// Not fused, short axes: few grids leave cuFFT waiting for its launches, many leave these too few butterflies a block.
// 4 grids on 18^3, 22^3, 24^3, 28^3 57 against 47, 78 and 50, 62 and 57, 75 and 53; 16 grids 57 and 53, 79 and 65, 71
// and 75, 94 and 101; 24 grids 57 and 54, 82 and 85, 79 and 103, 117 and 115; 96 grids 103 and 123, 193 and 205, 188
// and 260, 325 and 327.  On 30^3, 32^3, 36^3, 48^3 96 grids 456 against 421, 415 and 385, 700 and 627, 1793 and 1250.
bool f64_pays(const GridParams &gp, bool fused, int ngrids) {
    const int longest = std::max({gp.N[0], gp.N[1], gp.N[2]});
    if (fused) return gp.N[0] >= 14 || longest < 200 || std::min(gp.N[1], gp.N[2]) >= 40;
    return ngrids < 20 || std::min({gp.N[0], gp.N[1], gp.N[2]}) >= 30;
}

// Lines per block: up to 8 (full 128-byte rows of the strided passes) within about 56 KB of shared memory (4 blocks an
// SM), fewer where the grid has too few lines to give every SM two blocks.
constexpr size_t kF64Smem = 56 * 1024;

static int f64_lines(int N, int per_line, int64_t lines) {
    const size_t line = sizeof(double2) * 2 * (size_t)per_line * (N | 1);
    int L = 8;
    while (L > 1 && (line * L > kF64Smem || lines / L < 304)) L /= 2;
    return L;
}

// One value for every launch of a kernel (a line triple of the longest axis): calls from several threads agree.
constexpr int kF64SmemMax = (int)(sizeof(double2) * 6 * (kF64MaxN | 1));

template <typename K>
static int f64_smem(K kernel, size_t bytes) {
    if (bytes > 48 * 1024)
        MPS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kF64SmemMax));
    return MPS_OK;
}

static int f64_x(bool fwd, const double *gin, double *gout, double2 *spec, int ncomp, const GridParams &gp,
                 const F64Axis &px, cudaStream_t s) {
    const RowPairs rp((int64_t)gp.N[2] * gp.N[1]);
    const int64_t npairs = (int64_t)ncomp * rp.pairs;
    const int L = f64_lines(px.N, 1, npairs);
    const size_t smem = sizeof(double2) * 2 * (size_t)L * (px.N | 1);
    const unsigned blocks = grid_for((npairs + L - 1) / L, 1, INT32_MAX);
    if (fwd) {
        const int rc = f64_smem(k_f64_x_fwd, smem);
        if (rc) return rc;
        k_f64_x_fwd<<<blocks, kF64Threads, smem, s>>>(gin, spec, npairs, rp, px, L);
    } else {
        const int rc = f64_smem(k_f64_x_inv, smem);
        if (rc) return rc;
        k_f64_x_inv<<<blocks, kF64Threads, smem, s>>>(spec, gout, npairs, rp, px, L);
    }
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

// Transform along the middle axis of nplanes arrays of p.N x Nxh: y of every z plane, or z of whole spectra.
static int f64_y(double2 *spec, int64_t nplanes, int Nxh, const F64Axis &py, int inverse, cudaStream_t s) {
    const int L = f64_lines(py.N, 1, nplanes * Nxh);
    const size_t smem = sizeof(double2) * 2 * (size_t)L * (py.N | 1);
    const int rc = f64_smem(k_f64_y, smem);
    if (rc) return rc;
    k_f64_y<<<grid_for((nplanes * Nxh + L - 1) / L, 1, INT32_MAX), kF64Threads, smem, s>>>(spec, nplanes, Nxh, py, L, inverse);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

int f64_forward_xy(const double *grid, void *spec, int ncomp, const GridParams &gp, const F64Plan3 &pl,
                   cudaStream_t s) {
    if (!pl.ok) return MPS_BAD_ARG;
    const int rc = f64_x(true, grid, nullptr, (double2 *)spec, ncomp, gp, pl.ax[0], s);
    return rc ? rc : f64_y((double2 *)spec, (int64_t)ncomp * gp.N[2], gp.N[0] / 2 + 1, pl.ax[1], 0, s);
}

int f64_inverse_yx(void *spec, double *grid, int ncomp, const GridParams &gp, const F64Plan3 &pl, cudaStream_t s) {
    if (!pl.ok) return MPS_BAD_ARG;
    const int rc = f64_y((double2 *)spec, (int64_t)ncomp * gp.N[2], gp.N[0] / 2 + 1, pl.ax[1], 1, s);
    return rc ? rc : f64_x(false, nullptr, grid, (double2 *)spec, ncomp, gp, pl.ax[0], s);
}

int f64_z(void *spec, int ncomp, const GridParams &gp, const F64Plan3 &pl, int inverse, cudaStream_t s) {
    if (!pl.ok) return MPS_BAD_ARG;
    return f64_y((double2 *)spec, ncomp, (gp.N[0] / 2 + 1) * gp.N[1], pl.ax[2], inverse, s);
}

int f64_z_scale_dipole(void *spec, int nrhs, const GridParams &gp, const F64Plan3 &pl, const double *hs,
                       cudaStream_t s) {
    if (!pl.ok) return MPS_BAD_ARG;
    const int Nxh = gp.N[0] / 2 + 1, L = f64_lines(gp.N[2], 3, (int64_t)nrhs * gp.N[1] * Nxh);
    const int nblk = (Nxh + L - 1) / L;
    const size_t smem = sizeof(double2) * 6 * (size_t)L * (gp.N[2] | 1);
    const int rc = f64_smem(k_f64_z_scale, smem);
    if (rc) return rc;
    k_f64_z_scale<<<grid_for((int64_t)nrhs * gp.N[1] * nblk, 1, INT32_MAX), kF64Threads, smem, s>>>(
        (double2 *)spec, nrhs, gp, pl.ax[2], hs, L);
    MPS_LAUNCH_CHECK();
    return MPS_OK;
}

}  // namespace mps
