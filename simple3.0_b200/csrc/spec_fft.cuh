// spec_fft.cuh -- FP64 transforms over the angular samples, for the m-domain spectra of the search
// (k_search.cu), its re-score (k_stage2.cu) and the exact correlations (k_exact_fft.cu).
//
// The spectra are U(m, k) = sum_{n<P} v_m(n, k) w_N^{-mn}, m = 0..P, N = 2P, with v_m the
// real part of the polar sample a(n, k) for even m and its imaginary part for odd m: for m = 2j the
// length-P DFT of the real parts at j, for m = 2j + 1 that of the imaginary parts times w_N^{-n}.  Two
// shells k, k' go through one complex transform, Z = DFT(v_k + i v_k'), and come apart by the
// symmetry of real sequences,
//   even m:  U_k(2j) = (Z(j) + conj Z(P - j)) / 2,       U_k'(2j) = -i (Z(j) - conj Z(P - j)) / 2,
//   odd m:   the same with Z(P - 1 - j), as U(-m) = conj U(m) and w_N^{-n} shifts the frequencies by 1/2,
// so a shell pair costs one length-P transform per parity of m (and one for the squares that the
// normaliser needs) where a length-N transform per shell had four to eight times the operations.
// A transform is one Cooley-Tukey split P = P1 P2, in FP64 with FP64 twiddles:
//   pass 1, task (transform, n1): a length-P2 DFT over n2 of f(n1 + P1 n2), times w_P^{-n1 k2},
//           into row k2 of the transform's rows [P2][P1 | 1] (odd: conflict-free in both passes);
//   pass 2, task (transform, k2): a length-P1 DFT over n1 of row k2, in place: F(k2 + P2 k1) at k1.
#pragma once

#include <cuda_runtime.h>

namespace pftcc {
namespace sfft {

__device__ __forceinline__ double2 d_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 d_sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 d_mul(double2 a, double2 b)
{
    // rounded products, so that no caller's inlining contracts them differently
    return make_double2(fma(a.x, b.x, -__dmul_rn(a.y, b.y)), fma(a.x, b.y, __dmul_rn(a.y, b.x)));
}

// forward radix butterflies (the textbook radix-2/3/4/5 DFT formulas), FP64
template <int F> struct DBfly;
template <> struct DBfly<2> {
    __device__ static void run(double2 *v) { const double2 a = v[0], b = v[1]; v[0] = d_add(a, b); v[1] = d_sub(a, b); }
};
template <> struct DBfly<4> {
    __device__ static void run(double2 *v)
    {
        const double2 t0 = d_add(v[0], v[2]), t1 = d_sub(v[0], v[2]);
        const double2 t2 = d_add(v[1], v[3]), d = d_sub(v[1], v[3]);
        v[0] = d_add(t0, t2);
        v[2] = d_sub(t0, t2);
        v[1] = make_double2(t1.x + d.y, t1.y - d.x);   // t1 - i d
        v[3] = make_double2(t1.x - d.y, t1.y + d.x);   // t1 + i d
    }
};
template <> struct DBfly<3> {
    __device__ static void run(double2 *v)
    {
        const double s3 = 0.86602540378443864676;   // sin(2 pi / 3)
        const double2 a = v[0], t1 = d_add(v[1], v[2]), d = d_sub(v[1], v[2]);
        const double2 t2 = make_double2(fma(t1.x, -0.5, a.x), fma(t1.y, -0.5, a.y));
        v[0] = d_add(a, t1);
        v[1] = make_double2(fma(d.y, s3, t2.x), fma(d.x, -s3, t2.y));
        v[2] = make_double2(fma(d.y, -s3, t2.x), fma(d.x, s3, t2.y));
    }
};
template <> struct DBfly<5> {
    __device__ static void run(double2 *v)
    {
        const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;   // cos(2pi/5), cos(4pi/5)
        const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;    // sin(2pi/5), sin(4pi/5)
        const double2 a = v[0];
        const double2 t1 = d_add(v[1], v[4]), t2 = d_add(v[2], v[3]);
        const double2 t3 = d_sub(v[1], v[4]), t4 = d_sub(v[2], v[3]);
        const double2 m1 = make_double2(fma(c2, t2.x, fma(c1, t1.x, a.x)), fma(c2, t2.y, fma(c1, t1.y, a.y)));
        const double2 m2 = make_double2(fma(c1, t2.x, fma(c2, t1.x, a.x)), fma(c1, t2.y, fma(c2, t1.y, a.y)));
        const double2 n1 = make_double2(fma(s2, t4.x, __dmul_rn(s1, t3.x)), fma(s2, t4.y, __dmul_rn(s1, t3.y)));
        const double2 n2 = make_double2(fma(-s1, t4.x, __dmul_rn(s2, t3.x)), fma(-s1, t4.y, __dmul_rn(s2, t3.y)));
        v[0] = d_add(d_add(a, t1), t2);
        v[1] = make_double2(m1.x + n1.y, m1.y - n1.x);   // m1 - i n1
        v[4] = make_double2(m1.x - n1.y, m1.y + n1.x);
        v[2] = make_double2(m2.x + n2.y, m2.y - n2.x);
        v[3] = make_double2(m2.x - n2.y, m2.y + n2.x);
    }
};

// length-L forward DFT in registers, natural order in and out; w_L^e = tw[e * STEP], tw the
// w_N^{-e} table of the whole length N = L * STEP (in shared memory)
template <int L, int STEP> struct DFFT {
    static constexpr int F = (L % 4 == 0) ? 4 : (L % 2 == 0) ? 2 : (L % 3 == 0) ? 3 : (L % 5 == 0) ? 5 : 0;
    static_assert(F != 0, "transform length must factor into 2, 3, 5");
    static constexpr int M = L / F;
    __device__ static void run(double2 *x, const double2 *tw)
    {
        double2 s[F][M];
#pragma unroll
        for (int q = 0; q < F; ++q)
#pragma unroll
            for (int j = 0; j < M; ++j) s[q][j] = x[q + F * j];
#pragma unroll
        for (int q = 0; q < F; ++q) DFFT<M, STEP * F>::run(s[q], tw);
#pragma unroll
        for (int k = 0; k < M; ++k) {
            double2 v[F];
#pragma unroll
            for (int q = 0; q < F; ++q) v[q] = (q * k == 0) ? s[q][k] : d_mul(s[q][k], tw[q * k * STEP]);
            DBfly<F>::run(v);
#pragma unroll
            for (int r = 0; r < F; ++r) x[k + M * r] = v[r];
        }
    }
};
template <int STEP> struct DFFT<1, STEP> {
    __device__ static void run(double2 *, const double2 *) {}
};

// the shells per batch of the spectra kernels
constexpr int KB = 8;

template <int P1, int P2> struct Rows {
    static constexpr int P = P1 * P2, RS = P1 | 1, ROW = P2 * RS;   // double2 of one transform's rows
    __device__ static int at(int j) { return j % P2 * RS + j / P2; }

    // nf transforms: get(f, n) returns f(n) of transform f; their rows at buf + f ROW hold F afterwards, tw
    // the w_P^{-e} table.  All threads of the block take part; starts and ends with the block synchronised.
    template <class Get> __device__ static void run(int nf, const Get &get, double2 *buf, const double2 *tw)
    {
        __syncthreads();
        for (int e = threadIdx.x; e < nf * P1; e += blockDim.x) {
            const int f = e / P1, n1 = e - f * P1;
            double2 x[P2];
#pragma unroll
            for (int n2 = 0; n2 < P2; ++n2) x[n2] = get(f, n1 + P1 * n2);
            DFFT<P2, P1>::run(x, tw);
            double2 *row = buf + (size_t)f * ROW + n1;
#pragma unroll
            for (int k2 = 0; k2 < P2; ++k2) row[k2 * RS] = k2 == 0 ? x[k2] : d_mul(x[k2], tw[n1 * k2]);
        }
        __syncthreads();
        for (int e = threadIdx.x; e < nf * P2; e += blockDim.x) {
            double2 *row = buf + (size_t)(e / P2) * ROW + (e % P2) * RS;
            double2 x[P1];
#pragma unroll
            for (int n1 = 0; n1 < P1; ++n1) x[n1] = row[n1];
            DFFT<P1, P2>::run(x, tw);
#pragma unroll
            for (int k1 = 0; k1 < P1; ++k1) row[k1] = x[k1];
        }
        __syncthreads();
    }

    // the two shells of a pair at a frequency: z = Z(j), y = Z at its mirror
    __device__ static double2 first(double2 z, double2 y) { return make_double2(0.5 * (z.x + y.x), 0.5 * (z.y - y.y)); }
    __device__ static double2 second(double2 z, double2 y) { return make_double2(0.5 * (z.y + y.y), 0.5 * (y.x - z.x)); }
    // U(m) of the pair's two shells from the rows of its even transform (ze) and odd transform (zo)
    __device__ static void pair(int m, const double2 *ze, const double2 *zo, double2 &u, double2 &v)
    {
        const int j = m >> 1;
        const double2 *z = (m & 1) ? zo : ze;
        const double2 a = z[at(j)], b = z[at((m & 1) ? P - 1 - j : j == 0 ? 0 : P - j)];
        u = first(a, b);
        v = second(a, b);
    }
};

}  // namespace sfft
}  // namespace pftcc
