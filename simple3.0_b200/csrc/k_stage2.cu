// k_stage2.cu -- per-(particle, reference x shift) inverse transform of the m-domain
// spectrum, the correlation over all in-plane rotations, its argmax and the
// particle's running top-8; and the FP32 m-domain re-score of the final candidates.
//
// For one triple the spectrum X(m), m = 0..P (Hermitian over the full circle of
// N = 2P rotations) is packed into Z(j) = [X(j) + conj X(P-j)] + i [X(j) - conj X(P-j)]
// w_N^{-j}, j < P, whose length-P forward DFT z(l) = y(2l) + i y(2l+1) gives every
// rotation's correlation sum y(rot) = sum_{m<N} X(m) w_N^{-m rot} (the real-output
// half-length transform; the reference runs the equivalent FFTW c2r per shell in
// calc_corrs_over_k, simple_polarft_corrcalc.f90:1156).  The length-P DFT is one
// Cooley-Tukey split P = P1 * P2 evaluated entirely in registers with compile-time
// unrolled radix-2/3/4/5 butterflies:
//   pass A: for each residue class j1 < P1 a length-P2 DFT over j2 of Z(j1 + P1 j2),
//           times w_P^{-j1 l2}, into a thread-private shared-memory slab;
//   pass B: for each l2 < P2 a length-P1 DFT over j1 -> z(l2 + P2 l1).
// The search (k_stage2_fast; S2Split gives its splits) reads Z as stage 1 stored it, P planes of
// [col][row pair] (re, re, im, im); the FP32 re-score forms Z from X itself, processing classes j1 and P1 - j1 together so
// that every X element is computed once (Z(j) needs X(j) and X(P - j), which lie in the
// mirror class).
#include "pftcc_internal.cuh"
#include "spec_fft.cuh"

#include <algorithm>
#include <cstdio>
#include <cmath>

namespace pftcc {

constexpr int TW_MAX = 320;
struct TwTables {
    float2 wP[TW_MAX];   // w_P^{-e} = exp(-2 pi i e / P), e < P
    float2 wN[TW_MAX];   // w_N^{-e} = exp(-2 pi i e / N), e < P
    // the same w_P^{-e} = (c, s) as lane pairs for the two-lane transforms: (c, c), (s, s), (-s, -s)
    float2 pc[TW_MAX], ps[TW_MAX], pn[TW_MAX];
};

__device__ __forceinline__ float2 c_mul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 c_mi(float2 a) { return make_float2(a.y, -a.x); }   // -i * a

// forward radix butterflies (textbook radix-2/3/4/5 DFT formulas)
template <int F> struct Bfly;
template <> struct Bfly<2> {
    __device__ static void run(float2 *v) { const float2 a = v[0], b = v[1]; v[0] = c_add(a, b); v[1] = c_sub(a, b); }
};
template <> struct Bfly<4> {
    __device__ static void run(float2 *v)
    {
        const float2 t0 = c_add(v[0], v[2]), t1 = c_sub(v[0], v[2]);
        const float2 t2 = c_add(v[1], v[3]), t3 = c_mi(c_sub(v[1], v[3]));
        v[0] = c_add(t0, t2);
        v[2] = c_sub(t0, t2);
        v[1] = c_add(t1, t3);
        v[3] = c_sub(t1, t3);
    }
};
template <> struct Bfly<3> {
    __device__ static void run(float2 *v)
    {
        const float s3 = 0.86602540378443865f;   // sin(2 pi / 3)
        const float2 a = v[0], t1 = c_add(v[1], v[2]);
        const float2 t2 = make_float2(a.x - 0.5f * t1.x, a.y - 0.5f * t1.y);
        const float2 d = c_sub(v[1], v[2]);
        const float2 t3 = make_float2(s3 * d.y, -s3 * d.x);   // -i sin(2pi/3) (b - c)
        v[0] = c_add(a, t1);
        v[1] = c_add(t2, t3);
        v[2] = c_sub(t2, t3);
    }
};
template <> struct Bfly<5> {
    __device__ static void run(float2 *v)
    {
        const float c1 = 0.30901699437494742f, c2 = -0.80901699437494742f;   // cos(2pi/5), cos(4pi/5)
        const float s1 = 0.95105651629515357f, s2 = 0.58778525229247313f;    // sin(2pi/5), sin(4pi/5)
        const float2 a = v[0];
        const float2 t1 = c_add(v[1], v[4]), t2 = c_add(v[2], v[3]);
        const float2 t3 = c_sub(v[1], v[4]), t4 = c_sub(v[2], v[3]);
        const float2 m1 = make_float2(a.x + c1 * t1.x + c2 * t2.x, a.y + c1 * t1.y + c2 * t2.y);
        const float2 m2 = make_float2(a.x + c2 * t1.x + c1 * t2.x, a.y + c2 * t1.y + c1 * t2.y);
        const float2 n1 = make_float2(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y);
        const float2 n2 = make_float2(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y);
        v[0] = make_float2(a.x + t1.x + t2.x, a.y + t1.y + t2.y);
        v[1] = c_add(m1, c_mi(n1));
        v[4] = c_sub(m1, c_mi(n1));
        v[2] = c_add(m2, c_mi(n2));
        v[3] = c_sub(m2, c_mi(n2));
    }
};

// length-L forward DFT in registers, natural order in and out; w_L^e = wP[e * STEP]
template <int L, int STEP> struct SFFT {
    static constexpr int F = (L % 4 == 0) ? 4 : (L % 2 == 0) ? 2 : (L % 3 == 0) ? 3 : (L % 5 == 0) ? 5 : 0;
    static_assert(F != 0, "transform length must factor into 2, 3, 5");
    static constexpr int M = L / F;
    __device__ static void run(float2 *x, const TwTables &tw)
    {
        float2 s[F][M];
#pragma unroll
        for (int q = 0; q < F; ++q)
#pragma unroll
            for (int j = 0; j < M; ++j) s[q][j] = x[q + F * j];
#pragma unroll
        for (int q = 0; q < F; ++q) SFFT<M, STEP * F>::run(s[q], tw);
#pragma unroll
        for (int k = 0; k < M; ++k) {
            float2 v[F];
#pragma unroll
            for (int q = 0; q < F; ++q) v[q] = (q * k == 0) ? s[q][k] : c_mul(s[q][k], tw.wP[q * k * STEP]);
            Bfly<F>::run(v);
#pragma unroll
            for (int r = 0; r < F; ++r) x[k + M * r] = v[r];
        }
    }
};
template <int STEP> struct SFFT<1, STEP> {
    __device__ static void run(float2 *, const TwTables &) {}
};

// ---------------------------------------------------------------------------------------
// Two transforms at once with the packed two-lane FP32 instructions of sm_100 (one
// add / mul / fma on a register pair): C2 holds two complex numbers as r = (re_a, re_b),
// i = (im_a, im_b), so a butterfly of two independent transforms costs half the
// instructions of two scalar ones.  Each lane is rounded exactly as the scalar operation.
struct C2 { float2 r, i; };
__device__ __forceinline__ float2 f2_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 f2_sub(float2 a, float2 b)
{
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<unsigned long long *>(&a)),
        "l"(*reinterpret_cast<unsigned long long *>(&b)));
    return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float2 f2_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 f2_s(float s) { return make_float2(s, s); }
__device__ __forceinline__ C2 p_add(const C2 &a, const C2 &b) { return {f2_add(a.r, b.r), f2_add(a.i, b.i)}; }
__device__ __forceinline__ C2 p_sub(const C2 &a, const C2 &b) { return {f2_sub(a.r, b.r), f2_sub(a.i, b.i)}; }
// a * (c + i s) with c, s and -s given as lane pairs
__device__ __forceinline__ C2 p_twid(const C2 &a, float2 c, float2 s, float2 ns)
{
    return {f2_fma(a.r, c, f2_mul(a.i, ns)), f2_fma(a.r, s, f2_mul(a.i, c))};
}
__device__ __forceinline__ float max3f(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// the radix-2/3/4/5 butterflies above, on lane pairs (-i a = (a.i, -a.r) is folded into
// the adds that follow it)
template <int F> struct PBfly;
template <> struct PBfly<2> {
    __device__ static void run(C2 *v) { const C2 a = v[0], b = v[1]; v[0] = p_add(a, b); v[1] = p_sub(a, b); }
};
template <> struct PBfly<4> {
    __device__ static void run(C2 *v)
    {
        const C2 t0 = p_add(v[0], v[2]), t1 = p_sub(v[0], v[2]);
        const C2 t2 = p_add(v[1], v[3]), d = p_sub(v[1], v[3]);
        v[0] = p_add(t0, t2);
        v[2] = p_sub(t0, t2);
        v[1] = {f2_add(t1.r, d.i), f2_sub(t1.i, d.r)};
        v[3] = {f2_sub(t1.r, d.i), f2_add(t1.i, d.r)};
    }
};
template <> struct PBfly<3> {
    __device__ static void run(C2 *v)
    {
        const float s3 = 0.86602540378443865f;
        const C2 a = v[0], t1 = p_add(v[1], v[2]), d = p_sub(v[1], v[2]);
        const C2 t2 = {f2_fma(t1.r, f2_s(-0.5f), a.r), f2_fma(t1.i, f2_s(-0.5f), a.i)};
        v[0] = p_add(a, t1);
        v[1] = {f2_fma(d.i, f2_s(s3), t2.r), f2_fma(d.r, f2_s(-s3), t2.i)};
        v[2] = {f2_fma(d.i, f2_s(-s3), t2.r), f2_fma(d.r, f2_s(s3), t2.i)};
    }
};
template <> struct PBfly<5> {
    __device__ static void run(C2 *v)
    {
        const float c1 = 0.30901699437494742f, c2 = -0.80901699437494742f;
        const float s1 = 0.95105651629515357f, s2 = 0.58778525229247313f;
        const C2 a = v[0];
        const C2 t1 = p_add(v[1], v[4]), t2 = p_add(v[2], v[3]);
        const C2 t3 = p_sub(v[1], v[4]), t4 = p_sub(v[2], v[3]);
        const C2 m1 = {f2_fma(t2.r, f2_s(c2), f2_fma(t1.r, f2_s(c1), a.r)), f2_fma(t2.i, f2_s(c2), f2_fma(t1.i, f2_s(c1), a.i))};
        const C2 m2 = {f2_fma(t2.r, f2_s(c1), f2_fma(t1.r, f2_s(c2), a.r)), f2_fma(t2.i, f2_s(c1), f2_fma(t1.i, f2_s(c2), a.i))};
        const C2 n1 = {f2_fma(t4.r, f2_s(s2), f2_mul(t3.r, f2_s(s1))), f2_fma(t4.i, f2_s(s2), f2_mul(t3.i, f2_s(s1)))};
        const C2 n2 = {f2_fma(t4.r, f2_s(-s1), f2_mul(t3.r, f2_s(s2))), f2_fma(t4.i, f2_s(-s1), f2_mul(t3.i, f2_s(s2)))};
        v[0] = p_add(p_add(a, t1), t2);
        v[1] = {f2_add(m1.r, n1.i), f2_sub(m1.i, n1.r)};
        v[4] = {f2_sub(m1.r, n1.i), f2_add(m1.i, n1.r)};
        v[2] = {f2_add(m2.r, n2.i), f2_sub(m2.i, n2.r)};
        v[3] = {f2_sub(m2.r, n2.i), f2_add(m2.i, n2.r)};
    }
};

__host__ __device__ constexpr int gcd_c(int a, int b) { return b == 0 ? a : gcd_c(b, a % b); }
// the index o < F M with o = r (mod F) and o = k (mod M), gcd(F, M) = 1
__host__ __device__ constexpr int crt_c(int r, int k, int F, int M)
{
    int o = k;
    while (o % F != r) o += M;
    return o;
}

// two length-L forward DFTs, one per lane, natural order in and out (SFFT's recursion).
// When the radix F and the rest M = L / F are coprime (15 = 3 x 5, 12 = 4 x 3, 20 = 4 x 5)
// the Good-Thomas prime-factor mapping needs no twiddles between the two stages: input
// x((M q + F j) mod L) -> the M-point DFTs over j, the F-point butterflies over q, output
// index o with o = r (mod F) and o = k (mod M); otherwise the Cooley-Tukey split with the
// twiddles w_L^{qk}.
template <int L, int STEP> struct PFFT {
    static constexpr int F = SFFT<L, STEP>::F;
    static constexpr int M = L / F;
    static constexpr bool PFA = M > 1 && gcd_c(F, M) == 1;
    __device__ static void run(C2 *x, const TwTables &tw)
    {
        C2 s[F][M];
#pragma unroll
        for (int q = 0; q < F; ++q)
#pragma unroll
            for (int j = 0; j < M; ++j) s[q][j] = PFA ? x[(M * q + F * j) % L] : x[q + F * j];
#pragma unroll
        for (int q = 0; q < F; ++q) PFFT<M, STEP * F>::run(s[q], tw);
#pragma unroll
        for (int k = 0; k < M; ++k) {
            C2 v[F];
#pragma unroll
            for (int q = 0; q < F; ++q) {
                const int e = q * k * STEP;
                v[q] = (PFA || q * k == 0) ? s[q][k] : p_twid(s[q][k], tw.pc[e], tw.ps[e], tw.pn[e]);
            }
            PBfly<F>::run(v);
#pragma unroll
            for (int r = 0; r < F; ++r) x[PFA ? crt_c(r, k, F, M) : k + M * r] = v[r];
        }
    }
};
template <int STEP> struct PFFT<1, STEP> {
    __device__ static void run(C2 *, const TwTables &) {}
};

// ---------------------------------------------------------------------------------------
struct S2Fast {
    int nshifts, N, nrs_total, nwaves;
    float escale;   // the Euclidean objective: the transform's scale 1/(2N) (the factors are additive)
};

// (c, id) ranks above (c2, id2): larger correlation, then lower id
__device__ __forceinline__ bool ranks_above(float c, int id, float c2, int id2) { return c > c2 || (c == c2 && id < id2); }

// The search's split P = P1 x P2: pass A takes the P1 classes, a length-P2 DFT each, pass B the P2
// blocks, a length-P1 DFT each, one class or block at a time per role (warp) of a row group.
//   coprime factors (180 = 9 x 20, 300 = 12 x 25): the Good-Thomas mapping, class c holding the
//     inputs j = P2 c + P1 j2 (mod P) and block l2 giving the outputs l = l1 (mod P1) = l2 (mod P2):
//     no twiddles between the passes;
//   64 = 8 x 8: class c holds j = c + P1 j2, twiddles w_P^{-c l2}, block l2 the outputs l2 + P2 l1.
// Rotations 2l + b and 2l + b + P share their normalising factor, that is outputs l and l + P/2:
// at P = 180 blocks l2 and l2 + 10 (the same l1), at 64 and 300 the outputs l1 and l1 + P1/2 of a
// block.  A factor group q is the block(s) that use one set of DV factors, DQ its stride in memory
// (a multiple of four, for 16-byte loads): factor (l1, b) of group q at q DQ + 2 l1 + b.
// ROLES warps share 32 row pairs; MB blocks per SM.
template <int P> struct S2Split;
template <> struct S2Split<64> { static constexpr int P1 = 8, P2 = 8, PFA = 0, NQ = 8, BPQ = 1, DV = 8, DQ = 8, ROLES = 8, MB = 4; };
template <> struct S2Split<180> { static constexpr int P1 = 9, P2 = 20, PFA = 1, NQ = 10, BPQ = 2, DV = 18, DQ = 20, ROLES = 10, MB = 2; };
template <> struct S2Split<300> { static constexpr int P1 = 12, P2 = 25, PFA = 1, NQ = 25, BPQ = 1, DV = 12, DQ = 12, ROLES = 13, MB = 1; };

// the normalising factors of the length: floats per (reference, particle)
template <int P> __host__ __device__ constexpr int s2_dlen() { return S2Split<P>::NQ * S2Split<P>::DQ; }

// output index l of block l2 at l1
template <int P> __device__ __forceinline__ int s2_out(int l1, int l2)
{
    using S = S2Split<P>;
    if constexpr (S::PFA) {
        constexpr int E1 = crt_c(1, 0, S::P1, S::P2), E2 = crt_c(0, 1, S::P1, S::P2);   // 1 and 0 modulo (P1, P2), and 0 and 1
        return (E1 * l1 + E2 * l2) % P;
    } else {
        return l2 + S::P2 * l1;
    }
}

// What bounds it: the DRAM read of Z (1,440 B a triple at P = 180), with the transforms' FP32 pipe time
// at half of that.  A block takes one particle column, 32 row pairs (64 rows) at a time: lane = row
// pair, whose two rows go through the two lanes of the f32x2 instructions, so that a 16-byte load of Z
// (stage 1 stores re, re, im, im of a row pair) is an operand as it comes, and warp = role.  Per
// iteration: pass A from global memory into the slab [P2 blocks][P1][32 lanes] of 16 bytes, a barrier,
// pass B from the slab to the maximum over the rotations, a barrier.  The small per-role state lets
// 20 warps share an SM where one thread per class pair and row needed 254 registers and 8 warps; the
// coprime splits have no twiddles, the row pairs no packing moves, and the factors are read once for
// both rotations that share them.  Only what the caller uses is computed: with a re-score to follow
// (ROT false) a candidate is its row, so the winning rotation is not searched for.
// The last role keeps the block's running top 8 per lane in shared memory, fed a barrier later.
// Measured, ms before (a column per block, two threads per row, 128 rows, class pairs in the lanes) and
// now: 500 references x 81 shifts x 20,000 particles, P = 180: 395, 256 (4.6 TB/s of Z); 100 references
// x 1000 particles, P = 64: 0.159, 0.028; 300 x 5130 pairs' groups, P = 300: 1.26, 0.59.  At P = 180,
// 3.2e7 triples: 10 roles 9.5 ms (4.9 TB/s), 9 roles 10.5, 5 roles 10.0, 12 roles 13.2 (spills), the
// next rows prefetched into L2 9.8; P = 300, 2.5e6 triples: 13 roles 1.65, 12 1.68, 9 2.05, 8 1.93;
// P = 64, 5e6 triples: 8 roles x 4 blocks 0.56, x 3 0.64, x 5 0.72, 4 roles x 6 0.82.
template <int P, bool ROT, bool WRITE, bool EU>
__global__ void __launch_bounds__(32 * S2Split<P>::ROLES, S2Split<P>::MB)
k_stage2_fast(S2Fast sp, const __grid_constant__ TwTables tw, const S2Wave *__restrict__ waves, float2 *__restrict__ cand,
              float *__restrict__ ccall, const int *__restrict__ perm)
{
    using S = S2Split<P>;
    constexpr int P1 = S::P1, P2 = S::P2, NR = S::ROLES, DLEN = s2_dlen<P>();
    // this block's wave (the last one starting at or before it) and column within it
    int lo = 0, hi = sp.nwaves - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&waves[mid].blk0) <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const S2Wave *W = waves + lo;
    const int cl = (int)blockIdx.x - __ldg(&W->blk0);
    const float4 *X = reinterpret_cast<const float4 *>(__ldg(reinterpret_cast<const unsigned long long *>(&W->X)));
    const float *Dinv = reinterpret_cast<const float *>(__ldg(reinterpret_cast<const unsigned long long *>(&W->D)));
    const int w_rows = __ldg(&W->rows), w_row0 = __ldg(&W->row0), w_rofs = __ldg(&W->rofs);
    const int w_xrows = __ldg(&W->xrows), w_xcols = __ldg(&W->xcols), w_col0 = __ldg(&W->col0);
    const int w_zc0 = __ldg(&W->zc0), w_r0 = __ldg(&W->r0), w_dcols = __ldg(&W->dcols);
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, role = threadIdx.x >> 5;
    float4 *slab = smem4 + lane;                                                  // [P2 P1][32]
    float2 *xfer = reinterpret_cast<float2 *>(smem4 + P * 32);                    // [NR][32] the roles' maxima of the row pairs
    int2 *xrot = reinterpret_cast<int2 *>(xfer + NR * 32);                        // [NR][32] their rotations (ROT)
    float *kc = reinterpret_cast<float *>(xrot + (ROT ? NR * 32 : 0));            // [8][32] each lane's running top 8
    int *ki = reinterpret_cast<int *>(kc + 8 * 32);
    if (role == NR - 1)
        for (int k = 0; k < 8; ++k) { kc[k * 32 + lane] = -INFINITY; ki[k * 32 + lane] = 0x7fffffff; }
    // Z offsets in float4 units fit 32 bits (the launcher checks P xcols xrows < 2^32)
    const uint32_t plane = (uint32_t)w_xcols * (uint32_t)(w_xrows >> 1);
    const int pr0 = w_rofs >> 1, pr1 = (w_rofs + w_rows - 1) >> 1;                // the wave's row pairs of Z
    const float4 *Xc = X + (size_t)(w_zc0 + cl) * (w_xrows >> 1);
    const float *Dc = Dinv + (size_t)cl * DLEN;
    auto merge = [&](int base) {   // the row pairs base + lane, after their pass B
        const int r0 = 2 * (base + lane) - w_rofs;
        float2 b = make_float2(-INFINITY, -INFINITY);
        int2 br = make_int2(0, 0);
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const float2 v = xfer[r * 32 + lane];
            if constexpr (ROT) {
                const int2 o = xrot[r * 32 + lane];
                if (v.x > b.x || (v.x == b.x && o.x < br.x)) { b.x = v.x; br.x = o.x; }
                if (v.y > b.y || (v.y == b.y && o.y < br.y)) { b.y = v.y; br.y = o.y; }
            } else {
                b.x = fmaxf(b.x, v.x);
                b.y = fmaxf(b.y, v.y);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float c = i ? b.y : b.x;
            const int row = r0 + i;
            if (row < 0 || row >= w_rows || c == -INFINITY || c < kc[7 * 32 + lane]) continue;
            int id = (w_row0 + row) * sp.N + (ROT ? (i ? br.y : br.x) : 0);
            for (int k = 0; k < 8; ++k) {
                const float tc = kc[k * 32 + lane];
                const int ti = ki[k * 32 + lane];
                if (ranks_above(c, id, tc, ti)) { kc[k * 32 + lane] = c; ki[k * 32 + lane] = id; c = tc; id = ti; }
            }
        }
    };
#pragma unroll 1
    for (int base = pr0; base <= pr1; base += 32) {
        const int pr = min(base + lane, pr1);   // lanes past the end repeat the last pair
#pragma unroll 1
        for (int c = role; c < P1; c += NR) {
            const float4 *xr = Xc + pr;
            C2 z[P2];
#pragma unroll
            for (int j2 = 0; j2 < P2; ++j2) {
                int j = S::PFA ? P2 * c + P1 * j2 : c + P1 * j2;
                if (S::PFA && j >= P) j -= P;
                asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(z[j2].r.x), "=f"(z[j2].r.y), "=f"(z[j2].i.x), "=f"(z[j2].i.y)
                             : "l"(xr + (uint32_t)j * plane));
            }
            PFFT<P2, P1>::run(z, tw);
#pragma unroll
            for (int l2 = 0; l2 < P2; ++l2) {
                C2 o = z[l2];
                if (!S::PFA && l2 > 0) o = p_twid(o, tw.pc[c * l2], tw.ps[c * l2], tw.pn[c * l2]);
                slab[(l2 * P1 + c) * 32] = make_float4(o.r.x, o.r.y, o.i.x, o.i.y);
            }
        }
        if (role == NR - 1 && base > pr0) merge(base - 32);
        __syncthreads();
        const int row0 = min(max(2 * pr - w_rofs, 0), w_rows - 1), row1 = min(2 * pr + 1 - w_rofs, w_rows - 1);
        const float *D0 = Dc + (size_t)((w_row0 + row0) / sp.nshifts - w_r0) * w_dcols * DLEN;
        const float *D1 = Dc + (size_t)((w_row0 + row1) / sp.nshifts - w_r0) * w_dcols * DLEN;
        float *cc0 = nullptr, *cc1 = nullptr;
        if constexpr (WRITE) {
            const int r0 = 2 * (base + lane) - w_rofs;
            float *col = ccall + ((size_t)perm[w_col0 + cl] * sp.nrs_total + w_row0) * sp.N;
            if (r0 >= 0 && r0 < w_rows) cc0 = col + (size_t)r0 * sp.N;
            if (r0 + 1 < w_rows) cc1 = col + (size_t)(r0 + 1) * sp.N;
        }
        float2 best = make_float2(-INFINITY, -INFINITY);
        int2 brot = make_int2(0x7fffffff, 0x7fffffff);
#pragma unroll 1
        for (int q = role; q < S::NQ; q += NR) {
            float4 d0[S::DQ / 4], d1[S::DQ / 4];   // issued ahead of the transforms
#pragma unroll
            for (int e = 0; e < S::DQ / 4; ++e) {
                d0[e] = __ldg(reinterpret_cast<const float4 *>(D0 + q * S::DQ) + e);
                d1[e] = __ldg(reinterpret_cast<const float4 *>(D1 + q * S::DQ) + e);
            }
            const float *f0 = reinterpret_cast<const float *>(d0), *f1 = reinterpret_cast<const float *>(d1);
#pragma unroll
            for (int h = 0; h < S::BPQ; ++h) {
                const int l2 = q + S::NQ * h;
                C2 v[P1];
#pragma unroll
                for (int c = 0; c < P1; ++c) {
                    const float4 a = slab[(l2 * P1 + c) * 32];
                    v[c] = {make_float2(a.x, a.y), make_float2(a.z, a.w)};
                }
                PFFT<P1, P2>::run(v, tw);
#pragma unroll
                for (int l1 = 0; l1 < P1; ++l1) {
                    constexpr int HALF = S::BPQ == 2 ? P1 : P1 / 2;
                    const int e = 2 * (l1 % HALF);
                    const float a0 = EU ? fmaf(v[l1].r.x, sp.escale, f0[e]) : v[l1].r.x * f0[e];
                    const float a1 = EU ? fmaf(v[l1].i.x, sp.escale, f0[e + 1]) : v[l1].i.x * f0[e + 1];
                    const float b0 = EU ? fmaf(v[l1].r.y, sp.escale, f1[e]) : v[l1].r.y * f1[e];
                    const float b1 = EU ? fmaf(v[l1].i.y, sp.escale, f1[e + 1]) : v[l1].i.y * f1[e + 1];
                    if constexpr (ROT) {
                        const int rot = 2 * s2_out<P>(l1, l2);
                        if (a0 > best.x || (a0 == best.x && rot < brot.x)) { best.x = a0; brot.x = rot; }
                        if (a1 > best.x || (a1 == best.x && rot + 1 < brot.x)) { best.x = a1; brot.x = rot + 1; }
                        if (b0 > best.y || (b0 == best.y && rot < brot.y)) { best.y = b0; brot.y = rot; }
                        if (b1 > best.y || (b1 == best.y && rot + 1 < brot.y)) { best.y = b1; brot.y = rot + 1; }
                        if constexpr (WRITE) {
                            if (cc0) *reinterpret_cast<float2 *>(cc0 + rot) = make_float2(a0, a1);
                            if (cc1) *reinterpret_cast<float2 *>(cc1 + rot) = make_float2(b0, b1);
                        }
                    } else {
                        best.x = max3f(best.x, a0, a1);
                        best.y = max3f(best.y, b0, b1);
                    }
                }
            }
        }
        xfer[role * 32 + lane] = best;
        if constexpr (ROT) xrot[role * 32 + lane] = brot;
        __syncthreads();
    }
    if (role != NR - 1) return;
    merge(pr0 + (pr1 - pr0) / 32 * 32);
    // the lanes' lists and the particle's running top 8, whose slots follow them (lowest id among
    // equal correlations)
    __syncwarp();
    float2 *cp = cand + (size_t)(w_col0 + cl) * 8;
    float pc = -INFINITY;
    int pid = 0x7fffffff;
    if (lane < 8) {
        const float2 c = cp[lane];
        pc = c.x;
        pid = __float_as_int(c.y);
    }
    float keep_c = -INFINITY;
    int keep_i = -1, head = 0;   // each lane's list is sorted: its head is its best
    for (int it = 0; it < 8; ++it) {
        float bc = head < 8 ? kc[head * 32 + lane] : -INFINITY;
        int bi = head < 8 ? ki[head * 32 + lane] : 0x7fffffff;
        if (bc == -INFINITY) bi = 0x7fffffff;
        const bool old = pc != -INFINITY && ranks_above(pc, pid, bc, bi);
        if (old) { bc = pc; bi = pid; }
        float mc = bc;
        int mi = bi;
        for (int o = 16; o > 0; o >>= 1) {
            const float oc = __shfl_xor_sync(0xffffffffu, mc, o);
            const int oi = __shfl_xor_sync(0xffffffffu, mi, o);
            if (ranks_above(oc, oi, mc, mi)) { mc = oc; mi = oi; }
        }
        if (lane == it) { keep_c = mc; keep_i = mc == -INFINITY ? -1 : mi; }
        if (mc != -INFINITY && bc == mc && bi == mi) {   // ids are distinct: one lane's
            if (old) pc = -INFINITY; else ++head;
        }
    }
    if (lane < 8) cp[lane] = make_float2(keep_c, __int_as_float(keep_i));
}

// ---------------------------------------------------------------------------------------
// FP32 m-domain re-score of the top-ntop candidates of each particle (particle frame):
// X(m) = 4 sum_k UA[m][rs][k] conj(UB[m][col][k]) from the FP32 spectra, the FP64
// normaliser from the |ref|^2 and CTF^2 spectra, the same transform and argmax.  One block
// per particle, its ntop <= 8 candidates in four phases:
//   A  Y(c, j) = (wgt_j / P) sum_k conj(RU[r_c][j][k]) CV[col][j][k] in FP64, eight lanes per j;
//   B  D(c, rho) from Y by the length-P/2 FP64 transform of the packed half spectrum (the
//      normaliser's k_norm_fft, split H1 x H2 = P/2), stored as 1/sqrt(D * sqsum_ptcl);
//   C  X(c, m) in FP32, eight lanes per m;
//   D  the transforms and maxima, a thread per (candidate, class) and (candidate, block), then the
//      particle's best (lowest id among equal correlations).
// What bounds it: the candidates' spectra from L2 (16 B x J Ks + 8 B x M Ks each, 2.3 MB a particle at
// P = 300, Ks = 59).  5130 particles, P = 300: before, with one candidate's loads in flight at a time and
// the transforms in one warp, 3.65 ms; now 1.4 (0.72 of 2.07 for 2500 particles; 0.43 of 0.87 for 3000 at
// P = 180; 0.064 of 0.076 for 1000 at P = 64).  More of the candidates' loads unrolled: 0.77 at P = 300.
template <int P> struct HalfSplit;
template <> struct HalfSplit<64> { static constexpr int H1 = 8, H2 = 4; };
template <> struct HalfSplit<180> { static constexpr int H1 = 10, H2 = 9; };
template <> struct HalfSplit<300> { static constexpr int H1 = 15, H2 = 10; };
constexpr int RS_MAX = 8;     // candidates per particle
constexpr int RS_THREADS = 256;

// shared memory: the FP64 tables, one region for Y and its transform's rows (phases A and B) and then X and
// the transforms' slabs (C and D), the FP32 tables, the factors, the blocks' maxima.  59 KB at P = 300: three
// blocks on an SM, which is what hides the latency of the candidates' loads (with two, 18 of 24 cycles
// between a warp's instructions went to it).
template <int P1, int P2> struct RescoreSmem {
    static constexpr int P = P1 * P2, J = P / 2 + 1, H = P / 2, M = P + 1, H1 = HalfSplit<P>::H1, H2 = HalfSplit<P>::H2;
    static constexpr size_t rows = sizeof(double2) * ((size_t)RS_MAX * J + (size_t)RS_MAX * H2 * (H1 + 1));
    static constexpr size_t slabs = sizeof(float2) * ((size_t)RS_MAX * M + (size_t)RS_MAX * (P | 1));
    static constexpr size_t region = ((rows > slabs ? rows : slabs) + 15) / 16 * 16;
    static constexpr size_t bytes = sizeof(double2) * 2 * H + region + sizeof(float2) * 2 * P + sizeof(float) * RS_MAX * P +
                                    (sizeof(float) + sizeof(int)) * RS_MAX * P2;
};

// KL: shells of a lane, 8 KL >= Ks
template <int P1, int P2, bool EU, int KL>
__global__ void __launch_bounds__(RS_THREADS, P1 * P2 <= 64 ? 4 : 3) k_rescore_md(int ncols, int ntop, int Ks, int N, int nshifts,
                                                           int has_shifts, const TwTables tw,
                                                           const float2 *__restrict__ UA, int rows_pad,
                                                           const float2 *__restrict__ UB, int cols_pad,
                                                           const double2 *__restrict__ RU,
                                                           const double2 *__restrict__ CV, const float *__restrict__ sqp,
                                                           const float2 *__restrict__ cand, const int *__restrict__ perm,
                                                           int c0, pftcc_best *__restrict__ out)
{
    constexpr int P = P1 * P2, J = P / 2 + 1, H = P / 2, M = P + 1;
    constexpr int H1 = HalfSplit<P>::H1, H2 = HalfSplit<P>::H2;
    extern __shared__ float4 smem4[];
    double2 *tw_h = reinterpret_cast<double2 *>(smem4);            // [H] w_{P/2}^{-e}
    double2 *wp = tw_h + H;                                         // [H] w_P^{+e}
    unsigned char *region = reinterpret_cast<unsigned char *>(wp + H);
    double2 *Ys = reinterpret_cast<double2 *>(region);              // [RS_MAX][J]
    double2 *buf = Ys + RS_MAX * J;                                 // [RS_MAX][H2][H1 + 1]
    float2 *Xs = reinterpret_cast<float2 *>(region);                // [RS_MAX][M], after Ys and buf
    float2 *slab = Xs + RS_MAX * M;                                 // [RS_MAX][P | 1]
    float2 *wp_s = reinterpret_cast<float2 *>(region + RescoreSmem<P1, P2>::region);   // [P] w_P^{-e}
    float2 *wn_s = wp_s + P;                                        // [P] w_N^{-e}
    float *Ds = reinterpret_cast<float *>(wn_s + P);                // [RS_MAX][P]
    float *pbest = Ds + RS_MAX * P;                                 // [RS_MAX][P2] the blocks' maxima
    int *prot = reinterpret_cast<int *>(pbest + RS_MAX * P2);       // [RS_MAX][P2] and their rotations
    __shared__ int rs_s[RS_MAX];
    __shared__ float bc_s[RS_MAX];
    __shared__ int bi_s[RS_MAX];
    const int cl = c0 + blockIdx.x;
    if (cl >= c0 + ncols) return;
    const int t = threadIdx.x;
    const int nc = min(ntop, RS_MAX);
    if (t < nc) {
        const int id = __float_as_int(cand[(size_t)cl * 8 + t].y);
        rs_s[t] = id >= 0 ? id / N : -1;
    }
    for (int e = t; e < H; e += blockDim.x) {
        double sn, cs;
        sincospi(-2.0 * e / H, &sn, &cs);
        tw_h[e] = make_double2(cs, sn);
        sincospi(2.0 * e / P, &sn, &cs);
        wp[e] = make_double2(cs, sn);
    }
    for (int e = t; e < P; e += blockDim.x) { wp_s[e] = tw.wP[e]; wn_s[e] = tw.wN[e]; }
    __syncthreads();
    // A: Y, eight lanes per j over the shells (coalesced reads) and CPT candidates, GP at a time: the
    // particle's spectrum is read once for them and the loads of UA_ GP candidates are in flight together (an
    // empty candidate reads row 0 and is dropped at the end).  With few shells a lane has few loads: then four
    // candidates a task, all in flight.  The loop runs the same
    // trips in every warp so that the shuffles see all lanes
    constexpr int NGRP = RS_THREADS / 8, CPT = KL <= 3 ? 4 : 8, GP = KL <= 3 ? 4 : 1,
                  UA_ = KL <= 3 ? 1 : 2, UC = KL <= 3 ? 1 : 4;   // unrolled groups of GP: loads in flight
    const int l8 = t & 7, grp = t >> 3, nq = (nc + CPT - 1) / CPT;
    for (int base = 0; base < J * nq; base += NGRP) {
        const int e = min(base + grp, J * nq - 1), j = e / nq, c0 = CPT * (e - j * nq);
        double2 v[KL];
        const double2 *cv = CV + ((size_t)cl * J + j) * Ks;
#pragma unroll
        for (int i = 0; i < KL; ++i) v[i] = l8 + 8 * i < Ks ? cv[l8 + 8 * i] : make_double2(0.0, 0.0);
#pragma unroll UA_
        for (int cg = c0; cg < c0 + CPT; cg += GP) {
            double yr[GP], yi[GP];
#pragma unroll
            for (int u = 0; u < GP; ++u) {
                const int rs = cg + u < nc ? rs_s[cg + u] : -1;
                const double2 *ru = RU + ((size_t)(max(rs, 0) / nshifts) * J + j) * Ks;
                yr[u] = yi[u] = 0.0;
#pragma unroll
                for (int i = 0; i < KL; ++i) {
                    if (l8 + 8 * i >= Ks) continue;
                    const double2 r = ru[l8 + 8 * i];
                    yr[u] = fma(r.x, v[i].x, fma(r.y, v[i].y, yr[u]));
                    yi[u] = fma(r.x, v[i].y, fma(-r.y, v[i].x, yi[u]));
                }
            }
#pragma unroll
            for (int u = 0; u < GP; ++u) {
#pragma unroll
                for (int o = 4; o; o >>= 1) {
                    yr[u] += __shfl_xor_sync(0xffffffffu, yr[u], o);
                    yi[u] += __shfl_xor_sync(0xffffffffu, yi[u], o);
                }
                if (base + grp < J * nq && l8 == u && cg + u < nc) {
                    const double wgt = ((j == 0 || 2 * j == P) ? 1.0 : 2.0) / P;
                    Ys[(cg + u) * J + j] = make_double2(wgt * yr[u], wgt * yi[u]);
                }
            }
        }
    }
    __syncthreads();
    // B: D, pass 1 (c, n1) then pass 2 (c, k2)
    for (int e = t; e < nc * H1; e += blockDim.x) {
        const int c = e / H1, n1 = e - c * H1;
        const double2 *y = Ys + c * J;
        double2 x[H2];
#pragma unroll
        for (int n2 = 0; n2 < H2; ++n2) {
            const int j = n1 + H1 * n2;
            double2 hj, hh;
            if (j == 0) {
                hj = make_double2(y[0].x, 0.0);
                hh = make_double2(y[H].x, 0.0);
            } else {
                const double2 a = y[j], b = y[H - j];
                hj = make_double2(0.5 * a.x, 0.5 * a.y);
                hh = make_double2(0.5 * b.x, -0.5 * b.y);
            }
            const double2 ev = sfft::d_add(hj, hh), od = sfft::d_mul(sfft::d_sub(hj, hh), wp[j]);
            x[n2] = make_double2(ev.x - od.y, -(ev.y + od.x));   // conj(ev + i od)
        }
        sfft::DFFT<H2, H1>::run(x, tw_h);
        double2 *row = buf + (size_t)c * H2 * (H1 + 1) + n1;
#pragma unroll
        for (int k2 = 0; k2 < H2; ++k2)
            row[k2 * (H1 + 1)] = (k2 == 0 || n1 == 0) ? x[k2] : sfft::d_mul(x[k2], tw_h[n1 * k2]);
    }
    __syncthreads();
    const double sq = (double)sqp[cl];
    for (int e = t; e < nc * H2; e += blockDim.x) {
        const int c = e / H2, k2 = e - c * H2;
        const double2 *row = buf + ((size_t)c * H2 + k2) * (H1 + 1);
        double2 x[H1];
#pragma unroll
        for (int n1 = 0; n1 < H1; ++n1) x[n1] = row[n1];
        sfft::DFFT<H1, H2>::run(x, tw_h);
#pragma unroll
        for (int k1 = 0; k1 < H1; ++k1) {
            const int l = k2 + H2 * k1;
            if constexpr (EU) {   // -(D + sum_k w_k |ptcl_k|^2) / 2
                Ds[c * P + 2 * l] = (float)(-0.5 * (x[k1].x + sq));
                Ds[c * P + 2 * l + 1] = (float)(-0.5 * (-x[k1].y + sq));
            } else {
                Ds[c * P + 2 * l] = (float)(1.0 / sqrt(x[k1].x * sq));
                Ds[c * P + 2 * l + 1] = (float)(1.0 / sqrt(-x[k1].y * sq));
            }
        }
    }
    __syncthreads();   // X takes the place of Y and its rows
    // C: X, eight lanes per m over the shells as in A
    const size_t pa = (size_t)rows_pad * Ks, pb = (size_t)cols_pad * Ks;
    for (int base = 0; base < M * nq; base += NGRP) {
        const int e = min(base + grp, M * nq - 1), m = e / nq, c0 = CPT * (e - m * nq);
        float2 v[KL];
        const float2 *b = UB + (size_t)cl * Ks + (size_t)m * pb;
#pragma unroll
        for (int i = 0; i < KL; ++i) v[i] = l8 + 8 * i < Ks ? b[l8 + 8 * i] : make_float2(0.f, 0.f);
#pragma unroll UC
        for (int cg = c0; cg < c0 + CPT; cg += GP) {
            float xr[GP], xi[GP];
#pragma unroll
            for (int u = 0; u < GP; ++u) {
                const int rs = cg + u < nc ? rs_s[cg + u] : -1;
                const float2 *a = UA + (size_t)max(rs, 0) * Ks + (size_t)m * pa;
                xr[u] = xi[u] = 0.f;
#pragma unroll
                for (int i = 0; i < KL; ++i) {
                    if (l8 + 8 * i >= Ks) continue;
                    const float2 r = a[l8 + 8 * i];
                    xr[u] = fmaf(r.x, v[i].x, fmaf(r.y, v[i].y, xr[u]));
                    xi[u] = fmaf(r.y, v[i].x, fmaf(-r.x, v[i].y, xi[u]));
                }
            }
#pragma unroll
            for (int u = 0; u < GP; ++u) {
#pragma unroll
                for (int o = 4; o; o >>= 1) {
                    xr[u] += __shfl_xor_sync(0xffffffffu, xr[u], o);
                    xi[u] += __shfl_xor_sync(0xffffffffu, xi[u], o);
                }
                // X(0) and X(P) are real
                if (base + grp < M * nq && l8 == u && cg + u < nc)
                    Xs[(cg + u) * M + m] = make_float2(4.f * xr[u], (m == 0 || m == P) ? 0.f : 4.f * xi[u]);
            }
        }
    }
    __syncthreads();
    // D: the transform, pass A a thread per (candidate, class), pass B per (candidate, block) with the
    // block's maximum, then the candidates' maxima (the lowest rotation among equals)
    for (int e = t; e < nc * P1; e += blockDim.x) {
        const int c = e / P1, j1 = e - c * P1;
        const float2 *x = Xs + c * M;
        float2 z[P2];
#pragma unroll
        for (int j2 = 0; j2 < P2; ++j2) {
            const int j = j1 + P1 * j2;
            z[j2] = make_z(x[j], x[P - j], wn_s[j]);
        }
        SFFT<P2, P1>::run(z, tw);
#pragma unroll
        for (int l2 = 0; l2 < P2; ++l2) slab[c * (P | 1) + l2 * P1 + j1] = l2 == 0 ? z[l2] : c_mul(z[l2], wp_s[j1 * l2]);
    }
    __syncthreads();
    for (int e = t; e < nc * P2; e += blockDim.x) {
        const int c = e / P2, l2 = e - c * P2;
        const float2 *x = slab + c * (P | 1) + l2 * P1;
        const float *ds = Ds + c * P;
        const float scale = 1.0f / (2.0f * (float)N);
        float2 v[P1];
#pragma unroll
        for (int j1 = 0; j1 < P1; ++j1) v[j1] = x[j1];
        SFFT<P1, P2>::run(v, tw);
        float best = -INFINITY;
        int brot = 0;
#pragma unroll
        for (int l1 = 0; l1 < P1; ++l1) {
            const int r0 = 2 * (l2 + P2 * l1), r1 = r0 + 1;
            const float d0 = ds[r0 < P ? r0 : r0 - P], d1 = ds[r1 < P ? r1 : r1 - P];
            const float c0 = EU ? fmaf(scale, v[l1].x, d0) : scale * v[l1].x * d0;
            const float c1 = EU ? fmaf(scale, v[l1].y, d1) : scale * v[l1].y * d1;
            if (c0 > best) { best = c0; brot = r0; }     // rotations rise with l1
            if (c1 > best) { best = c1; brot = r1; }
        }
        pbest[c * P2 + l2] = best;
        prot[c * P2 + l2] = brot;
    }
    __syncthreads();
    if (t < nc) {
        const int rs = rs_s[t];
        float best = -INFINITY;
        int brot = 0;
        for (int l2 = 0; l2 < P2; ++l2) {
            const float c = pbest[t * P2 + l2];
            const int r = prot[t * P2 + l2];
            if (c > best || (c == best && r < brot)) { best = c; brot = r; }
        }
        bc_s[t] = rs < 0 ? -INFINITY : best;
        bi_s[t] = rs < 0 ? 0x7fffffff : rs * N + brot;
    }
    __syncthreads();
    if (t == 0) {
        float b = -INFINITY;
        int bid = 0x7fffffff;
        for (int i = 0; i < nc; ++i) {
            const float c = bc_s[i];
            const int id = bi_s[i];
            if (id != 0x7fffffff && (c > b || (c == b && id < bid))) { b = c; bid = id; }
        }
        pftcc_best o;
        if (bid == 0x7fffffff) { o.iref = 0; o.irot = 0; o.ishift = -1; o.corr = -INFINITY; }
        else {
            const int rs2 = bid / N, rot = bid - rs2 * N;
            o.iref = rs2 / nshifts + 1;
            o.ishift = has_shifts ? rs2 % nshifts : -1;
            o.irot = rot + 1;
            o.corr = b;
        }
        out[perm[cl]] = o;
    }
}

// ---------------------------------------------------------------------------------------
static void fill_tw(TwTables &tw, int P)
{
    for (int e = 0; e < P; ++e) {
        const double a = -2.0 * M_PI * e / P, b = -2.0 * M_PI * e / (2.0 * P);
        tw.wP[e] = make_float2((float)cos(a), (float)sin(a));
        tw.wN[e] = make_float2((float)cos(b), (float)sin(b));
        tw.pc[e] = make_float2(tw.wP[e].x, tw.wP[e].x);
        tw.ps[e] = make_float2(tw.wP[e].y, tw.wP[e].y);
        tw.pn[e] = make_float2(-tw.wP[e].y, -tw.wP[e].y);
    }
}

bool stage2_fast_supported(int P) { return P == 64 || P == 180 || P == 300; }

// floats of normalising factors per (reference, particle) the search's pass B reads, and the group
// layout k_norm_fft writes them in (S2Split)
int stage2_fast_dlen(int P)
{
    switch (P) {
    case 64: return s2_dlen<64>();
    case 180: return s2_dlen<180>();
    case 300: return s2_dlen<300>();
    default: return P;
    }
}

template <int P, bool ROT, bool WRITE, bool EU>
static cudaError_t launch_s2_k(pftcc_handle *h, const S2Fast &sp, int blocks, const S2Wave *waves_dev, float2 *cand,
                               float *ccall, const int *perm)
{
    using S = S2Split<P>;
    TwTables tw;
    fill_tw(tw, P);
    const size_t smem = (size_t)P * 32 * sizeof(float4) + (size_t)S::ROLES * 32 * (sizeof(float2) + (ROT ? sizeof(int2) : 0)) +
                        8 * 32 * (sizeof(float) + sizeof(int));
    const cudaError_t e = smem_limit((const void *)k_stage2_fast<P, ROT, WRITE, EU>, smem);
    if (e != cudaSuccess) return e;
    PFTCC_LAUNCH(h);
    KTimer kt(h, PFTCC_K_STAGE2);
    k_stage2_fast<P, ROT, WRITE, EU><<<blocks, 32 * S::ROLES, smem, h->stream>>>(sp, tw, waves_dev, cand, ccall, perm);
    return cudaGetLastError();
}

template <int P>
static cudaError_t launch_s2(pftcc_handle *h, const S2Fast &sp, int blocks, const S2Wave *waves_dev, float2 *cand,
                             float *ccall, const int *perm, bool eu, bool rot)
{
    if (ccall) return eu ? launch_s2_k<P, true, true, true>(h, sp, blocks, waves_dev, cand, ccall, perm)
                         : launch_s2_k<P, true, true, false>(h, sp, blocks, waves_dev, cand, ccall, perm);
    if (rot) return eu ? launch_s2_k<P, true, false, true>(h, sp, blocks, waves_dev, cand, ccall, perm)
                       : launch_s2_k<P, true, false, false>(h, sp, blocks, waves_dev, cand, ccall, perm);
    return eu ? launch_s2_k<P, false, false, true>(h, sp, blocks, waves_dev, cand, ccall, perm)
              : launch_s2_k<P, false, false, false>(h, sp, blocks, waves_dev, cand, ccall, perm);
}

// every wave of the list in one launch, one block per column (blk0 filled in); rot: the candidates
// carry their rotation (nothing re-scores them).  The waves are in column order and share no column: a block
// merges its rows into its column's top 8 with no order between blocks
cudaError_t launch_stage2_waves(pftcc_handle *h, int P, std::vector<S2Wave> &waves, int nshifts, int nrs_total,
                                float2 *cand, float *ccall, const int *perm, int eu, int rot)
{
    UmmaState &us = h->ws.umma;
    const int nw = (int)waves.size();
    if (nw == 0) return cudaSuccess;
    long long blocks = 0;
    int next_col = 0;
    for (S2Wave &w : waves) {
        if (w.col0 < next_col || (unsigned long long)P * w.xcols * w.xrows >= (1ull << 32) || w.cols <= 0 || w.rows <= 0 ||
            w.zc0 + w.cols > w.xcols || w.rofs + w.rows > w.xrows || (w.xrows & 1))
            return cudaErrorInvalidValue;
        w.blk0 = (int)blocks;
        blocks += w.cols;
        next_col = w.col0 + w.cols;
    }
    if (blocks >= (1LL << 31)) return cudaErrorInvalidValue;
    if (us.s2waves_cap < nw) {
        dev_free(h, us.d_s2waves);
        us.d_s2waves = nullptr;
        us.s2waves_cap = 0;
        const int cap = std::max(nw, 16);
        if (dev_alloc(h, (void **)&us.d_s2waves, (size_t)cap * sizeof(S2Wave), "stage-2 waves") != PFTCC_OK)
            return cudaErrorMemoryAllocation;
        us.s2waves_cap = cap;
    }
    if (stage_upload(h, us.d_s2waves, waves.data(), (size_t)nw * sizeof(S2Wave), "stage-2 waves") != PFTCC_OK)
        return cudaErrorInvalidValue;
    S2Fast sp{nshifts, 2 * P, nrs_total, nw, 1.0f / (2.0f * (float)(2 * P))};
    switch (P) {
    case 64: return launch_s2<64>(h, sp, (int)blocks, us.d_s2waves, cand, ccall, perm, eu != 0, rot != 0);
    case 180: return launch_s2<180>(h, sp, (int)blocks, us.d_s2waves, cand, ccall, perm, eu != 0, rot != 0);
    case 300: return launch_s2<300>(h, sp, (int)blocks, us.d_s2waves, cand, ccall, perm, eu != 0, rot != 0);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_stage2_fast(pftcc_handle *h, int P, int rows, int xrows, int xcols, int row0, int nshifts, int r0,
                               int dcols, int col0, int cols, int nrs_total, const float2 *X, const float *Dinv,
                               float2 *cand, float *ccall, const int *perm, int eu, int rot)
{
    std::vector<S2Wave> w(1);
    w[0] = S2Wave{X, Dinv, row0, rows, 0, xrows, xcols, col0, cols, 0, r0, dcols, 0, 0};
    return launch_stage2_waves(h, P, w, nshifts, nrs_total, cand, ccall, perm, eu, rot);
}

template <int P1, int P2, bool EU>
static cudaError_t launch_rs(pftcc_handle *h, int ncols, int ntop, int Ks, int nshifts, int has_shifts,
                             const float2 *UA, int rows_pad, const float2 *UB, int cols_pad, const double2 *RU,
                             const double2 *CV, const float *sqp, const float2 *cand, const int *perm, int c0,
                             pftcc_best *out)
{
    constexpr int P = P1 * P2;
    TwTables tw;
    fill_tw(tw, P);
    if (ntop < 1 || ntop > RS_MAX) return cudaErrorInvalidValue;
    const size_t smem = RescoreSmem<P1, P2>::bytes;
    auto k = Ks <= 24 ? k_rescore_md<P1, P2, EU, 3> : Ks <= 40 ? k_rescore_md<P1, P2, EU, 5> : k_rescore_md<P1, P2, EU, 8>;
    if (Ks > 64) return cudaErrorInvalidValue;
    cudaError_t e = smem_limit((const void *)k, smem);
    if (e != cudaSuccess) return e;
    PFTCC_LAUNCH(h);
    KTimer kt(h, PFTCC_K_EXACT);
    k<<<ncols, RS_THREADS, smem, h->stream>>>(
        ncols, ntop, Ks, 2 * P, nshifts, has_shifts, tw, UA, rows_pad, UB, cols_pad, RU, CV, sqp, cand, perm, c0, out);
    return cudaGetLastError();
}

template <int P1, int P2>
static cudaError_t launch_rs_eu(pftcc_handle *h, int eu, int ncols, int ntop, int Ks, int nshifts, int has_shifts,
                                const float2 *UA, int rows_pad, const float2 *UB, int cols_pad, const double2 *RU,
                                const double2 *CV, const float *sqp, const float2 *cand, const int *perm, int c0,
                                pftcc_best *out)
{
    if (eu)
        return launch_rs<P1, P2, true>(h, ncols, ntop, Ks, nshifts, has_shifts, UA, rows_pad, UB, cols_pad, RU, CV,
                                       sqp, cand, perm, c0, out);
    return launch_rs<P1, P2, false>(h, ncols, ntop, Ks, nshifts, has_shifts, UA, rows_pad, UB, cols_pad, RU, CV, sqp,
                                    cand, perm, c0, out);
}

cudaError_t launch_rescore_md(pftcc_handle *h, int P, int ncols, int ntop, int Ks, int nshifts, int has_shifts,
                              const float2 *UA, int rows_pad, const float2 *UB, int cols_pad, const double2 *RU,
                              const double2 *CV, const float *sqp, const float2 *cand, const int *perm, int c0,
                              pftcc_best *out, int eu)
{
    switch (P) {
    case 64: return launch_rs_eu<8, 8>(h, eu, ncols, ntop, Ks, nshifts, has_shifts, UA, rows_pad, UB, cols_pad, RU, CV, sqp, cand, perm, c0, out);
    case 180: return launch_rs_eu<12, 15>(h, eu, ncols, ntop, Ks, nshifts, has_shifts, UA, rows_pad, UB, cols_pad, RU, CV, sqp, cand, perm, c0, out);
    case 300: return launch_rs_eu<15, 20>(h, eu, ncols, ntop, Ks, nshifts, has_shifts, UA, rows_pad, UB, cols_pad, RU, CV, sqp, cand, perm, c0, out);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pftcc
