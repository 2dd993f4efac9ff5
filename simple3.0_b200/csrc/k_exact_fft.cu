// k_exact_fft.cu -- the exact correlations of k_exact (every rotation of a prepared reference
// against a particle, FP32 operands, FP64 sums) by FP64 transforms over the polar angle.
//
// With the particle continued over the full circle by conjugate symmetry, its real part repeats
// after P = N/2 samples and its imaginary part changes sign, so that
//   corr(s) = sum_k sum_n Re A Re Q(n + s) + Im A Im Q(n + s) = Ce(s) + Co(s),
//   corr(s + P) = Ce(s) - Co(s),  s < P,
// Ce the cyclic correlation of the real parts and Co the sign-changing one of the imaginary parts,
// which the twist w_N^{-n} makes cyclic: with a'(n) = a(n) w_N^{-n} and b' likewise,
// sum_n a'(n) conj b'(n + s) = w_N^s sum_n a(n) conj b(n + s).  Two shells go through one complex
// transform, a = a_k + i a_k': Re sum_n a(n) conj b(n + s) is the sum of both shells' correlations,
// so nothing has to be separated.  Per shell pair and channel (real parts, imaginary parts, and in
// the particle frame |ref|^2 against CTF^2 for the normaliser D(s)) one length-P transform of the
// reference and one of the particle are multiplied, the products summed over the pairs in registers,
// and one transform of the sums gives every rotation: R(s) = (1/P) sum_j T(j) w_P^{-js}.
//
// A normaliser that is small beside the squares it is made of (the reference's energy lies where the CTF
// almost vanishes) is within the transforms' rounding; it is formed term by term instead (ex_direct_norm).
//
// Operands are prepared as k_exact prepares them (FP32 products with the FP32-rounded shift phases
// of the FP64 recurrence); everything after that is FP64, as there: measured on the cases' ranges
// against 64-bit results the error is that of the final FP32 rounding (5e-8 to 9e-8), as before.
//
// Work per (reference, shift, particle): 2 ceil(Ks/2) transforms of length P in place of N P Ks
// complex products, 29 times fewer FP64 operations at P = 180, Ks = 39.
#include "pftcc_internal.cuh"
#include "spec_fft.cuh"

#include <algorithm>
#include <cmath>

namespace pftcc {

// the best of one block's share of a group's items
struct ExPart { float cc; int item, rot, pad; };

struct ExArgs {
    Geom g;
    const float2 *refs_even, *refs_odd, *ptcls;
    const float *ctfmats;
    const uint8_t *iseven;
    const float *sqsums;
    const double *argtransf, *argtransf1;
    const double2 *wn;            // w_N^{-e}, e < N
    const Group *groups;
    const Work *work;
    const float *shifts;
    const float *sig2, *pxls, *snorm;
    int mode, cc1_kstop, nrefs, per;   // per: items of a group for each block (a multiple of R)
    float *out;
    pftcc_best *best;
    ExPart *part;                 // per (group, block) when a group's items are shared between blocks
    const uint8_t *rotmask;
    int one;                      // the single request below instead of the tables
    Group one_group;
    Work one_work;
    float one_shift[2];
};

template <int FRAME> __host__ __device__ constexpr int ex_channels() { return FRAME == PFTCC_FRAME_PTCL ? 3 : 2; }

// shared memory: the twiddles w_N^{-e} and w_P^{-e}, e < P, the transforms' rows, the staged operands
// of the iteration's shells (and in the particle frame their squares), the Euclidean shell weights
template <int P1, int P2, int FRAME, int R, int G> static size_t ex_smem(int K)
{
    constexpr int P = P1 * P2, CH = ex_channels<FRAME>(), RS = P1 | 1;
    return (size_t)2 * P * sizeof(double2) + (size_t)(R + 1) * G * CH * P2 * RS * sizeof(double2) +
           (size_t)(R + 1) * 2 * G * P * (sizeof(float2) + (CH == 3 ? sizeof(float) : 0)) +
           (FRAME == FRAME_EUCLID ? (size_t)K * sizeof(double) : 0);
}

// (c, item, rot) ranks above (c2, item2, rot2): larger value, then the earlier item, then the lower rotation
__device__ __forceinline__ bool ex_above(float c, int item, int rot, float c2, int item2, int rot2)
{
    return c > c2 || (c == c2 && (item < item2 || (item == item2 && rot < rot2)));
}

// The roundings are spelled out (fma and rounded products) wherever the compiler could choose to contract:
// a request gives the same bits alone, in a batch and in a search.
__device__ __forceinline__ double sqsum(float a, float b) { return fma((double)a, (double)a, __dmul_rn((double)b, (double)b)); }

__device__ __forceinline__ pftcc_best ex_best(const Work *work, int first, float cc, int item, int rot)
{
    pftcc_best b;
    b.iref = 0; b.irot = 0; b.ishift = -1; b.corr = -INFINITY;
    if (item >= 0) {
        const Work w = work[first + item];
        b.iref = w.iref + 1; b.irot = rot + 1; b.ishift = w.ishift; b.corr = cc;
    }
    return b;
}

// D(s) = sum_k sum_n |ref(k, n)|^2 CTF^2(k, n + s) term by term, s < P.  The transforms leave D with an error
// of a few 2^-53 of B = sum over the shell pairs of (sum_n of both shells' |ref|^2) (sum_n of both shells'
// CTF^2): by Cauchy-Schwarz they round at eps |a|_2 |b|_2 a pair, and the squares are not negative.  Above 1e-7 B
// that is 1e-8 of D at most, 5e-9 of a correlation (2^-24, its rounding, is 6e-8); below it this takes over.
__device__ __noinline__ double ex_direct_norm(const float2 *ref, const float *sn, const float *ctf, int Ks, int P, int s)
{
    double d = 0.0;
    for (int ik = 0; ik < Ks; ++ik)
        for (int n = 0; n < P; ++n) {
            float2 v = ref[ik * P + n];
            if (sn) { v.x *= sn[ik]; v.y *= sn[ik]; }
            const float c = ctf ? ctf[ik * P + (n + s < P ? n + s : n + s - P)] : 1.f;
            d = fma((double)fmaf(v.x, v.x, __fmul_rn(v.y, v.y)), (double)(c * c), d);
        }
    return d;
}

// One block takes `per` items of one group, R at a time, G shell pairs per iteration:
//   stage   every item's prepared samples and the particle's, 2 G shells, into shared memory
//   pass 1  task (transform, n1): a length-P2 DFT over n2 of the channel's sequence, times the twiddles
//   pass 2  task (transform, k2): a length-P1 DFT over n1, in place: row k2 then holds F(k2 + P2 k1)
//   sum     the products with the particle's spectra, each (item, channel, j) in one thread's registers
// R = 4 items share the particle's transforms (a quarter more work than none at all, against twice
// the work for R = 1); a single item instead takes G = 4 shell pairs at once, to have enough tasks
// for the block.
template <int P1, int P2, int FRAME, int R, int G, int T, int MB>
__global__ void __launch_bounds__(T, MB) k_exact_fft(const __grid_constant__ ExArgs x)
{
    constexpr int P = P1 * P2, N = 2 * P, CH = ex_channels<FRAME>(), RS = P1 | 1, ROW = P2 * RS, KK = 2 * G;
    constexpr int NF = (R + 1) * G * CH;              // transforms of an iteration; index ((x G + g) CH + ch)
    constexpr int NPT = (R * P + T - 1) / T;          // (item, n) per thread in the staging
    constexpr int NQ = (P + T - 1) / T;
    constexpr int NACC = (R * CH * P + T - 1) / T;    // sums per thread
    extern __shared__ float4 smem4[];
    double2 *wn = reinterpret_cast<double2 *>(smem4);                 // [P] w_N^{-e}
    double2 *tw = wn + P;                                              // [P] w_P^{-e}
    double2 *buf = tw + P;                                             // [NF][P2][RS]
    float2 *stg = reinterpret_cast<float2 *>(buf + NF * ROW);          // [R + 1][KK][P]
    float *stg2 = reinterpret_cast<float *>(stg + (R + 1) * KK * P);   // [R + 1][KK][P] squares
    double *W = reinterpret_cast<double *>(stg + (R + 1) * KK * P);    // [K] Euclidean shell weights (no squares then)
    __shared__ double sums[R + 1];
    __shared__ double dmag[R];    // B of ex_direct_norm
    __shared__ float imax[R];
    __shared__ float bcc[T / 32];
    __shared__ int bit[T / 32], brt[T / 32];
    const Geom &g = x.g;
    const int t = threadIdx.x, K = g.K, Ks = g.Ks;
    const Group grp = x.one ? x.one_group : x.groups[blockIdx.x];
    const int slot = grp.slot;
    const float2 *q = x.ptcls + (long long)slot * K * P;
    const float *ctf = x.ctfmats ? x.ctfmats + (long long)slot * K * P : nullptr;
    const bool even = x.iseven[slot] != 0;
    const float2 *refs = even ? x.refs_even : x.refs_odd;
    const float sqp = x.sqsums[slot];
    for (int e = t; e < P; e += T) {
        wn[e] = x.wn[e];
        tw[e] = x.wn[2 * e];
    }
    if (FRAME == FRAME_EUCLID) {
        for (int ik = t; ik < K; ik += T) W[ik] = (double)x.pxls[ik] / ((double)P * (double)x.sig2[(long long)slot * K + ik]);
        __syncthreads();
    }
    float run_cc = -INFINITY;
    int run_rot = 0x7fffffff, run_item = -1;
    const int it_end = min(grp.count, ((int)blockIdx.y + 1) * x.per);
    for (int it0 = blockIdx.y * x.per; it0 < it_end; it0 += R) {
        const int ni = min(R, it_end - it0);
        // this thread's samples: reference pointer, shift phase and its step over the shells
        const float2 *rp[NPT];
        const float *sn[NPT];
        double2 st[NPT], sv[NPT];
        double sq[NPT], sqq[NQ];
        bool sh[NPT];
#pragma unroll
        for (int i = 0; i < NPT; ++i) {
            const int e = t + i * T, r = e / P, n = e - r * P;
            rp[i] = nullptr; sn[i] = nullptr; sh[i] = false; sq[i] = 0.0;
            st[i] = make_double2(1.0, 0.0); sv[i] = make_double2(1.0, 0.0);
            if (r < ni) {
                const Work w = x.one ? x.one_work : x.work[grp.first + it0 + r];
                rp[i] = refs + (long long)w.iref * K * P + n;
                sh[i] = w.ishift >= 0;
                if (x.snorm && (FRAME != FRAME_EUCLID || !sh[i])) sn[i] = x.snorm + ((size_t)(even ? 0 : 1) * x.nrefs + w.iref) * Ks;
                if (sh[i]) {
                    const float *s = x.one ? x.one_shift : x.shifts + 2 * w.ishift;
                    const double sx = (double)s[0], sy = (double)s[1];
                    sincos(x.argtransf[n] * sx + x.argtransf[P + n] * sy, &st[i].y, &st[i].x);
                    sincos(x.argtransf1[n] * sx + x.argtransf1[P + n] * sy, &sv[i].y, &sv[i].x);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NQ; ++i) sqq[i] = 0.0;
        double2 acc[NACC];
#pragma unroll
        for (int i = 0; i < NACC; ++i) acc[i] = make_double2(0.0, 0.0);
        double mag = 0.0;   // B, of item t < R
        // cc_2 sums the reference's squares over all shells, cc_1 to kstop; the Euclidean sums to kstop
        for (int k0 = 0; k0 < K; k0 += KK) {
            const bool spectra = k0 < Ks;
#pragma unroll
            for (int i = 0; i < NPT; ++i) {
                const int e = t + i * T, r = e / P, n = e - r * P;
                if (r >= R) continue;
                float2 rv[KK];
                float cf[KK];
#pragma unroll
                for (int kk = 0; kk < KK; ++kk) {
                    const int ik = k0 + kk;
                    rv[kk] = make_float2(0.f, 0.f);
                    cf[kk] = 1.f;
                    if (rp[i] && ik < K) {
                        rv[kk] = rp[i][(long long)ik * P];
                        if (FRAME != PFTCC_FRAME_PTCL && ctf) cf[kk] = ctf[ik * P + n];
                    }
                }
#pragma unroll
                for (int kk = 0; kk < KK; ++kk) {
                    const int ik = k0 + kk;
                    float2 v = rv[kk];
                    if (sn[i] && ik < Ks) { v.x *= sn[i][ik]; v.y *= sn[i][ik]; }
                    float ar = v.x, ai = v.y;
                    if (FRAME != PFTCC_FRAME_PTCL && ctf) { ar *= cf[kk]; ai *= cf[kk]; }
                    if (sh[i]) {
                        const float sr = (float)st[i].x, si = (float)st[i].y;
                        const float tr = fmaf(ar, sr, -__fmul_rn(ai, si)), ti = fmaf(ar, si, __fmul_rn(ai, sr));
                        ar = tr; ai = ti;
                        // the recurrence: shmat(:, k + 1) = shmat(:, k) * shvec
                        st[i] = sfft::d_mul(st[i], sv[i]);
                    }
                    const double a2 = sqsum(ar, ai);
                    if (FRAME == FRAME_EUCLID) {
                        if (ik < Ks) sq[i] = fma(W[ik], a2, sq[i]);
                    } else if (ik < Ks || sh[i] || !x.cc1_kstop) {
                        sq[i] += a2;
                    }
                    if (spectra) {   // shells past kstop take no part in the correlation
                        stg[((size_t)r * KK + kk) * P + n] = ik < Ks ? make_float2(ar, ai) : make_float2(0.f, 0.f);
                        if (CH == 3) stg2[((size_t)r * KK + kk) * P + n] = ik < Ks ? fmaf(v.x, v.x, __fmul_rn(v.y, v.y)) : 0.f;
                    }
                }
            }
            if (!spectra) continue;
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                const int n = T - 1 - t + i * T;   // from the other end: the threads with fewer items first
                if (n >= P) continue;
#pragma unroll
                for (int kk = 0; kk < KK; ++kk) {
                    const int ik = k0 + kk;
                    float2 v = make_float2(0.f, 0.f);
                    float c = 0.f;
                    if (ik < Ks) {
                        v = q[(long long)ik * P + n];
                        c = 1.f;
                        if (FRAME == PFTCC_FRAME_PTCL) {
                            if (ctf) c = ctf[ik * P + n];
                            v.x *= c; v.y *= c;
                        }
                        if (FRAME == FRAME_EUCLID) sqq[i] = fma(W[ik], sqsum(v.x, v.y), sqq[i]);
                    }
                    stg[((size_t)R * KK + kk) * P + n] = v;
                    if (CH == 3) stg2[((size_t)R * KK + kk) * P + n] = c * c;
                }
            }
            __syncthreads();
            for (int e = t; e < NF * P1; e += T) {
                const int f = e / P1, n1 = e - f * P1, ch = f % CH, gq = f / CH % G, xi = f / (CH * G);
                const size_t base = ((size_t)xi * KK + 2 * gq) * P + n1;
                double wa = 1.0, wb = 1.0;   // the Euclidean shell weights, on the reference's side
                if (FRAME == FRAME_EUCLID && xi < R) {
                    wa = W[min(k0 + 2 * gq, Ks - 1)];
                    wb = W[min(k0 + 2 * gq + 1, Ks - 1)];
                }
                double2 z[P2];
                if (ch == 2) {
                    const float *s = stg2 + base;
#pragma unroll
                    for (int n2 = 0; n2 < P2; ++n2) z[n2] = make_double2((double)s[P1 * n2], (double)s[P + P1 * n2]);
                } else {
                    const float *s = reinterpret_cast<const float *>(stg + base) + ch;
#pragma unroll
                    for (int n2 = 0; n2 < P2; ++n2) {
                        z[n2] = make_double2((double)s[2 * P1 * n2], (double)s[2 * (P + P1 * n2)]);
                        if (FRAME == FRAME_EUCLID) z[n2] = make_double2(__dmul_rn(z[n2].x, wa), __dmul_rn(z[n2].y, wb));
                        if (ch == 1) z[n2] = sfft::d_mul(z[n2], wn[n1 + P1 * n2]);
                    }
                }
                sfft::DFFT<P2, P1>::run(z, tw);
                double2 *row = buf + (size_t)f * ROW + n1;
#pragma unroll
                for (int k2 = 0; k2 < P2; ++k2) row[k2 * RS] = (k2 == 0) ? z[k2] : sfft::d_mul(z[k2], tw[n1 * k2]);
            }
            __syncthreads();
            for (int e = t; e < NF * P2; e += T) {
                double2 *row = buf + (size_t)(e / P2) * ROW + (e % P2) * RS;
                double2 z[P1];
#pragma unroll
                for (int n1 = 0; n1 < P1; ++n1) z[n1] = row[n1];
                sfft::DFFT<P1, P2>::run(z, tw);
#pragma unroll
                for (int k1 = 0; k1 < P1; ++k1) row[k1] = z[k1];
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < NACC; ++i) {
                const int e = t + i * T, r = e / (CH * P), ch = e / P % CH, j = e % P, at = j / P1 * RS + j % P1;
                if (r >= R) continue;
#pragma unroll
                for (int gq = 0; gq < G; ++gq) {
                    const double2 a = buf[(size_t)((r * G + gq) * CH + ch) * ROW + at];
                    const double2 b = buf[(size_t)((R * G + gq) * CH + ch) * ROW + at];
                    acc[i].x = fma(a.x, b.x, fma(a.y, b.y, acc[i].x));     // a conj(b)
                    acc[i].y = fma(a.y, b.x, fma(-a.x, b.y, acc[i].y));
                }
            }
            if (CH == 3 && t < R) {
#pragma unroll
                for (int gq = 0; gq < G; ++gq) {   // j = 0: the sums of the pair's two shells
                    const double2 a = buf[(size_t)((t * G + gq) * CH + 2) * ROW], b = buf[(size_t)((R * G + gq) * CH + 2) * ROW];
                    mag = fma(a.x + a.y, b.x + b.y, mag);
                }
            }
            // the next iteration's barrier after the staging keeps pass 1 off the rows still read here
        }
        __syncthreads();
        // the square sums: partials by sample in a fixed order, a warp per item
        double *pt = reinterpret_cast<double *>(stg);   // [R + 1][P]
#pragma unroll
        for (int i = 0; i < NPT; ++i)
            if (t + i * T < R * P) pt[t + i * T] = sq[i];
#pragma unroll
        for (int i = 0; i < NQ; ++i)
            if (T - 1 - t + i * T < P) pt[R * P + T - 1 - t + i * T] = sqq[i];
        // T(j) = row k2, entry k1 of its transform (j = k2 + P2 k1) into natural order for the transform back
#pragma unroll
        for (int i = 0; i < NACC; ++i) {
            const int e = t + i * T, f = e / P, j = e % P, k2 = j / P1, k1 = j % P1;
            if (f < R * CH) buf[(size_t)f * ROW + k2 + P2 * k1] = acc[i];
        }
        if (t < R) {
            imax[t] = -INFINITY;
            dmag[t] = mag;
        }
        __syncthreads();
        for (int r = t >> 5; r <= R; r += T / 32) {
            double s = 0.0;
            for (int n = t & 31; n < P; n += 32) s += pt[r * P + n];
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if ((t & 31) == 0) sums[r] = s;
        }
        double2 z[(R * CH * P1 + T - 1) / T][P2];
#pragma unroll
        for (int i = 0; i < (R * CH * P1 + T - 1) / T; ++i) {
            const int e = t + i * T, f = e / P1, n1 = e - f * P1;
            if (e >= R * CH * P1) continue;
#pragma unroll
            for (int n2 = 0; n2 < P2; ++n2) z[i][n2] = buf[(size_t)f * ROW + n1 + P1 * n2];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < (R * CH * P1 + T - 1) / T; ++i) {
            const int e = t + i * T, f = e / P1, n1 = e - f * P1;
            if (e >= R * CH * P1) continue;
            sfft::DFFT<P2, P1>::run(z[i], tw);
            double2 *row = buf + (size_t)f * ROW + n1;
#pragma unroll
            for (int k2 = 0; k2 < P2; ++k2) row[k2 * RS] = (k2 == 0) ? z[i][k2] : sfft::d_mul(z[i][k2], tw[n1 * k2]);
        }
        __syncthreads();
        for (int e = t; e < R * CH * P2; e += T) {
            double2 *row = buf + (size_t)(e / P2) * ROW + (e % P2) * RS;
            double2 v[P1];
#pragma unroll
            for (int n1 = 0; n1 < P1; ++n1) v[n1] = row[n1];
            sfft::DFFT<P1, P2>::run(v, tw);
#pragma unroll
            for (int k1 = 0; k1 < P1; ++k1) row[k1] = v[k1];
        }
        __syncthreads();
        for (int e = t; e < ni * P; e += T) {
            const int r = e / P, s = e - r * P, at = s % P2 * RS + s / P2;
            const double ce = buf[(size_t)(r * CH) * ROW + at].x / P;
            const double2 o = buf[(size_t)(r * CH + 1) * ROW + at], w = wn[s];
            const double co = fma(o.x, w.x, -__dmul_rn(o.y, w.y)) / P;      // Re(R'(s) w_N^{-s})
            float c0, c1;
            if (FRAME == FRAME_EUCLID) {
                const double half = __dmul_rn(0.5, sums[r] + sums[R]);
                c0 = (float)(ce + co - half);
                c1 = (float)(ce - co - half);
            } else {
                double d = sums[r];
                if (FRAME == PFTCC_FRAME_PTCL) {
                    d = buf[(size_t)(r * CH + CH - 1) * ROW + at].x / P;
                    if (d <= 1e-7 * dmag[r]) {
                        const int iref = x.one ? x.one_work.iref : x.work[grp.first + it0 + r].iref;
                        d = dmag[r] == 0.0 ? 0.0
                                           : ex_direct_norm(refs + (long long)iref * K * P,
                                                            x.snorm ? x.snorm + ((size_t)(even ? 0 : 1) * x.nrefs + iref) * Ks : nullptr,
                                                            ctf, Ks, P, s);
                        // no sample where neither |ref| nor the CTF is zero: 0 / 0 as the direct sums have it, the
                        // numerator being left as rounding
                        if (d == 0.0) d = NAN;
                    }
                }
                const double den = sqrt(d * sqp);
                c0 = (float)((ce + co) / den);
                c1 = (float)((ce - co) / den);
            }
            if (x.mode == MODE_FULL) {
                float *o2 = x.out + (x.one ? x.one_work.out : x.work[grp.first + it0 + r].out);
                o2[s] = c0;
                o2[s + P] = c1;
                continue;
            }
            // rotmask [group][N] (optional): rotations outside the mask take no part in the maximum
            const uint8_t *mk = x.rotmask ? x.rotmask + (size_t)blockIdx.x * N : nullptr;
            float c = -INFINITY;
            int rot = s;
            if (!mk || mk[s]) c = c0 > c ? c0 : c;
            if ((!mk || mk[s + P]) && c1 > c) { c = c1; rot = s + P; }
            if (c == -INFINITY) continue;
            if (x.mode == MODE_BEST) {
                if (run_item < 0 || ex_above(c, it0 + r, rot, run_cc, run_item, run_rot)) { run_cc = c; run_item = it0 + r; run_rot = rot; }
            } else if (c >= 0.f) {
                atomicMax(reinterpret_cast<int *>(imax + r), __float_as_int(c + 0.f));   // -0 as +0
            } else {
                atomicMin(reinterpret_cast<unsigned *>(imax + r), __float_as_uint(c));
            }
        }
        __syncthreads();
        if (x.mode == MODE_ITEMMAX && t < ni) x.out[(x.one ? x.one_work : x.work[grp.first + it0 + t]).out] = imax[t];
        __syncthreads();
    }
    if (x.mode != MODE_BEST) return;
    for (int o = 16; o > 0; o >>= 1) {
        const float oc = __shfl_xor_sync(0xffffffffu, run_cc, o);
        const int oi = __shfl_xor_sync(0xffffffffu, run_item, o), orot = __shfl_xor_sync(0xffffffffu, run_rot, o);
        if (oi >= 0 && (run_item < 0 || ex_above(oc, oi, orot, run_cc, run_item, run_rot))) { run_cc = oc; run_item = oi; run_rot = orot; }
    }
    if ((t & 31) == 0) { bcc[t >> 5] = run_cc; bit[t >> 5] = run_item; brt[t >> 5] = run_rot; }
    __syncthreads();
    if (t == 0) {
        for (int w = 1; w < T / 32; ++w)
            if (bit[w] >= 0 && (run_item < 0 || ex_above(bcc[w], bit[w], brt[w], run_cc, run_item, run_rot))) {
                run_cc = bcc[w]; run_item = bit[w]; run_rot = brt[w];
            }
        if (x.part) x.part[(size_t)blockIdx.x * gridDim.y + blockIdx.y] = ExPart{run_cc, run_item, run_rot, 0};
        else x.best[grp.out_best] = ex_best(x.work, grp.first, run_cc, run_item, run_rot);
    }
}

// a group's best out of its blocks' (a thread per group; the blocks hold ascending items)
__global__ void k_exact_merge(const ExPart *__restrict__ part, int ny, const Group *__restrict__ groups, int ngroups,
                              const Work *__restrict__ work, pftcc_best *__restrict__ best)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ngroups) return;
    const Group grp = groups[i];
    ExPart b{-INFINITY, -1, 0, 0};
    for (int y = 0; y < ny; ++y) {
        const ExPart p = part[(size_t)i * ny + y];
        if (p.item >= 0 && (b.item < 0 || ex_above(p.cc, p.item, p.rot, b.cc, b.item, b.rot))) b = p;
    }
    best[grp.out_best] = ex_best(work, grp.first, b.cc, b.item, b.rot);
}

template <int P1, int P2, int FRAME, int R, int G, int T, int MB>
static cudaError_t launch_ex_k(pftcc_handle *h, const ExArgs &x, int ngroups, int ny)
{
    const size_t smem = ex_smem<P1, P2, FRAME, R, G>(h->g.K);
    const cudaError_t e = smem_limit((const void *)k_exact_fft<P1, P2, FRAME, R, G, T, MB>, smem);
    if (e != cudaSuccess) return e;
    PFTCC_LAUNCH(h);
    KTimer kt(h, PFTCC_K_EXACT);
    k_exact_fft<P1, P2, FRAME, R, G, T, MB><<<dim3(ngroups, ny), T, smem, h->stream>>>(x);
    return cudaGetLastError();
}

// Threads and blocks per SM: the FP64 transforms hold 60 to 80 registers of data, so a block has few
// warps and the kernel waits on its own chains (at P = 180 FP64 pipe 22 %, issue slots 30 %, 12 warps an SM);
// the shapes below are the fastest of 96 to 416 threads and 1 to 4 blocks, with 1 or 2 shell pairs at
// once for four items.  36,000 triples (100 particles, 40 references, 9 shifts) of the exact search:
//   P = 64:   0.55 ms (G = 2, 160 threads, 3 blocks); 0.58 (G = 1, 128); 0.66 (G = 2, 160, 1)
//   P = 180:  3.97 ms (G = 2, 384); 4.66 (G = 1, 256); 5.65 (G = 1, 192); the direct sums 92 ms
//   P = 300: 12.8 ms (G = 1, 256); 12.3 but 16.5 against 15.1 in the particle frame (G = 2, 320)
// single pairs (1000, and 500 at P = 300): 32, 132 and 223 us; the direct sums 6.2 ms at P = 300.
template <int P1, int P2, int FRAME, int G4, int T4, int MB4, int T1, int MB1>
static cudaError_t launch_ex(pftcc_handle *h, ExArgs &x, int ngroups, int max_items)
{
    // one or two items: nothing to share, the shells side by side instead
    if (max_items <= 2) {
        x.per = std::max(1, max_items);
        return launch_ex_k<P1, P2, FRAME, 1, 4, T1, MB1>(h, x, ngroups, 1);
    }
    // more items than the top-ntop re-score has, and too few groups to fill the GPU's blocks (148 SMs,
    // two or three blocks each): a group's items in shares of at least 8
    int ny = 1;
    if (max_items > 8) ny = std::min((max_items + 7) / 8, std::max(1, (4 * 148 + ngroups - 1) / ngroups));
    x.per = ((max_items + ny - 1) / ny + 3) / 4 * 4;
    ny = (max_items + x.per - 1) / x.per;
    if (x.mode == MODE_BEST && ny > 1) {
        if (ensure(h, (void **)&h->d_expart, &h->expart_cap, (size_t)ngroups * ny * sizeof(ExPart), "exact search partials") != PFTCC_OK)
            return cudaErrorMemoryAllocation;
        x.part = reinterpret_cast<ExPart *>(h->d_expart);
    }
    const cudaError_t e = launch_ex_k<P1, P2, FRAME, 4, G4, T4, MB4>(h, x, ngroups, ny);
    if (e != cudaSuccess || !x.part) return e;
    PFTCC_LAUNCH(h);
    k_exact_merge<<<(ngroups + 127) / 128, 128, 0, h->stream>>>(x.part, ny, x.groups, ngroups, x.work, x.best);
    return cudaGetLastError();
}

template <int P1, int P2, int G4, int T4, int MB4, int T1, int MB1>
static cudaError_t launch_ex_frame(pftcc_handle *h, ExArgs &x, int frame, int ngroups, int max_items)
{
    if (frame == PFTCC_FRAME_PTCL) return launch_ex<P1, P2, PFTCC_FRAME_PTCL, G4, T4, MB4, T1, MB1>(h, x, ngroups, max_items);
    if (frame == FRAME_EUCLID) return launch_ex<P1, P2, FRAME_EUCLID, G4, T4, MB4, T1, MB1>(h, x, ngroups, max_items);
    return launch_ex<P1, P2, PFTCC_FRAME_REF, G4, T4, MB4, T1, MB1>(h, x, ngroups, max_items);
}

bool exact_fft_supported(int P) { return P == 64 || P == 180 || P == 300; }

cudaError_t launch_exact_fft(pftcc_handle *h, const Group *groups, int ngroups, const Work *work, const float *shifts,
                             int mode, int frame, int cc1_kstop, int max_items, float *out, pftcc_best *best,
                             const uint8_t *rotmask, const ExactOne *one)
{
    ExArgs x{};
    x.g = h->g;
    x.refs_even = h->refs_even; x.refs_odd = h->refs_odd; x.ptcls = h->ptcls;
    x.ctfmats = (h->cfg.with_ctf && h->ctf_ready) ? h->ctfmats : nullptr;
    x.iseven = h->d_iseven; x.sqsums = h->sqsums;
    x.argtransf = h->argtransf; x.argtransf1 = h->argtransf1; x.wn = h->d_wn;
    x.groups = groups; x.work = work; x.shifts = shifts;
    x.sig2 = h->d_sig2; x.pxls = h->d_pxls; x.snorm = snorm_ptr(h);
    x.mode = mode; x.cc1_kstop = cc1_kstop; x.nrefs = h->nrefs;
    x.out = out; x.best = best; x.rotmask = rotmask;
    if (one) {
        x.one = 1;
        x.one_group = Group{one->slot, 0, 1, 0};
        x.one_work = Work{one->iref, one->has_shift ? 0 : -1, 0};
        x.one_shift[0] = one->sx; x.one_shift[1] = one->sy;
    }
    switch (h->g.P) {
    case 64: return launch_ex_frame<8, 8, 2, 160, 3, 128, 4>(h, x, frame, ngroups, max_items);
    case 180: return launch_ex_frame<12, 15, 2, 384, 1, 256, 2>(h, x, frame, ngroups, max_items);
    case 300: return launch_ex_frame<15, 20, 1, 256, 1, 320, 1>(h, x, frame, ngroups, max_items);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pftcc
