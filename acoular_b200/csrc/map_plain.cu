// Stage B, plain FP64 form: h^H C h per (grid point, bin) as in _freqBeamformer_FullCSM
// (acoular/fastFuncs.py:217-311), batched over bins, and its eigenvalue and custom-steering forms.
//
// CTA = 16 grid points x one bin.
//   1. distances |g - m| in FP64 (same contraction as the reference's dist_mat), phase
//      fl32(k*r), float32 cos/sin (correctly rounded, optionally corrected to the C library's
//      cosf/sinf by the exception table), steering h = cos - i sin, times r (inverse) or 1/r
//      (true level / true location); h lives only in shared memory.
//   2. B = 2 Re sum_{a<b} conj(h_a) C_ab h_b (+ sum_a C_aa |h_a|^2 without diagonal removal) on the FP64
//      matrix instruction (mma.sync m16n8k8: tcgen05 has no FP64 kind): Y = H C^T for the 16 points, a warp
//      per group of 16 rows a, then Re(conj(h_a) y_a).
//   3. cross-warp sum, normalisation of the steering type, optional clipping of negatives.
// Bound: the FP64 pipe (4 M^2 flop per point and bin at 37 TFLOP/s, DFMA and the matrix instruction alike).  The
// matrix instruction needs no masks, no broadcasts and 1/30 of the instructions of an FMA form, and 16-point tiles
// leave room for three CTAs per SM at 256 mics.  Measured (B200): 12 bins x 160,801 points x 256 mics 41.0 -> 20.4 ms
// (14.5 ms of it the matrix instruction alone, 24.4 TFLOP/s of its 4 M^2); 6 bins x 15,903 points x 300 mics
// 8.4 -> 1.39 ms; 5 bins x 1681 points x 64 mics 45 -> 22 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "map_internal.h"

namespace acb {

constexpr int kPts = 16;       // grid points per CTA (the M of the matrix instruction)
// double2 slots per mic in the steering tile: 18 instead of 16, so that the 8 lanes of one 128-bit shared-memory
// phase (2 points x 4 mics) fall on different banks
constexpr int kPtsPad = 18;
constexpr int kGroup = 16;     // rows of C (or eigenvectors) per warp and pass: two 8-column accumulators

struct MapArgs {
    int M;
    int64_t G;
    int steer_type;
    int r_diag;
    int clip;
    double norm;
    int ref_mode;
    double ref0, ref1, ref2, ref_dist;
    int faithful;
    const uint64_t *table;
    uint64_t table_mask;
};


// Steering value of a grid point and a mic at distance r (acoular/fastFuncs.py:258-273): the phase
// rounded to float32, cos - i sin of it as the C library's float32 functions give them, then the
// weight w: r (inverse) or 1/r (true level, true location; the product is within an ulp of the quotient).
// In two halves, so that a caller with several values has their table lookups in flight together.
__device__ __forceinline__ float steer_phase(double k, double r) { return __double2float_rn(__dmul_rn(k, r)); }

__device__ __forceinline__ double2 steer_value(int steer_type, float c, float s, double w)
{
    double2 h = make_double2((double)c, -(double)s);
    if (steer_type >= 2) {
        h.x *= w;
        h.y *= w;
    }
    return h;
}

__device__ __forceinline__ double steer_weight(int steer_type, double r)
{
    return steer_type == 2 ? r : steer_type >= 3 ? 1.0 / r : 1.0;
}

// Distance of a grid point and a mic, and the steering weight: r (inverse) or 1/r (true level, true location; within
// an ulp).  r is the correctly rounded square root that dist3 gives, formed from one reciprocal square root y, which
// the weight needs anyway (P. Markstein's correction: s = d y, r = s + (d - s^2) y / 2).
__device__ __forceinline__ double dist3_weight(int steer_type, double g0, double g1, double g2, double m0, double m1,
                                               double m2, double &w)
{
    const double d0 = __dsub_rn(g0, m0), d1 = __dsub_rn(g1, m1), d2 = __dsub_rn(g2, m2);
    const double d = __fma_rn(d2, d2, __fma_rn(d1, d1, __dmul_rn(d0, d0)));
    const double y = rsqrt(d);
    const double s = d * y;
    double r = fma(fma(-s, s, d), 0.5 * y, s);
    if (!(d > 0.0)) r = d;   // a grid point on a microphone: r = 0, w = infinity; NaN stays NaN
    w = steer_type == 2 ? r : y;
    return r;
}

// Steering values of mics [m0, m0 + n) for this CTA's 16 grid points into hs[(m - m0) * kPtsPad + point], zeros
// for points past the grid and rows n .. up to a multiple of 16.  With `sum` the steering type's normalisation
// terms (inverse: r^2; true level / true location: 1/r^2; custom: |h|^2) are added to S: without given distances
// a thread owns point tid % 16 (S[0]), else a warp owns points warp + NW i (S[i], partial per lane; the given
// values are contiguous along the mics).
template <bool USE_RM, bool CUSTOM, int NW>
__device__ __forceinline__ void synth_tile(const MapArgs &a, const SincosTable &sct, const double *__restrict__ rm,
                                           double k, int64_t gb, double g0, double g1, double g2,
                                           const double *__restrict__ mpos, const double2 *__restrict__ hv, int m0,
                                           int n, double2 *hs, bool sum, double (&S)[kPts / NW])
{
    const int np = (n + 15) & ~15;
    if (USE_RM || CUSTOM) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int i = 0; i < kPts / NW; ++i) {
            const int p = warp + NW * i;
            const int64_t g = gb + p;
            for (int m = lane; m < np; m += 32) {
                double2 h = make_double2(0.0, 0.0);
                if (m < n && g < a.G) {
                    if (CUSTOM) {
                        h = __ldg(hv + g * a.M + m0 + m);
                        if (sum) S[i] += h.x * h.x + h.y * h.y;
                    } else {
                        const double r = __ldg(rm + g * a.M + m0 + m);
                        const double w = steer_weight(a.steer_type, r);
                        float c, s;
                        sincos_f32_arg(steer_phase(k, r), sct, c, s);
                        h = steer_value(a.steer_type, c, s, w);
                        if (sum) S[i] += w * w;
                    }
                }
                hs[m * kPtsPad + p] = h;
            }
        }
    } else {
        // kSynth mics at a time per thread; mics past the chunk repeat its last one and are stored as zeros
        constexpr int kStep = 32 * NW / kPts, kSynth = 4;
        const int p = threadIdx.x & (kPts - 1);
        const bool ok = gb + p < a.G;
        for (int mb = threadIdx.x / kPts; mb < np; mb += kSynth * kStep) {
            double w[kSynth];
            SincosPending<kSynth> v;
#pragma unroll
            for (int u = 0; u < kSynth; ++u) {
                const int m = m0 + min(mb + u * kStep, n - 1);
                const double r = dist3_weight(a.steer_type, g0, g1, g2, __ldg(mpos + m), __ldg(mpos + a.M + m),
                                              __ldg(mpos + 2 * a.M + m), w[u]);
                v.x[u] = steer_phase(k, r);
            }
            sincos_begin(v, sct);
            sincos_finish(v, sct);
#pragma unroll
            for (int u = 0; u < kSynth; ++u) {
                const int m = mb + u * kStep;
                double2 h = steer_value(a.steer_type, v.c[u], v.s[u], w[u]);
                if (!ok || m >= n) h = make_double2(0.0, 0.0);
                else if (sum) S[0] += w[u] * w[u];
                if (m < np) hs[m * kPtsPad + p] = h;
            }
        }
    }
}

// Quadratic-form contribution of rows [ra0, ra0 + na) x columns [cb0, cb0 + nb) of C: returns this lane's parts of
// sum Re(conj(h_a) C_ab h_b) for points g = lane / 4 and g + 8.  `diag`: the two ranges are the same mics, only
// b > a counts, and half the (real) diagonal with `with_diag`.  Rows of C are read from global memory (L2) straight
// into the B operand, two steps of 4 columns ahead: a lane's element C[a][b] serves the real and the imaginary
// product, and every element is read once per CTA.  What does not count takes no part, so that it may be infinite or NaN
// (the diagonal of a CSM whose removal was asked for, say): entries left of the diagonal, a diagonal that is not wanted
// and columns past the range enter as zeros, and rows past the range (their loads repeat the last one) are left out.
template <int NW, int Q>
__device__ __forceinline__ void quad_tile(const double2 *__restrict__ C, int M, const double2 *ha, int ra0, int na,
                                          const double2 *hb, int cb0, int nb, bool diag, bool with_diag, double &off0,
                                          double &off1)
{
    constexpr int kRows = 8 * Q;   // rows per group
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int ngrp = (na + kRows - 1) / kRows, whole = nb & ~3;
    for (int j = 0; j < ngrp; ++j) {
        // snake order over the warps (the groups' lengths fall with j), started at another warp in each CTA
        const int pos = j % NW;
        if ((((j / NW) & 1 ? NW - 1 - pos : pos) + (int)blockIdx.x) % NW != warp) continue;
        const int a0 = j * kRows;
        const double2 *cp[Q];   // this lane's rows
#pragma unroll
        for (int q = 0; q < Q; ++q) cp[q] = C + (int64_t)(ra0 + min(a0 + 8 * q + g, na - 1)) * M + cb0;
        double re[Q][4], im[Q][4];
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int e = 0; e < 4; ++e) re[q][e] = im[q][e] = 0.0;
        int b = diag ? a0 : 0;
        const double2 *hp = hb + (b + t) * kPtsPad + g;
        const double2 *hend = hb + (((nb + 15) & ~15) - 4 + t) * kPtsPad + g;
        double2 c0[Q], c1[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            c0[q] = __ldg(cp[q] + min(b + t, nb - 1));
            c1[q] = __ldg(cp[q] + min(b + 4 + t, nb - 1));
        }
        double2 n0 = hp[0], n1 = hp[8];
        if (diag) {   // the group's own columns: left of the diagonal nothing counts
            const int bend = min(a0 + kRows, nb);
            for (; b < bend; b += 4) {
                const double2 h0 = n0, h1 = n1;
                hp = hp < hend ? hp + 4 * kPtsPad : hp;
                n0 = hp[0];
                n1 = hp[8];
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    double2 x = c0[q];
                    c0[q] = c1[q];
                    c1[q] = __ldg(cp[q] + min(b + 8 + t, nb - 1));
                    const int d = b + t - a0 - 8 * q - g;   // column less row
                    if (d <= 0 || b + t >= nb) x = make_double2(d == 0 && with_diag && b + t < nb ? 0.5 * x.x : 0.0, 0.0);
                    if (b >= a0 + 8 * q) {
                        mma_f64(re[q], h0.x, h1.x, h0.y, h1.y, x.x, -x.y);
                        mma_f64(im[q], h0.x, h1.x, h0.y, h1.y, x.y, x.x);
                    }
                }
            }
        }
#pragma unroll 2
        for (; b < whole; b += 4) {
            const double2 h0 = n0, h1 = n1;
            hp = hp < hend ? hp + 4 * kPtsPad : hp;
            n0 = hp[0];
            n1 = hp[8];
            const int o = min(b + 8 + t, nb - 1);
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const double2 x = c0[q];
                c0[q] = c1[q];
                c1[q] = __ldg(cp[q] + o);
                mma_f64(re[q], h0.x, h1.x, h0.y, h1.y, x.x, -x.y);
                mma_f64(im[q], h0.x, h1.x, h0.y, h1.y, x.y, x.x);
            }
        }
        if (b < nb) {   // one to three columns left
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const double2 x = b + t < nb ? c0[q] : make_double2(0.0, 0.0);
                mma_f64(re[q], n0.x, n1.x, n0.y, n1.y, x.x, -x.y);
                mma_f64(im[q], n0.x, n1.x, n0.y, n1.y, x.y, x.x);
            }
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (a0 + 8 * q + 2 * t + e >= na) break;   // no such row
                const double2 *r = ha + (a0 + 8 * q + 2 * t + e) * kPtsPad + g;
                double2 h = r[0];
                off0 = fma(h.x, re[q][e], fma(h.y, im[q][e], off0));
                h = r[8];
                off1 = fma(h.x, re[q][2 + e], fma(h.y, im[q][2 + e], off1));
            }
        }
    }
}

// Normalisation of the steering type (acoular/fastFuncs.py:293-310) and clipping of negatives.
__device__ __forceinline__ void finish_plain(const MapArgs &a, double scalar, double S, double r0, int bin, int64_t g,
                                             double *out_map, double *out_norm)
{
    const double Md = (double)a.M;
    double res, ns;
    if (a.steer_type == 0) {   // custom steering: no steering normalisation, S = sum |h|^2
        ns = S;
        res = scalar * a.norm;
    } else if (a.steer_type == 1) {
        ns = 1.0 / Md;
        res = scalar / (Md * Md) * a.norm;
    } else if (a.steer_type == 2) {
        const double nf = Md * r0;
        const double nf2 = nf * nf;
        ns = S / nf2;
        res = scalar / nf2 * a.norm;
    } else if (a.steer_type == 3) {
        const double nf = r0 * S;
        ns = 1.0 / (r0 * r0) / S;
        res = scalar / (nf * nf) * a.norm;
    } else {
        const double nf = Md * S;
        ns = 1.0 / Md;
        res = scalar / nf * a.norm;
    }
    if (a.clip && res < 0.0) res = 0.0;
    out_map[(int64_t)bin * a.G + g] = res;
    if (out_norm) out_norm[(int64_t)bin * a.G + g] = ns;
}

// Cross-warp sums of a point's quadratic form and steering normalisation, in a fixed order.
template <int NW>
struct TileSums {
    double off[NW][kPts];
    double s[2 * NW][kPts];
};

template <bool USE_RM, bool CUSTOM, int NW>
__device__ __forceinline__ void put_sums(TileSums<NW> &red, double off0, double off1, double (&S)[kPts / NW])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        off0 += __shfl_xor_sync(0xffffffffu, off0, o);
        off1 += __shfl_xor_sync(0xffffffffu, off1, o);
    }
    if ((lane & 3) == 0) {
        red.off[warp][lane >> 2] = off0;
        red.off[warp][(lane >> 2) + 8] = off1;
    }
    if (USE_RM || CUSTOM) {
#pragma unroll
        for (int i = 0; i < kPts / NW; ++i) {
            double v = S[i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) red.s[0][warp + NW * i] = v;
        }
    } else {
        red.s[threadIdx.x / kPts][threadIdx.x & (kPts - 1)] = S[0];
    }
}

template <bool USE_RM, bool CUSTOM, int NW>
__device__ __forceinline__ void get_sums(const TileSums<NW> &red, int p, double &o, double &S)
{
    o = S = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) o += red.off[w][p];
#pragma unroll
    for (int w = 0; w < (USE_RM || CUSTOM ? 1 : 2 * NW); ++w) S += red.s[w][p];
}

template <bool USE_RM, bool CUSTOM>
__device__ __forceinline__ double ref_distance(const MapArgs &a, const double *r0_in, int64_t g, double g0, double g1,
                                               double g2)
{
    if (CUSTOM) return 0.0;
    if (a.ref_mode == 1) return a.ref_dist;
    if (USE_RM) return r0_in[g];
    return dist3(g0, g1, g2, a.ref0, a.ref1, a.ref2);
}

// Full-CSM map.  Mics in chunks of `mc` (one chunk for all of them where their steering fits shared memory: then
// every steering value is synthesised once; else the chunk pairs a <= b are walked and the steering of chunk b is
// synthesised again for each).
template <bool USE_RM, bool CUSTOM, int NW>
__global__ void __launch_bounds__(32 * NW, NW == 4 ? 4 : 2) map_f64_kernel(MapArgs a, const double2 *__restrict__ csm,
                                                          const double *__restrict__ wavenumber, double k_scalar,
                                                          const double *__restrict__ mpos,
                                                          const double *__restrict__ gpos,
                                                          const double *__restrict__ r0_in,
                                                          const double *__restrict__ rm, int mc,
                                                          double *__restrict__ out_map, double *__restrict__ out_norm,
                                                          const double2 *__restrict__ steer)
{
    extern __shared__ double2 map_sm[];
    __shared__ TileSums<NW> red;
    double2 *ha = map_sm;                                          // [mc to 16][kPtsPad]
    double2 *hb = ha + (size_t)((mc + 15) & ~15) * kPtsPad;         // the same, only if M > mc
    const int M = a.M, bin = blockIdx.y;
    const int64_t gb = (int64_t)blockIdx.x * kPts;
    const int64_t g = gb + (threadIdx.x & (kPts - 1));
    const double k = wavenumber ? wavenumber[bin] : k_scalar;
    const double2 *C = csm + (int64_t)bin * M * M;
    const double2 *hv = CUSTOM ? steer + (int64_t)bin * a.G * M : nullptr;
    const SincosTable sct = sincos_table(a.table, a.table_mask, !CUSTOM && a.faithful != 0);
    double g0 = 0, g1 = 0, g2 = 0;
    if (g < a.G && !USE_RM && !CUSTOM) {
        g0 = gpos[g];
        g1 = gpos[a.G + g];
        g2 = gpos[2 * a.G + g];
    }
    double S[kPts / NW];
#pragma unroll
    for (int i = 0; i < kPts / NW; ++i) S[i] = 0.0;
    double off0 = 0.0, off1 = 0.0;
    for (int ma0 = 0; ma0 < M; ma0 += mc) {
        const int na = min(mc, M - ma0);
        if (ma0) __syncthreads();   // the previous chunk's readers
        synth_tile<USE_RM, CUSTOM, NW>(a, sct, rm, k, gb, g0, g1, g2, mpos, hv, ma0, na, ha, true, S);
        __syncthreads();
        quad_tile<NW, 2>(C, M, ha, ma0, na, ha, ma0, na, true, a.r_diag == 0, off0, off1);
        for (int mb0 = ma0 + mc; mb0 < M; mb0 += mc) {
            const int nb = min(mc, M - mb0);
            __syncthreads();
            synth_tile<USE_RM, CUSTOM, NW>(a, sct, rm, k, gb, g0, g1, g2, mpos, hv, mb0, nb, hb, false, S);
            __syncthreads();
            quad_tile<NW, 2>(C, M, ha, ma0, na, hb, mb0, nb, false, false, off0, off1);
        }
    }
    put_sums<USE_RM, CUSTOM, NW>(red, off0, off1, S);
    __syncthreads();
    if (threadIdx.x < kPts && g < a.G) {
        double o, sn;
        get_sums<USE_RM, CUSTOM, NW>(red, threadIdx.x, o, sn);
        finish_plain(a, 2.0 * o, sn, ref_distance<USE_RM, CUSTOM>(a, r0_in, g, g0, g1, g2), bin, g, out_map, out_norm);
    }
}

// ------------------------------------------------------------------------------------------------
// Eigenvalue form of _freqBeamformer_EigValues (acoular/fastFuncs.py:313-411): with eigenvalues
// lambda_e and eigenvectors V[:, e] of the CSM (E of them),
//     scalar = sum_e lambda_e (|sum_m conj(V[m][e]) h[m]|^2 - [r_diag] sum_m |conj(V[m][e]) h[m]|^2),
// then the steering-type normalisation of the full-CSM form.  Same steering synthesis as the full-CSM form;
// the projections T = H conj(V) are a matrix product on the FP64 matrix instruction, a warp per group of 16
// eigenvectors, squared and weighted in the epilogue (no cancellation: each term is a square times lambda_e).
// The diagonal's part is sum_m |h_m|^2 w_m with w_m = sum_e lambda_e |V[m][e]|^2.  Cost O(G M E) per bin.
// Bound: the FP64 pipe (8 M E flop per point and bin).  Measured (B200): 64 bins x 3721 points x 112 mics and
// components 7.2 -> 1.09 ms (the earlier form read every eigenvector entry as a broadcast for 32 points).
// ------------------------------------------------------------------------------------------------
template <bool USE_RM, bool CUSTOM, int NW>
__global__ void __launch_bounds__(32 * NW) map_eig_kernel(MapArgs a, int E, const double *__restrict__ eigval,
                                                          const double2 *__restrict__ eigvec,
                                                          const double *__restrict__ wavenumber, double k_scalar,
                                                          const double *__restrict__ mpos,
                                                          const double *__restrict__ gpos,
                                                          const double *__restrict__ r0_in,
                                                          const double *__restrict__ rm, int mc,
                                                          double *__restrict__ out_map, double *__restrict__ out_norm,
                                                          const double2 *__restrict__ steer,
                                                          const int *__restrict__ active)
{
    extern __shared__ double2 map_sm[];
    __shared__ TileSums<NW> red;
    const int bin = blockIdx.y;
    if (active && !active[bin]) return;   // a bin whose iteration has stopped (CLEAN-SC)
    const int M = a.M;
    double2 *hs = map_sm;                                                       // [mc to 16][kPtsPad]
    double *wd = reinterpret_cast<double *>(hs + (size_t)((mc + 15) & ~15) * kPtsPad);   // [mc], with r_diag only
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gl = lane >> 2, t = lane & 3;
    const int64_t gb = (int64_t)blockIdx.x * kPts;
    const int64_t g = gb + (threadIdx.x & (kPts - 1));
    const double k = wavenumber ? wavenumber[bin] : k_scalar;
    const double *lam = eigval + (int64_t)bin * E;
    const double2 *V = eigvec + (int64_t)bin * M * E;
    const double2 *hv = CUSTOM ? steer + (int64_t)bin * a.G * M : nullptr;
    const SincosTable sct = sincos_table(a.table, a.table_mask, !CUSTOM && a.faithful != 0);
    double g0 = 0, g1 = 0, g2 = 0;
    if (g < a.G && !USE_RM && !CUSTOM) {
        g0 = gpos[g];
        g1 = gpos[a.G + g];
        g2 = gpos[2 * a.G + g];
    }
    double S[kPts / NW];
#pragma unroll
    for (int i = 0; i < kPts / NW; ++i) S[i] = 0.0;
    double off0 = 0.0, off1 = 0.0;
    // passes of NW groups of 16 eigenvectors; the steering stays in shared memory over the passes when it is one chunk
    for (int e0 = 0; e0 < E; e0 += NW * kGroup) {
        const int eb = e0 + ((warp + (int)blockIdx.x) % NW) * kGroup;   // this warp's eigenvectors
        double re0[4] = {0, 0, 0, 0}, im0[4] = {0, 0, 0, 0}, re1[4] = {0, 0, 0, 0}, im1[4] = {0, 0, 0, 0};
        for (int m0 = 0; m0 < M; m0 += mc) {
            const int n = min(mc, M - m0);
            if (e0 == 0 || mc < M) {
                if (e0 || m0) __syncthreads();   // the previous chunk's readers
                synth_tile<USE_RM, CUSTOM, NW>(a, sct, rm, k, gb, g0, g1, g2, mpos, hv, m0, n, hs, e0 == 0, S);
                if (a.r_diag && e0 == 0)
                    for (int m = warp; m < n; m += NW) {
                        double w = 0.0;
                        for (int e = lane; e < E; e += 32) {
                            const double2 v = __ldg(V + (int64_t)(m0 + m) * E + e);
                            w += lam[e] * (v.x * v.x + v.y * v.y);
                        }
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
                        if (lane == 0) wd[m] = w;
                    }
                __syncthreads();
                if (a.r_diag && e0 == 0)
                    for (int m = warp * 4 + t; m < n; m += NW * 4) {
                        const double2 h0 = hs[m * kPtsPad + gl], h1 = hs[m * kPtsPad + gl + 8];
                        off0 -= (h0.x * h0.x + h0.y * h0.y) * wd[m];
                        off1 -= (h1.x * h1.x + h1.y * h1.y) * wd[m];
                    }
            }
            if (eb < E) {
                // eigenvectors and mics past the end repeat the last one (their lambda is not read, their
                // steering is zero)
                const double2 *vx = V + (int64_t)m0 * E + min(eb + gl, E - 1);
                const double2 *vy = V + (int64_t)m0 * E + min(eb + 8 + gl, E - 1);
                auto load = [&](int m, double2 &x, double2 &y) {
                    const int64_t o = (int64_t)min(m, n - 1) * E;
                    x = __ldg(vx + o);
                    y = __ldg(vy + o);
                };
                double2 x0, y0, x1, y1;
                load(t, x0, y0);
                load(4 + t, x1, y1);
                for (int m = 0; m < n; m += 4) {
                    const double2 h0 = hs[(m + t) * kPtsPad + gl], h1 = hs[(m + t) * kPtsPad + gl + 8];
                    const double2 x = x0, y = y0;
                    x0 = x1;
                    y0 = y1;
                    load(m + 8 + t, x1, y1);
                    // conj(V) h: re = v.x h.x + v.y h.y, im = v.x h.y - v.y h.x
                    mma_f64(re0, h0.x, h1.x, h0.y, h1.y, x.x, x.y);
                    mma_f64(im0, h0.x, h1.x, h0.y, h1.y, -x.y, x.x);
                    if (eb + 8 < E) {
                        mma_f64(re1, h0.x, h1.x, h0.y, h1.y, y.x, y.y);
                        mma_f64(im1, h0.x, h1.x, h0.y, h1.y, -y.y, y.x);
                    }
                }
            }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int q0 = eb + 2 * t + e, q1 = q0 + 8;
            if (q0 < E) {
                const double l = lam[q0];
                off0 = fma(l, re0[e] * re0[e] + im0[e] * im0[e], off0);
                off1 = fma(l, re0[2 + e] * re0[2 + e] + im0[2 + e] * im0[2 + e], off1);
            }
            if (q1 < E) {
                const double l = lam[q1];
                off0 = fma(l, re1[e] * re1[e] + im1[e] * im1[e], off0);
                off1 = fma(l, re1[2 + e] * re1[2 + e] + im1[2 + e] * im1[2 + e], off1);
            }
        }
    }
    put_sums<USE_RM, CUSTOM, NW>(red, off0, off1, S);
    __syncthreads();
    if (threadIdx.x < kPts && g < a.G) {
        double sc, sn;
        get_sums<USE_RM, CUSTOM, NW>(red, threadIdx.x, sc, sn);
        finish_plain(a, sc, sn, ref_distance<USE_RM, CUSTOM>(a, r0_in, g, g0, g1, g2), bin, g, out_map, out_norm);
    }
}

// Eigenvalue form for a few components (E <= kEigSmall, e.g. BeamformerEig's default n = -1 and each
// CLEAN-SC iteration's single component): one thread per grid point and NB bins walks the mics in order,
// computes a mic's distance and weight once, synthesises the steering value of each bin and accumulates the
// projections and the normalisation sum in registers.  Each component's mic sum runs in the reference's order.
// Bound: issue slots of the steering synthesis.  Measured (B200): 16 bins x 160,801 points x 256 mics 5.1 -> 3.7 ms
// with four bins per thread and their table lookups in flight together (two bins: 3.8 too; one: 4.5).
constexpr int kEigSmall = 4;
constexpr int kEigSmallThreads = 128;

template <bool USE_RM, bool CUSTOM, int EMAX, int NB>
__global__ void __launch_bounds__(kEigSmallThreads)
    map_eig_small_kernel(MapArgs a, int nbins, int E, const double *__restrict__ eigval,
                         const double2 *__restrict__ eigvec, const double *__restrict__ wavenumber, double k_scalar,
                         const double *__restrict__ mpos, const double *__restrict__ gpos,
                         const double *__restrict__ r0_in, const double *__restrict__ rm,
                         double *__restrict__ out_map, double *__restrict__ out_norm,
                         const double2 *__restrict__ steer, const int *__restrict__ active)
{
    const int bin0 = blockIdx.y * NB;
    if (active && !active[bin0]) return;   // a bin whose iteration has stopped (CLEAN-SC; NB = 1 there)
    const int64_t g = (int64_t)blockIdx.x * kEigSmallThreads + threadIdx.x;
    if (g >= a.G) return;
    const int M = a.M;
    const SincosTable sct = sincos_table(a.table, a.table_mask, !CUSTOM && a.faithful != 0);
    double k[NB];
    const double2 *V[NB];
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        const int bin = min(bin0 + q, nbins - 1);   // the last group repeats its last bin; not written twice
        k[q] = wavenumber ? wavenumber[bin] : k_scalar;
        V[q] = eigvec + (int64_t)bin * M * E;
    }
    const double2 *hv = CUSTOM ? steer + ((int64_t)bin0 * a.G + g) * M : nullptr;
    double g0 = 0, g1 = 0, g2 = 0;
    if (!USE_RM && !CUSTOM) {
        g0 = gpos[g];
        g1 = gpos[a.G + g];
        g2 = gpos[2 * a.G + g];
    }
    double fr[NB][EMAX], fi[NB][EMAX], dg[NB][EMAX];
#pragma unroll
    for (int q = 0; q < NB; ++q)
#pragma unroll
        for (int j = 0; j < EMAX; ++j) fr[q][j] = fi[q][j] = dg[q][j] = 0.0;
    double S = 0.0;
    for (int m = 0; m < M; ++m) {
        double r = 0.0, w = 0.0;
        if (!CUSTOM) {
            if (USE_RM) {
                r = __ldg(rm + g * M + m);
                w = steer_weight(a.steer_type, r);
            } else {
                r = dist3_weight(a.steer_type, g0, g1, g2, __ldg(mpos + m), __ldg(mpos + M + m),
                                 __ldg(mpos + 2 * M + m), w);
            }
            S = fma(w, w, S);
        }
        constexpr int KP = NB < 2 ? NB : 2;   // all four at once spill (5.36 -> 5.62 ms); pairs 5.30
        SincosPending<KP> pend[NB / KP];
        if (!CUSTOM) {
#pragma unroll
            for (int q = 0; q < NB; ++q) pend[q / KP].x[q % KP] = steer_phase(k[q], r);
#pragma unroll
            for (int q = 0; q < NB / KP; ++q) sincos_begin(pend[q], sct);
#pragma unroll
            for (int q = 0; q < NB / KP; ++q) sincos_finish(pend[q], sct);
        }
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            double2 h;
            if (CUSTOM) {
                h = __ldg(hv + m);
                S += fma(h.x, h.x, __dmul_rn(h.y, h.y));
            } else {
                h = steer_value(a.steer_type, pend[q / KP].c[q % KP], pend[q / KP].s[q % KP], w);
            }
            const double2 *vrow = V[q] + (int64_t)m * E;
#pragma unroll
            for (int j = 0; j < EMAX; ++j) {
                if (j >= E) break;
                const double2 v = __ldg(vrow + j);
                // temp1 = conj(V[m][e]) * h[m]; the FMAs are spelled out, so that every instance of this kernel
                // gives the same bits
                const double tr = fma(v.x, h.x, __dmul_rn(v.y, h.y)), ti = fma(v.x, h.y, -__dmul_rn(v.y, h.x));
                fr[q][j] += tr;
                fi[q][j] += ti;
                if (a.r_diag) dg[q][j] = fma(tr, tr, fma(ti, ti, dg[q][j]));
            }
        }
    }
    const double r0 = ref_distance<USE_RM, CUSTOM>(a, r0_in, g, g0, g1, g2);
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        if (bin0 + q >= nbins) break;
        const double *lam = eigval + (int64_t)(bin0 + q) * E;
        double scal = 0.0;
#pragma unroll
        for (int j = 0; j < EMAX; ++j) {
            if (j >= E) break;
            const double full = fma(fr[q][j], fr[q][j], __dmul_rn(fi[q][j], fi[q][j]));
            scal = fma(a.r_diag ? full - dg[q][j] : full, lam[j], scal);
        }
        finish_plain(a, scal, S, r0, bin0 + q, g, out_map, out_norm);
    }
}

static int make_args(const acb_map_params *p, MapArgs &a)
{
    if (!p) return ACB_ERR_ARG;
    if (p->num_mics < 2 || p->num_mics > 2048 || p->num_grid <= 0 || p->num_bins <= 0 || p->num_bins > 65535)
        return ACB_ERR_SHAPE;
    if (p->steer_type < 1 || p->steer_type > 4) return ACB_ERR_ARG;
    if (p->glibc_faithful && (!p->sincos_table || p->sincos_table_slots <= 0 ||
                              (p->sincos_table_slots & (p->sincos_table_slots - 1))))
        return ACB_ERR_ARG;
    a.M = p->num_mics;
    a.G = p->num_grid;
    a.steer_type = p->steer_type;
    a.r_diag = p->r_diag;
    a.clip = p->clip_negative;
    a.norm = p->norm;
    a.ref_mode = p->ref_mode;
    a.ref0 = p->ref_point[0];
    a.ref1 = p->ref_point[1];
    a.ref2 = p->ref_point[2];
    a.ref_dist = p->ref_distance;
    a.faithful = p->glibc_faithful;
    a.table = p->sincos_table;
    a.table_mask = p->glibc_faithful ? (uint64_t)p->sincos_table_slots - 1 : 0;
    return ACB_OK;
}

// Chunk of mics whose steering tile a CTA holds, and the warps per CTA.  All mics in one tile up to 768 (221 KB);
// above, pairs of 384-mic tiles.  Four warps per CTA up to 256 mics (three CTAs or more per SM, so that one's
// synthesis runs under another's matrix products), eight where only one or two CTAs fit.
constexpr int kMapOneTile = 768, kMapPairTile = 384, kMapFourWarps = 256;
// the largest tile, with the eigenvalue form's diagonal
constexpr size_t kMapSmem = kMapOneTile * (kPtsPad * sizeof(double2) + sizeof(double));

template <bool USE_RM, bool CUSTOM, int NW>
static int launch_map_nw(const MapArgs &a, int nbins, const void *csm, const double *k, double k_scalar,
                         const double *mpos, const double *gpos, const double *r0, const double *rm, double *out_map,
                         double *out_norm, cudaStream_t s, const void *steer)
{
    const int mc = a.M <= kMapOneTile ? a.M : kMapPairTile;
    const size_t smem = (size_t)(a.M <= mc ? 1 : 2) * ((mc + 15) & ~15) * kPtsPad * sizeof(double2);
    auto kern = map_f64_kernel<USE_RM, CUSTOM, NW>;
    if (const int st = allow_smem(kern, smem, kMapSmem)) return st;
    const dim3 grid((unsigned)((a.G + kPts - 1) / kPts), nbins);
    kern<<<grid, 32 * NW, smem, s>>>(a, reinterpret_cast<const double2 *>(csm), k, k_scalar, mpos, gpos, r0, rm, mc,
                                     out_map, out_norm, reinterpret_cast<const double2 *>(steer));
    return check_launch();
}

template <bool USE_RM, bool CUSTOM = false>
static int launch_plain(const MapArgs &a, int nbins, const void *csm, const double *k, double k_scalar,
                        const double *mpos, const double *gpos, const double *r0, const double *rm, double *out_map,
                        double *out_norm, cudaStream_t s, const void *steer = nullptr)
{
    if (a.M <= kMapFourWarps)
        return launch_map_nw<USE_RM, CUSTOM, 4>(a, nbins, csm, k, k_scalar, mpos, gpos, r0, rm, out_map, out_norm, s,
                                                steer);
    return launch_map_nw<USE_RM, CUSTOM, 8>(a, nbins, csm, k, k_scalar, mpos, gpos, r0, rm, out_map, out_norm, s,
                                            steer);
}

template <bool USE_RM, bool CUSTOM, int NW>
static int launch_eig_nw(const MapArgs &a, int nbins, int E, const double *eigval, const void *eigvec, const double *k,
                         double k_scalar, const double *mpos, const double *gpos, const double *r0, const double *rm,
                         double *out_map, double *out_norm, cudaStream_t s, const void *steer, const int *active)
{
    const int mc = a.M <= kMapOneTile ? a.M : kMapPairTile;
    const size_t smem = (size_t)((mc + 15) & ~15) * kPtsPad * sizeof(double2) + (a.r_diag ? mc * sizeof(double) : 0);
    auto kern = map_eig_kernel<USE_RM, CUSTOM, NW>;
    if (const int st = allow_smem(kern, smem, kMapSmem)) return st;
    const dim3 grid((unsigned)((a.G + kPts - 1) / kPts), nbins);
    kern<<<grid, 32 * NW, smem, s>>>(a, E, eigval, reinterpret_cast<const double2 *>(eigvec), k, k_scalar, mpos, gpos,
                                     r0, rm, mc, out_map, out_norm, reinterpret_cast<const double2 *>(steer), active);
    return check_launch();
}

template <bool USE_RM, bool CUSTOM, int EMAX, int NB>
static int launch_eig_small(const MapArgs &a, int nbins, int E, const double *eigval, const void *eigvec,
                            const double *k, double k_scalar, const double *mpos, const double *gpos, const double *r0,
                            const double *rm, double *out_map, double *out_norm, cudaStream_t s, const void *steer,
                            const int *active)
{
    const dim3 grid((unsigned)((a.G + kEigSmallThreads - 1) / kEigSmallThreads), (nbins + NB - 1) / NB);
    map_eig_small_kernel<USE_RM, CUSTOM, EMAX, NB><<<grid, kEigSmallThreads, 0, s>>>(
        a, nbins, E, eigval, reinterpret_cast<const double2 *>(eigvec), k, k_scalar, mpos, gpos, r0, rm, out_map,
        out_norm, reinterpret_cast<const double2 *>(steer), active);
    return check_launch();
}

template <bool USE_RM, bool CUSTOM = false>
static int launch_eig(const MapArgs &a, int nbins, int E, const double *eigval, const void *eigvec, const double *k,
                      double k_scalar, const double *mpos, const double *gpos, const double *r0, const double *rm,
                      double *out_map, double *out_norm, cudaStream_t s, const void *steer = nullptr,
                      const int *active = nullptr)
{
#define ACB_EIG_ARGS a, nbins, E, eigval, eigvec, k, k_scalar, mpos, gpos, r0, rm, out_map, out_norm, s, steer, active
    if (E == 1) {
        // four bins per thread share the distances, as long as that leaves every SM eight CTAs (32 warps)
        if (!CUSTOM && !active && (a.G + kEigSmallThreads - 1) / kEigSmallThreads * ((nbins + 3) / 4) >= 8 * kNumSMs)
            return launch_eig_small<USE_RM, CUSTOM, 1, CUSTOM ? 1 : 4>(ACB_EIG_ARGS);
        return launch_eig_small<USE_RM, CUSTOM, 1, 1>(ACB_EIG_ARGS);
    }
    if (E <= kEigSmall) return launch_eig_small<USE_RM, CUSTOM, kEigSmall, 1>(ACB_EIG_ARGS);
    if (a.M <= kMapFourWarps) return launch_eig_nw<USE_RM, CUSTOM, 4>(ACB_EIG_ARGS);
    return launch_eig_nw<USE_RM, CUSTOM, 8>(ACB_EIG_ARGS);
#undef ACB_EIG_ARGS
}

// Launchers for other translation units (map_internal.h).
int map_plain_launch(const acb_map_params *p, int nbins, const void *csm, const double *k, const double *mpos,
                     const double *gpos, const double *r0, const double *rm, double *out_map, cudaStream_t s)
{
    MapArgs a;
    const int rc = make_args(p, a);
    if (rc != ACB_OK) return rc;
    if (rm) {
        a.ref_mode = 0;   // r0 is given
        return launch_plain<true>(a, nbins, csm, k, 0.0, nullptr, nullptr, r0, rm, out_map, nullptr, s);
    }
    return launch_plain<false>(a, nbins, csm, k, 0.0, mpos, gpos, nullptr, nullptr, out_map, nullptr, s);
}

int map_eig_launch(const acb_map_params *p, int nbins, int E, const double *eigval, const void *eigvec,
                   const double *k, const double *mpos, const double *gpos, const double *r0, const double *rm,
                   double *out_map, const int *active, cudaStream_t s)
{
    MapArgs a;
    const int rc = make_args(p, a);
    if (rc != ACB_OK) return rc;
    if (rm) {
        a.ref_mode = 0;
        return launch_eig<true>(a, nbins, E, eigval, eigvec, k, 0.0, nullptr, nullptr, r0, rm, out_map, nullptr, s,
                                nullptr, active);
    }
    return launch_eig<false>(a, nbins, E, eigval, eigvec, k, 0.0, mpos, gpos, nullptr, nullptr, out_map, nullptr, s,
                             nullptr, active);
}

int map_eig_custom_launch(const acb_map_params *p, int nbins, int E, const double *eigval, const void *eigvec,
                          const void *steer, double *out_map, const int *active, cudaStream_t s);

}  // namespace acb

using namespace acb;

extern "C" {

int acb_map_f64(const acb_map_params *p, const void *csm, const double *wavenumber, const double *mpos,
                const double *gpos, double *out_map, double *out_steer_norm, int * /*error_word: no device-side wait*/,
                void *stream)
{
    MapArgs a;
    int st = make_args(p, a);
    if (st) return st;
    if (!csm || !wavenumber || !mpos || !gpos || !out_map) return ACB_ERR_ARG;
    if ((a.G + kPts - 1) / kPts > 0x7fffffffLL) return ACB_ERR_SHAPE;
    return launch_plain<false>(a, p->num_bins, csm, wavenumber, 0.0, mpos, gpos, nullptr, nullptr, out_map,
                               out_steer_norm, as_stream(stream));
}

int acb_map_eig_f64(const acb_map_params *p, int num_eigs, const double *eigval, const void *eigvec,
                    const double *wavenumber, const double *mpos, const double *gpos, double *out_map,
                    double *out_steer_norm, void *stream)
{
    MapArgs a;
    int st = make_args(p, a);
    if (st) return st;
    if (!eigval || !eigvec || !wavenumber || !mpos || !gpos || !out_map) return ACB_ERR_ARG;
    if (num_eigs < 1 || num_eigs > p->num_mics) return ACB_ERR_SHAPE;
    if ((a.G + kPts - 1) / kPts > 0x7fffffffLL) return ACB_ERR_SHAPE;
    return launch_eig<false>(a, p->num_bins, num_eigs, eigval, eigvec, wavenumber, 0.0, mpos, gpos, nullptr, nullptr,
                             out_map, out_steer_norm, as_stream(stream));
}

int acb_beamformer_freq_eig_f64(const acb_map_params *p, int num_eigs, const double *eigval, const void *eigvec,
                                double wavenumber, const double *r0, const double *rm, double *out_map,
                                double *out_steer_norm, void *stream)
{
    MapArgs a;
    int st = make_args(p, a);
    if (st) return st;
    if (p->num_bins != 1) return ACB_ERR_SHAPE;
    if (!eigval || !eigvec || !r0 || !rm || !out_map) return ACB_ERR_ARG;
    if (num_eigs < 1 || num_eigs > p->num_mics) return ACB_ERR_SHAPE;
    a.ref_mode = 0;
    return launch_eig<true>(a, 1, num_eigs, eigval, eigvec, nullptr, wavenumber, nullptr, nullptr, r0, rm, out_map,
                            out_steer_norm, as_stream(stream));
}

int acb_map_rm_f64(const acb_map_params *p, const void *csm, const double *wavenumber, const double *r0,
                   const double *rm, double *out_map, double *out_steer_norm, void *stream)
{
    MapArgs a;
    int st = make_args(p, a);
    if (st) return st;
    if (!csm || !wavenumber || !r0 || !rm || !out_map) return ACB_ERR_ARG;
    if ((a.G + kPts - 1) / kPts > 0x7fffffffLL) return ACB_ERR_SHAPE;
    a.ref_mode = 0;
    return launch_plain<true>(a, p->num_bins, csm, wavenumber, 0.0, nullptr, nullptr, r0, rm, out_map, out_steer_norm,
                              as_stream(stream));
}

// Custom steering: p->steer_type is ignored; steer: complex128 [num_bins][G][M].
static int custom_args(const acb_map_params *p, MapArgs &a)
{
    if (!p) return ACB_ERR_ARG;
    acb_map_params q = *p;
    q.steer_type = 1;            // any valid type for the shared checks; replaced below
    q.glibc_faithful = 0;        // the steering is given: no phase synthesis
    int st = make_args(&q, a);
    if (st) return st;
    a.steer_type = 0;
    return ACB_OK;
}

int acb_map_custom_f64(const acb_map_params *p, const void *csm, const void *steer, double *out_map,
                       double *out_steer_norm, void *stream)
{
    MapArgs a;
    int st = custom_args(p, a);
    if (st) return st;
    if (!csm || !steer || !out_map) return ACB_ERR_ARG;
    if ((a.G + kPts - 1) / kPts > 0x7fffffffLL) return ACB_ERR_SHAPE;
    return launch_plain<false, true>(a, p->num_bins, csm, nullptr, 0.0, nullptr, nullptr, nullptr, nullptr, out_map,
                                     out_steer_norm, as_stream(stream), steer);
}

int acb_map_eig_custom_f64(const acb_map_params *p, int num_eigs, const double *eigval, const void *eigvec,
                           const void *steer, double *out_map, double *out_steer_norm, void *stream)
{
    MapArgs a;
    int st = custom_args(p, a);
    if (st) return st;
    if (!eigval || !eigvec || !steer || !out_map) return ACB_ERR_ARG;
    if (num_eigs < 1 || num_eigs > p->num_mics) return ACB_ERR_SHAPE;
    if ((a.G + kPts - 1) / kPts > 0x7fffffffLL) return ACB_ERR_SHAPE;
    return launch_eig<false, true>(a, p->num_bins, num_eigs, eigval, eigvec, nullptr, 0.0, nullptr, nullptr, nullptr,
                                   nullptr, out_map, out_steer_norm, as_stream(stream), steer);
}

int acb_beamformer_freq_f64(const acb_map_params *p, const void *csm, double wavenumber, const double *r0,
                            const double *rm, double *out_map, double *out_steer_norm, void *stream)
{
    MapArgs a;
    int st = make_args(p, a);
    if (st) return st;
    if (p->num_bins != 1) return ACB_ERR_SHAPE;
    if (!csm || !r0 || !rm || !out_map) return ACB_ERR_ARG;
    a.ref_mode = 0;
    st = launch_plain<true>(a, 1, csm, nullptr, wavenumber, nullptr, nullptr, r0, rm, out_map, out_steer_norm,
                            as_stream(stream));
    return st;
}

}  // extern "C"

namespace acb {

int map_eig_custom_launch(const acb_map_params *p, int nbins, int E, const double *eigval, const void *eigvec,
                          const void *steer, double *out_map, const int *active, cudaStream_t s)
{
    MapArgs a;
    const int rc = custom_args(p, a);
    if (rc != ACB_OK) return rc;
    return launch_eig<false, true>(a, nbins, E, eigval, eigvec, nullptr, 0.0, nullptr, nullptr, nullptr, nullptr,
                                   out_map, nullptr, s, steer, active);
}

}  // namespace acb
