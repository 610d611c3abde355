// Stage A: cross-spectral matrix estimation (PowerSpectra.calc_csm, acoular/spectra.py:366-416).
//
// Data flow per chunk of windows (all on the device, samples resident in HBM):
//   fft_window_kernel : samples [S][M] (f32|f64) -> window (FP64) -> rFFT (FP64, radix-2 in shared
//                       memory) -> spectra [bin][window][mic] rounded to the CSM precision
//   gram_f64_kernel   : csm_upper[bin][r][c] += sum_w conj(X[bin][w][c]) * X[bin][w][r], r <= c,
//   gram_c64_kernel     32x32 (FP64 matrix instruction) or 64x64 (packed FP32 FMAs) upper-triangular tiles,
//                       windows streamed through shared memory; or the finished matrix where the
//                       windows are one chunk
//   finalize_kernel   : Hermitian completion and the 2/(N*sum(w^2)*num_blocks) scale
//
// The per-element accumulation runs sequentially over windows with the same two chained FMAs per
// component that the reference's fastmath calcCSM (acoular/fastFuncs.py:53-57) compiles to, so
// given identical spectra the Welch sums are bit-identical to the reference.
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <type_traits>

#include <cuda_bf16.h>

#include "common.cuh"
#include "csm_internal.h"
#include "tc_layout.cuh"

namespace acb {

static thread_local std::string g_last_cuda_error;

void set_cuda_error(cudaError_t e) { g_last_cuda_error = cudaGetErrorString(e); }

// ------------------------------------------------------------------------------------------------
// Windowed real FFT.  One CTA = one window x `mpb` mics (a power of two); FFT of the N/2-point complex sequence
// z[j] = x[2j] + i x[2j+1], then the split into the N/2+1 real-input bins.
//
// The radix-2 DIT stages run in passes of up to three: a thread loads the 2^s points that s consecutive stages
// combine among themselves, applies the s stages' butterflies in registers and stores them back: one
// shared-memory round trip and one barrier per pass instead of per stage.  The first three stages take their points
// straight from the samples (bit-reversed order: 8 rows H/8 apart), lanes along the mics.  In the later passes a
// thread keeps its task's twiddles for all of its mics, and it reads four of the seven: the others are those times -i.
// Bound: shared memory (seven 16-byte accesses per point) and the FP64 pipe, about 0.5 ms each for 999 windows x 256
// mics x 1024 samples.  Measured (B200): that transform 2.65 -> 1.24 ms (before: two more trips through shared
// memory, a twiddle load per butterfly and runtime divisions by the mic count in the index arithmetic).  The lane order of the load
// and the paired bins of the split give 4 to 8 % of a whole CSM where few mics fit a CTA (113 mics, block 4096, 75 %
// overlap, complex64, in the six-FMA form: 995 -> 958 us; 16 mics, block 16384: 371 -> 342) and 0.2 to 1 % elsewhere.
// ------------------------------------------------------------------------------------------------
// Shared-memory slot of point j of a mic's sequence: one padding slot after every 8 points, so that
// 8 threads reading 16-byte points 8 apart (the first pass) or 64 apart hit different banks.
__device__ __forceinline__ int zp(int j) { return j + (j >> 3); }
// padded length of one mic's sequence of H points (an odd number of 16-byte slots past the padding)
__host__ __device__ constexpr int fft_stride(int H) { return H + (H >> 3) + 1; }

// (a, b) -> (a + w b, a - w b), the difference as 2 a - (a + w b): six FMAs; PLAIN: w b first, then the sum and the
// difference.  Spectra that are rounded to complex64 take the plain form with every twiddle from the table: their
// rounding then falls the same way as with one stage at a time, where the six-FMA form moves one value in 10^7 by an ulp
// (113 mics, block 4096, complex64: 957 -> 1010 us, the price of it).  So do the sub-sequences of the largest blocks.
template <bool PLAIN>
__device__ __forceinline__ void butterfly(double2 &a, double2 &b, double2 w)
{
    if (PLAIN) {
        const double br = b.x * w.x - b.y * w.y;
        const double bi = b.x * w.y + b.y * w.x;
        b = make_double2(a.x - br, a.y - bi);
        a = make_double2(a.x + br, a.y + bi);
        return;
    }
    const double re = fma(b.x, w.x, fma(-b.y, w.y, a.x)), im = fma(b.x, w.y, fma(b.y, w.x, a.y));
    b = make_double2(fma(2.0, a.x, -re), fma(2.0, a.y, -im));
    a = make_double2(re, im);
}

// Twiddles of one task of a pass of S stages, the first of length 2 half1: with tb = task mod half1, stage q uses
// W_{2 half1 2^q}^{tb + u half1}, u < 2^q; w[q] holds u = 0 and w3 u = 1 of the third stage; u + 2^{q-1} is -i times u
// (PLAIN: all from the table, u at 2^q - 1 + u).
template <int S, bool PLAIN>
struct PassTwiddles {
    double2 w[PLAIN ? (1 << S) - 1 : S], w3;
    __device__ __forceinline__ void load(int sg, int task, int logN, const double2 *__restrict__ tw)
    {
        const int half1 = 1 << sg, tb = task & (half1 - 1);
        if (PLAIN) {
#pragma unroll
            for (int q = 0; q < S; ++q)
#pragma unroll
                for (int u = 0; u < (1 << q); ++u)
                    w[(1 << q) - 1 + u] = __ldg(tw + ((tb + u * half1) << (logN - (sg + 1 + q))));
            return;
        }
#pragma unroll
        for (int q = 0; q < S; ++q) w[q] = __ldg(tw + (tb << (logN - (sg + 1 + q))));
        if (S == 3) w3 = __ldg(tw + ((tb + half1) << (logN - (sg + 3))));
    }
};

// s (1..3) consecutive radix-2 DIT stages of lengths L1 = 2^(sg + 1), 2 L1, .., on a bit-reversed
// sequence z (one mic).  Task `task` in [0, H / 2^s) owns points base + t * L1/2, t = 0 .. 2^s - 1.
template <int S, bool PLAIN>
__device__ __forceinline__ void fft_pass(double2 *__restrict__ z, int sg, int task, const PassTwiddles<S, PLAIN> &tws)
{
    const int half1 = 1 << sg;
    const int base = ((task >> sg) << (sg + S)) + (task & (half1 - 1));   // the pass spans 2^(sg + S) points
    double2 v[1 << S];
#pragma unroll
    for (int t = 0; t < (1 << S); ++t) v[t] = z[zp(base + t * half1)];
#pragma unroll
    for (int q = 0; q < S; ++q)
#pragma unroll
        for (int t = 0; t < (1 << S); ++t) {
            if (t & (1 << q)) continue;
            const int u = t & ((1 << q) - 1);
            if (PLAIN) {
                butterfly<true>(v[t], v[t + (1 << q)], tws.w[(1 << q) - 1 + u]);
                continue;
            }
            const double2 w1 = S == 3 && q == 2 && (u & 1) ? tws.w3 : tws.w[q];
            const bool rot = q > 0 && (u >> (q - 1));   // the upper half of the u: times -i
            butterfly<false>(v[t], v[t + (1 << q)], rot ? make_double2(w1.y, -w1.x) : w1);
        }
#pragma unroll
    for (int t = 0; t < (1 << S); ++t) z[zp(base + t * half1)] = v[t];
}

// The remaining stages st .. logH - 1 of `nm` sequences in shared memory.  A thread keeps one task per pass and
// its twiddles, and walks the mics (all of them, or every ngrp-th where the CTA holds ngrp threads per task).
template <int S, bool PLAIN>
__device__ __forceinline__ void fft_pass_mics(double2 *zs, int nm, int stride, int st, int logH, int logN,
                                              const double2 *__restrict__ tw)
{
    const int logT = logH - S, T = 1 << logT;   // H / 2^S tasks per mic
    const int nt = blockDim.x;
    const int grp = T < nt ? threadIdx.x >> logT : 0, ngrp = T < nt ? nt >> logT : 1;
    for (int task = T < nt ? threadIdx.x & (T - 1) : threadIdx.x; task < T; task += nt) {
        PassTwiddles<S, PLAIN> w;
        w.load(st, task, logN, tw);
        for (int ml = grp; ml < nm; ml += ngrp) fft_pass<S, PLAIN>(zs + ml * stride, st, task, w);
    }
    __syncthreads();
}

template <bool PLAIN>
__device__ __forceinline__ void fft_passes(double2 *zs, int nm, int stride, int st, int logH, int logN,
                                           const double2 *__restrict__ tw)
{
    while (st < logH) {
        const int left = logH - st;
        // four left: 2 + 2 rather than 3 + 1
        const int S = left == 4 ? 2 : (left >= 3 ? 3 : left);
        if (S == 3) fft_pass_mics<3, PLAIN>(zs, nm, stride, st, logH, logN, tw);
        else if (S == 2) fft_pass_mics<2, PLAIN>(zs, nm, stride, st, logH, logN, tw);
        else fft_pass_mics<1, PLAIN>(zs, nm, stride, st, logH, logN, tw);
        st += S;
    }
}

// The first three stages (twiddles 1, -i and the odd eighth roots) of 8 points in bit-reversed order.
__device__ __forceinline__ void first_stages(double2 (&v)[8])
{
    auto pair = [](double2 &a, double2 &b) {
        const double2 s = make_double2(a.x + b.x, a.y + b.y);
        b = make_double2(a.x - b.x, a.y - b.y);
        a = s;
    };
    auto turn = [](double2 &a) { a = make_double2(a.y, -a.x); };   // times -i
#pragma unroll
    for (int t = 0; t < 8; t += 2) pair(v[t], v[t + 1]);
#pragma unroll
    for (int t = 0; t < 8; t += 4) {
        pair(v[t], v[t + 2]);
        turn(v[t + 3]);
        pair(v[t + 1], v[t + 3]);
    }
    const double h = 0.70710678118654752440;
    pair(v[0], v[4]);
    butterfly<false>(v[1], v[5], make_double2(h, -h));
    turn(v[6]);
    pair(v[2], v[6]);
    butterfly<false>(v[3], v[7], make_double2(-h, -h));
}
// The same from the table's W_4^1, W_8^1 and W_8^3 (see butterfly).
__device__ __forceinline__ void first_stages_plain(double2 (&v)[8], double2 w41, double2 w81, double2 w83)
{
    const double2 one = make_double2(1.0, 0.0);
#pragma unroll
    for (int t = 0; t < 8; t += 2) butterfly<true>(v[t], v[t + 1], one);
#pragma unroll
    for (int t = 0; t < 8; t += 4) {
        butterfly<true>(v[t], v[t + 2], one);
        butterfly<true>(v[t + 1], v[t + 3], w41);
    }
    butterfly<true>(v[0], v[4], one);
    butterfly<true>(v[1], v[5], w81);
    butterfly<true>(v[2], v[6], w41);
    butterfly<true>(v[3], v[7], w83);
}

// The low n bits of x in reverse order.
__device__ __forceinline__ int bit_reverse(int x, int n) { return n ? (int)(__brev((unsigned)x) >> (32 - n)) : 0; }

// The pairs (u, H - u), u = u0 .. u0 + n - 1 <= H / 2, that hold the bins bin_lo .. bin_lo + nbins - 1 of 0 .. H.
struct SplitPairs {
    int u0, n;
    __device__ __forceinline__ SplitPairs(int bin_lo, int nbins, int H)
    {
        const int last = bin_lo + nbins - 1, a = min(bin_lo, H - bin_lo), b = min(last, H - last);
        u0 = min(a, b);
        n = (2 * bin_lo <= H && 2 * last >= H ? H >> 1 : max(a, b)) - u0 + 1;
    }
};

// Blocks from this size on take wide CTAs (more mics, 512 threads; see fft_mics_per_block and fft4_mics_per_block).
// (Measured, CSM of 256 mics x 300,000 samples, block 8192, complex64: 6.29 -> 5.52 ms; 113 mics, block 2048: 0.93 ->
// 0.91; block 512, 256 mics: 2.53 -> 2.65, so not below 2048.)
constexpr int FFT_WIDE_N = 2048;

// Output forms of the spectra (OUT): complex128 or complex64 [bin][window][mic] for the FP64 /
// FP32 Gram; or the tensor-core Gram's operand tiles, TF32 (OUT_TF32) or split BF16 hi + lo
// (OUT_BF16), 32 x 32 tiles [bin][window/32][component/32] with component 2m = Re, 2m + 1 = Im of
// mic m (row) and the window within the chunk (column); `R` row tiles per bin and window block,
// `KC` window blocks; BF16 lo tiles start `lo_elems` elements after the hi tiles.
enum { OUT_C128 = 0, OUT_C64 = 1, OUT_TF32 = 2, OUT_BF16 = 3 };

// Store bin `b` (relative to bin_lo) of window `wi` (within the chunk of nw windows), mic m, in form OUT.
template <int OUT>
__device__ __forceinline__ void put_bin(void *__restrict__ out, int64_t nw, int wi, int M, int m, int b, double xr,
                                        double xi, int R, int KC, int64_t lo_elems)
{
    if (OUT <= OUT_C64) {
        const int64_t o = ((int64_t)b * nw + wi) * M + m;
        if (OUT == OUT_C64)
            reinterpret_cast<float2 *>(out)[o] = make_float2(__double2float_rn(xr), __double2float_rn(xi));
        else reinterpret_cast<double2 *>(out)[o] = make_double2(xr, xi);
    } else {
        const int rowc = 2 * m, col = wi & 31;
        const int64_t tile = ((int64_t)b * KC + (wi >> 5)) * R + (rowc >> 5);
        const float fr = __double2float_rn(xr), fi = __double2float_rn(xi);
        if (OUT == OUT_TF32) {
            uint32_t *t = reinterpret_cast<uint32_t *>(out) + tile * 1024;
            t[tile_off_tf32(rowc & 31, col)] = tf32_bits(fr);
            t[tile_off_tf32((rowc & 31) + 1, col)] = tf32_bits(fi);
        } else {
            __nv_bfloat16 *t = reinterpret_cast<__nv_bfloat16 *>(out) + tile * 1024;
            const __nv_bfloat16 hr = __float2bfloat16_rn(fr), hi = __float2bfloat16_rn(fi);
            const int o0 = tile_off(rowc & 31, col), o1 = tile_off((rowc & 31) + 1, col);
            t[o0] = hr;
            t[o1] = hi;
            t[lo_elems + o0] = __float2bfloat16_rn(fr - __bfloat162float(hr));
            t[lo_elems + o1] = __float2bfloat16_rn(fi - __bfloat162float(hi));
        }
    }
}

template <typename TS, int OUT>
__global__ void __launch_bounds__(512) fft_window_kernel(const TS *__restrict__ samples, int M, int N, int hop,
                                                         int64_t w0, int64_t nw, int mpb,
                                                         const double *__restrict__ window,
                                                         const double2 *__restrict__ tw, int bin_lo, int nbins,
                                                         void *__restrict__ out, int R, int KC, int64_t lo_elems)
{
    extern __shared__ double2 zs[];  // [mpb][fft_stride(H)], point j of mic ml at zs[ml * stride + zp(j)]
    const int H = N >> 1, stride = fft_stride(H);
    const int logH = 31 - __clz(H), logP = 31 - __clz(mpb);
    const int64_t w = w0 + blockIdx.y;
    const int m0 = blockIdx.x * mpb;
    const int nm = min(mpb, M - m0);
    const TS *src = samples + (w * (int64_t)hop) * M + m0;
    constexpr bool PLAIN = OUT == OUT_C64;   // see butterfly
    const double2 w41 = __ldg(tw + (N >> 2)), w81 = __ldg(tw + (N >> 3)), w83 = __ldg(tw + 3 * (N >> 3));

    // load + window + the first three stages: task = 8 consecutive slots of the bit-reversed order, i.e. points
    // rev(task) + H/8 {0, 4, 2, 6, 1, 5, 3, 7} (H >= 8)
    const int logT = logH - 3;
    // Lanes run along the mics, then (fewer than 8 mics) along the task, so that eight lanes store to eight banks, then
    // along the rows: the window's values of a warp lie next to one another.
    const int tl = min(max(3 - logP, 0), logT);
    for (int idx = threadIdx.x; idx < mpb << logT; idx += blockDim.x) {
        const int ml = idx & (mpb - 1), a = idx >> logP, jl = a >> tl, low = a & ((1 << tl) - 1);
        if (ml >= nm) continue;
        const int task = low | (bit_reverse(jl, logT - tl) << tl);
        const int j0 = jl | (bit_reverse(low, tl) << (logT - tl));
        double2 v[8];
        TS x0[8], x1[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const int j = j0 + ((((t & 1) << 2) | (t & 2) | (t >> 2)) << logT);
            x0[t] = __ldg(src + (int64_t)(2 * j) * M + ml);
            x1[t] = __ldg(src + (int64_t)(2 * j + 1) * M + ml);
        }
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const int j = j0 + ((((t & 1) << 2) | (t & 2) | (t >> 2)) << logT);
            const double a0 = __ldg(window + 2 * j), a1 = __ldg(window + 2 * j + 1);
            v[t] = PLAIN ? make_double2(__dmul_rn((double)x0[t], a0), __dmul_rn((double)x1[t], a1))
                         : make_double2((double)x0[t] * a0, (double)x1[t] * a1);
        }
        if (PLAIN) first_stages_plain(v, w41, w81, w83);
        else first_stages(v);
        double2 *z = zs + ml * stride + 9 * task;   // zp(8 task + t) = 9 task + t
#pragma unroll
        for (int t = 0; t < 8; ++t) z[t] = v[t];
    }
    __syncthreads();
    fft_passes<PLAIN>(zs, nm, stride, 3, logH, logH + 1, tw);

    // real-input split: X[k] = E + W^k O,  E = (Z[k] + conj(Z[H-k]))/2,  O = -i (Z[k] - conj(Z[H-k]))/2
    // (bins k and H - k share their two points: read once for both)
    const SplitPairs sp(bin_lo, nbins, H);
    for (int idx = threadIdx.x; idx < sp.n << logP; idx += blockDim.x) {
        const int ml = idx & (mpb - 1);
        if (ml >= nm) continue;
        const int u = sp.u0 + (idx >> logP);
        const double2 *z = zs + ml * stride;
        const double2 za = z[zp(u)], zb = z[zp((H - u) & (H - 1))];
        auto bin = [&](int k, double2 zk, double2 zc) {
            if (k < bin_lo || k >= bin_lo + nbins) return;
            const double er = 0.5 * (zk.x + zc.x), ei = 0.5 * (zk.y - zc.y);
            const double orr = 0.5 * (zk.y + zc.y), oi = -0.5 * (zk.x - zc.x);
            const double2 wk = k < H ? __ldg(tw + k) : make_double2(-1.0, 0.0);
            const double xr = PLAIN ? er + (wk.x * orr - wk.y * oi) : fma(wk.x, orr, fma(-wk.y, oi, er));
            const double xi = PLAIN ? ei + (wk.x * oi + wk.y * orr) : fma(wk.x, oi, fma(wk.y, orr, ei));
            put_bin<OUT>(out, nw, (int)blockIdx.y, M, m0 + ml, k - bin_lo, xr, xi, R, KC, lo_elems);
        };
        bin(u, za, zb);
        if (2 * u != H) bin(H - u, zb, za);
    }
}

// ------------------------------------------------------------------------------------------------
// Tensor-core operand tiles straight from the samples, four windows per CTA (fft4_tc_kernel).
// The tile layout is K-major: a 16-byte core-matrix row holds 4 consecutive windows (TF32) or 8
// (BF16) of one spectrum component, so a CTA that transforms 4 consecutive windows of `mpb` mics
// stores whole 16-byte rows (TF32) or half rows (BF16) instead of one 4-byte value per window.
// Bound: shared-memory wavefronts (81 % of their rate): three passes' worth of 8-byte accesses and the split's.  The
// first three stages run on the points as they are loaded, and a thread keeps its task's twiddles over the sequences.
// Measured (B200): 999 windows x 256 mics x 1024 samples to TF32 tiles 1.06 -> 0.92 ms; CSM of 64 mics x 300,000
// samples, block 4096: 0.56 -> 0.36 ms (wide CTAs).
// The transform runs in FP32 (the operands are rounded to TF32 or split into BF16 hi + lo right
// after it, so FP64 arithmetic buys nothing): complex points are 8 bytes, half the shared-memory
// traffic of the FP64 transform.  Padded windows (>= the chunk's count, up to 32 KC) and padded
// mics (up to 16 R) are written as zeros, so the operand buffer needs no clearing beforehand.
// ------------------------------------------------------------------------------------------------
// Shared-memory slot of point j: one padding slot per 16 points (8-byte points), so that the passes'
// strided accesses spread over the banks.
__device__ __forceinline__ int zpf(int j) { return j + (j >> 4); }
// Padded length of one sequence: at least H + H/16 slots and congruent to 32 / mpb modulo 16.  In the real
// split a warp reads Z[k] of mpb mics x 32 / mpb consecutive bins; with that stride the mics' slots fall
// on different bank pairs (with the stride 1 modulo 16 of a first version, 4 mics x 8 bins put up to 4
// threads on one bank pair).
__host__ __device__ constexpr int fft_stride_f(int H, int mpb)
{
    return H + (H >> 4) + ((((32 / mpb) & 15) - (H + (H >> 4))) & 15);
}

// s (1..3) consecutive radix-2 DIT stages, the first of length 2 half1, on the 2^s points of a task (see fft_pass).
// The twiddles come from a shared-memory table in stage order: the stage of length L = 2 hf reads W_L^i (i < hf) at
// tws[hf + i], so consecutive threads read consecutive entries (the natural-order table read with the stride N / L put
// up to 16 threads on one bank).  The entries are the FP32 roundings of the same W_N^e as the natural-order table.
// A task's twiddle at stage q is entry (task mod half1) + (t mod 2^q) half1 of the stage's table: 2^q distinct values.
template <int S>
struct PassTwiddlesF {
    float2 w[(1 << S) - 1];   // stage q at 2^q - 1 + u
    __device__ __forceinline__ void load(int sg, int task, const float2 *__restrict__ tws)
    {
        const int half1 = 1 << sg, tb = task & (half1 - 1);
#pragma unroll
        for (int q = 0; q < S; ++q)
#pragma unroll
            for (int u = 0; u < (1 << q); ++u) w[(1 << q) - 1 + u] = tws[(half1 << q) + tb + u * half1];
    }
};

template <int S>
__device__ __forceinline__ void stages_f(float2 (&v)[1 << S], const PassTwiddlesF<S> &tw)
{
#pragma unroll
    for (int q = 0; q < S; ++q)
#pragma unroll
        for (int t = 0; t < (1 << S); ++t) {
            if (t & (1 << q)) continue;
            const float2 w = tw.w[(1 << q) - 1 + (t & ((1 << q) - 1))];
            const float2 b = v[t + (1 << q)];
            const float br = b.x * w.x - b.y * w.y;
            const float bi = b.x * w.y + b.y * w.x;
            const float2 a = v[t];
            v[t] = make_float2(a.x + br, a.y + bi);
            v[t + (1 << q)] = make_float2(a.x - br, a.y - bi);
        }
}

// One pass over `nseq` sequences: a thread keeps one task and its twiddles and walks the sequences.
template <int S>
__device__ __forceinline__ void fft_pass_f(float2 *__restrict__ zs, int nseq, int st, int sg, int logH,
                                           const float2 *__restrict__ tws)
{
    const int logT = logH - S, T = 1 << logT, nt = blockDim.x, half1 = 1 << sg;
    const int grp = T < nt ? threadIdx.x >> logT : 0, ngrp = T < nt ? nt >> logT : 1;
    for (int task = T < nt ? threadIdx.x & (T - 1) : threadIdx.x; task < T; task += nt) {
        const int base = ((task >> sg) << (sg + S)) + (task & (half1 - 1));
        PassTwiddlesF<S> w;
        w.load(sg, task, tws);
        for (int q = grp; q < nseq; q += ngrp) {
            float2 *z = zs + q * st;
            float2 v[1 << S];
#pragma unroll
            for (int t = 0; t < (1 << S); ++t) v[t] = z[zpf(base + t * half1)];
            stages_f<S>(v, w);
#pragma unroll
            for (int t = 0; t < (1 << S); ++t) z[zpf(base + t * half1)] = v[t];
        }
    }
    __syncthreads();
}

constexpr int FFT4_WIN = 4;   // windows per CTA

// V consecutive samples of one row, as float (V = 1, 2 or 4; the address is aligned to the vector)
template <int V>
__device__ __forceinline__ void ld_row(const float *__restrict__ p, float (&x)[V])
{
    if (V == 4) {
        const float4 u = __ldg(reinterpret_cast<const float4 *>(p));
        x[0] = u.x;
        x[1] = u.y;
        x[2] = u.z;
        x[3] = u.w;
    } else if (V == 2) {
        const float2 u = __ldg(reinterpret_cast<const float2 *>(p));
        x[0] = u.x;
        x[1] = u.y;
    } else {
        x[0] = __ldg(p);
    }
}
template <int V>
__device__ __forceinline__ void ld_row(const double *__restrict__ p, float (&x)[V])
{
    if (V == 1) {
        x[0] = (float)__ldg(p);
    } else {
#pragma unroll
        for (int e = 0; e < V; e += 2) {
            const double2 u = __ldg(reinterpret_cast<const double2 *>(p + e));
            x[e] = (float)u.x;
            x[e + 1] = (float)u.y;
        }
    }
}

// Load, window and the first three stages of the CTA's 4 windows x mpb mics: one thread per (window, group of V mics,
// task), the task fastest.  A task is 8 consecutive slots of the bit-reversed order, i.e. points rev(task) + H/8
// {0, 4, 2, 6, 1, 5, 3, 7}; the thread loads rows 2j and 2j + 1 of each as one vector of V mics.  Windows past the
// chunk and padding mics are zeros (M % V == 0: a group is all in or all out).
template <typename TS, int V>
__device__ __forceinline__ void fft4_load(const TS *__restrict__ samples, int M, int hop, int64_t w0, int64_t nw,
                                          int wg, int m0, int mpb, int H, int logH, int st,
                                          const float *__restrict__ wf, const float2 *__restrict__ tws,
                                          float2 *__restrict__ zs)
{
    constexpr int logV = V == 4 ? 2 : (V == 2 ? 1 : 0);
    int logG = 0;
    while ((V << logG) < mpb) ++logG;                          // mpb / V groups
    const int logT = logH - 3;
    PassTwiddlesF<3> w3;
    w3.load(0, 0, tws);
    for (int idx = threadIdx.x; idx < (FFT4_WIN << logG) << logT; idx += blockDim.x) {
        const int task = idx & ((1 << logT) - 1);
        const int mg = (idx >> logT) & ((1 << logG) - 1);
        const int wi = idx >> (logT + logG);
        const int64_t w = (int64_t)wg * FFT4_WIN + wi;
        const int m = m0 + (mg << logV);
        const int j0 = logT ? (int)(__brev((unsigned)task) >> (32 - logT)) : 0;
        float x0[8][V], x1[8][V];
        const bool in = w < nw && m < M;
        const TS *src = samples + ((w0 + w) * (int64_t)hop) * M + m;
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const int j = j0 + ((((t & 1) << 2) | (t & 2) | (t >> 2)) << logT);
            if (in) {
                ld_row<V>(src + (int64_t)(2 * j) * M, x0[t]);
                ld_row<V>(src + (int64_t)(2 * j + 1) * M, x1[t]);
            } else {
#pragma unroll
                for (int e = 0; e < V; ++e) x0[t][e] = x1[t][e] = 0.f;
            }
        }
        float2 a[8];
#pragma unroll
        for (int t = 0; t < 8; ++t)
            a[t] = *reinterpret_cast<const float2 *>(wf + 2 * (j0 + ((((t & 1) << 2) | (t & 2) | (t >> 2)) << logT)));
        float2 *z = zs + (wi * mpb + (mg << logV)) * st;
#pragma unroll
        for (int e = 0; e < V; ++e) {
            float2 v[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) v[t] = make_float2(__fmul_rn(x0[t][e], a[t].x), __fmul_rn(x1[t][e], a[t].y));
            stages_f<3>(v, w3);
#pragma unroll
            for (int t = 0; t < 8; ++t) z[e * st + zpf(8 * task + t)] = v[t];
        }
    }
    __syncthreads();
}

template <typename TS, int OUT>
__global__ void __launch_bounds__(512) fft4_tc_kernel(const TS *__restrict__ samples, int M, int N, int hop, int64_t w0,
                                                      int64_t nw, int mpb, int vw, const double *__restrict__ window,
                                                      const double2 *__restrict__ tw, int bin_lo, int nbins,
                                                      void *__restrict__ out, int R, int KC, int64_t lo_elems)
{
    extern __shared__ __align__(16) uint8_t fsm[];
    const int H = N >> 1;
    const int st = fft_stride_f(H, mpb);
    float2 *zs = reinterpret_cast<float2 *>(fsm);                 // [FFT4_WIN][mpb][st]
    float2 *tws = zs + FFT4_WIN * mpb * st;                       // [H] twiddles in stage order (fft_pass_f)
    float *wf = reinterpret_cast<float *>(tws + H);               // [N]
    int logH = 0, logP = 0;
    while ((1 << logH) < H) ++logH;
    while ((1 << logP) < mpb) ++logP;                              // mpb is a power of two
    const int wg = blockIdx.y;                                     // windows 4 wg .. 4 wg + 3 of the chunk
    const int m0 = blockIdx.x * mpb;
    for (int i = threadIdx.x + 1; i < H; i += blockDim.x) {
        // i = hf + r, hf the largest power of two <= i: W_{2 hf}^r = W_N^(r H / hf), N = 2 H
        const int lhf = 31 - __clz(i);
        const double2 u = tw[(i - (1 << lhf)) << (logH - lhf)];
        tws[i] = make_float2((float)u.x, (float)u.y);
    }
    for (int i = threadIdx.x; i < N; i += blockDim.x) wf[i] = (float)window[i];
    __syncthreads();

    if (vw == 4) fft4_load<TS, 4>(samples, M, hop, w0, nw, wg, m0, mpb, H, logH, st, wf, tws, zs);
    else if (vw == 2) fft4_load<TS, 2>(samples, M, hop, w0, nw, wg, m0, mpb, H, logH, st, wf, tws, zs);
    else fft4_load<TS, 1>(samples, M, hop, w0, nw, wg, m0, mpb, H, logH, st, wf, tws, zs);

    // the other stages, up to three per pass, over all 4 mpb sequences
    for (int sg = 3; sg < logH;) {
        const int S = logH - sg >= 3 ? 3 : logH - sg;
        if (S == 3) fft_pass_f<3>(zs, FFT4_WIN * mpb, st, sg, logH, tws);
        else if (S == 2) fft_pass_f<2>(zs, FFT4_WIN * mpb, st, sg, logH, tws);
        else fft_pass_f<1>(zs, FFT4_WIN * mpb, st, sg, logH, tws);
        sg += S;
    }

    // real split of each bin for the 4 windows, then one store per tile row (Re row 2m, Im row 2m+1)
    const int col0 = (wg * FFT4_WIN) & 31;
    const int64_t kc = (wg * FFT4_WIN) >> 5;
    for (int idx = threadIdx.x; idx < nbins * mpb; idx += blockDim.x) {
        const int ml = idx & (mpb - 1);
        const int b = idx >> logP;
        const int k = bin_lo + b;
        const int kh = k & (H - 1), kc2 = (H - kh) & (H - 1);
        float2 wk = make_float2(-1.f, 0.f);
        if (k < H) {
            const double2 t = __ldg(tw + k);
            wk = make_float2((float)t.x, (float)t.y);
        }
        float xr[FFT4_WIN], xi[FFT4_WIN];
#pragma unroll
        for (int wi = 0; wi < FFT4_WIN; ++wi) {
            const float2 *z = zs + (wi * mpb + ml) * st;
            const float2 zk = z[zpf(kh)], zc = z[zpf(kc2)];
            const float er = 0.5f * (zk.x + zc.x), ei = 0.5f * (zk.y - zc.y);
            const float orr = 0.5f * (zk.y + zc.y), oi = -0.5f * (zk.x - zc.x);
            xr[wi] = er + (wk.x * orr - wk.y * oi);
            xi[wi] = ei + (wk.x * oi + wk.y * orr);
        }
        const int m = m0 + ml;                                    // padded mics carry zeros
        const int rowc = 2 * m;
        const int64_t tile = ((int64_t)b * KC + kc) * R + (rowc >> 5);
        const int r0 = rowc & 31;
        if (OUT == OUT_TF32) {
            uint32_t *t = reinterpret_cast<uint32_t *>(out) + tile * 1024;
            *reinterpret_cast<uint4 *>(t + tile_off_tf32(r0, col0)) =
                make_uint4(tf32_bits(xr[0]), tf32_bits(xr[1]), tf32_bits(xr[2]), tf32_bits(xr[3]));
            *reinterpret_cast<uint4 *>(t + tile_off_tf32(r0 + 1, col0)) =
                make_uint4(tf32_bits(xi[0]), tf32_bits(xi[1]), tf32_bits(xi[2]), tf32_bits(xi[3]));
        } else {
            __nv_bfloat16 *t = reinterpret_cast<__nv_bfloat16 *>(out) + tile * 1024;
#pragma unroll
            for (int part = 0; part < 2; ++part) {   // Re row, Im row
                const float *x = part ? xi : xr;
                uint32_t hv[2], lv[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const __nv_bfloat162 hi = __floats2bfloat162_rn(x[2 * h], x[2 * h + 1]);
                    const float2 hf = __bfloat1622float2(hi);
                    const __nv_bfloat162 lo = __floats2bfloat162_rn(x[2 * h] - hf.x, x[2 * h + 1] - hf.y);
                    hv[h] = *reinterpret_cast<const uint32_t *>(&hi);
                    lv[h] = *reinterpret_cast<const uint32_t *>(&lo);
                }
                const int o = tile_off(r0 + part, col0);
                *reinterpret_cast<uint2 *>(t + o) = make_uint2(hv[0], hv[1]);
                *reinterpret_cast<uint2 *>(t + lo_elems + o) = make_uint2(lv[0], lv[1]);
            }
        }
    }
}

// Mics per CTA of fft4_tc_kernel (a power of two <= 16, so that the 16 R padded mics split evenly) and its threads: up
// to 72 KB of FP32 sequences and 256 threads; for blocks of 2048 samples and more, of which that would hold one or two
// mics and load 4 or 8 bytes of a row at a time, up to 148 KB and 512 threads.  0 mics if even one mic's 4 windows do
// not fit.
static int fft4_threads(int N) { return N >= FFT_WIDE_N ? 512 : 256; }
static int fft4_mics_per_block(int N)
{
    const size_t tables = (size_t)(N / 2) * sizeof(float2) + (size_t)N * sizeof(float);
    if ((size_t)FFT4_WIN * fft_stride_f(N / 2, 1) * sizeof(float2) + tables >= 200 * 1024) return 0;
    const size_t most = (N >= FFT_WIDE_N ? 148 : 72) * 1024;
    int mpb = 16;
    while (mpb > 1 && (size_t)mpb * FFT4_WIN * fft_stride_f(N / 2, mpb) * sizeof(float2) > most) mpb >>= 1;
    return mpb;
}

bool fft_tiles_written_whole(int block_size) { return fft4_mics_per_block(block_size) > 0; }

static size_t fft4_smem_bytes(int N, int mpb)
{
    return (size_t)FFT4_WIN * mpb * fft_stride_f(N / 2, mpb) * sizeof(float2) + (size_t)(N / 2) * sizeof(float2) +
           (size_t)N * sizeof(float);
}

// ------------------------------------------------------------------------------------------------
// Large blocks (N > 16384): one mic's N/2-point sequence no longer fits a CTA's shared memory.  It is
// split by decimation in time into D = N / 16384 interleaved sub-sequences z[d + D i] of 8192 points:
// fft_sub_kernel transforms each one in shared memory with the passes above (sub-spectra Y_d to a
// scratch region [window][mic][d][8192]), and fft_combine_kernel forms, for the requested bins only,
// Z[k] = sum_d W_H^{d k} Y_d[k mod 8192] and Z[H - k] before the same real split.
// ------------------------------------------------------------------------------------------------
constexpr int FFT_MAX_N = 16384;                 // largest block transformed by one CTA
constexpr int FFT_SUB_H = FFT_MAX_N / 2;         // points of each sub-sequence of a larger block

size_t fft_scratch_bytes(int num_mics, int block_size, int64_t num_windows)
{
    if (block_size <= FFT_MAX_N) return 0;
    return (size_t)num_windows * (size_t)num_mics * (size_t)(block_size / 2) * sizeof(double2);
}

template <typename TS>
__global__ void __launch_bounds__(256) fft_sub_kernel(const TS *__restrict__ samples, int M, int N, int hop,
                                                      int64_t w0, const double *__restrict__ window,
                                                      const double2 *__restrict__ tw, double2 *__restrict__ scratch)
{
    extern __shared__ double2 zs[];   // [zp(j)], j < FFT_SUB_H
    const int D = (N >> 1) / FFT_SUB_H;
    int logHs = 0;
    while ((1 << logHs) < FFT_SUB_H) ++logHs;
    const int64_t wi = blockIdx.y;
    const int m = blockIdx.x, d = blockIdx.z;
    const TS *src = samples + ((w0 + wi) * (int64_t)hop) * M + m;
    for (int i = threadIdx.x; i < FFT_SUB_H; i += blockDim.x) {
        const int64_t j = d + (int64_t)D * i;    // complex point j = (x[2j], x[2j+1])
        const double x0 = (double)src[(2 * j) * M] * window[2 * j];
        const double x1 = (double)src[(2 * j + 1) * M] * window[2 * j + 1];
        zs[zp((int)(__brev((unsigned)i) >> (32 - logHs)))] = make_double2(x0, x1);
    }
    __syncthreads();
    fft_passes<true>(zs, 1, 0, 0, logHs, 31 - __clz(N), tw);
    double2 *dst = scratch + ((wi * M + m) * D + d) * (int64_t)FFT_SUB_H;
    for (int k = threadIdx.x; k < FFT_SUB_H; k += blockDim.x) dst[k] = zs[zp(k)];
}

// W_N^e for any integer exponent e (the table holds e < N/2; W_N^{e + N/2} = -W_N^e)
__device__ __forceinline__ double2 twiddle_any(const double2 *__restrict__ tw, int N, int64_t e)
{
    e %= N;
    const int h = N >> 1;
    if (e < h) return tw[e];
    const double2 t = tw[e - h];
    return make_double2(-t.x, -t.y);
}

// Z[k] of one (window, mic) from its D sub-spectra
__device__ __forceinline__ double2 combine_point(const double2 *__restrict__ y, int N, int D, int k,
                                                 const double2 *__restrict__ tw)
{
    const int kk = k % FFT_SUB_H;
    double zr = 0.0, zi = 0.0;
    for (int d = 0; d < D; ++d) {
        const double2 v = y[(int64_t)d * FFT_SUB_H + kk];
        const double2 w = twiddle_any(tw, N, 2 * (int64_t)d * k);   // W_H^{d k} = W_N^{2 d k}
        zr += v.x * w.x - v.y * w.y;
        zi += v.x * w.y + v.y * w.x;
    }
    return make_double2(zr, zi);
}

template <int OUT>
__global__ void __launch_bounds__(256) fft_combine_kernel(const double2 *__restrict__ scratch, int M, int N,
                                                          int64_t nw, int bin_lo, int nbins,
                                                          const double2 *__restrict__ tw, void *__restrict__ out,
                                                          int R, int KC, int64_t lo_elems)
{
    const int H = N >> 1, D = H / FFT_SUB_H;
    const int wi = blockIdx.y;
    const int k = bin_lo + blockIdx.x;
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        const double2 *y = scratch + ((int64_t)wi * M + m) * D * FFT_SUB_H;
        const double2 zk = combine_point(y, N, D, k % H, tw);
        const double2 zc = combine_point(y, N, D, (H - k % H) % H, tw);
        const double er = 0.5 * (zk.x + zc.x), ei = 0.5 * (zk.y - zc.y);
        const double orr = 0.5 * (zk.y + zc.y), oi = -0.5 * (zk.x - zc.x);
        const double2 wk = k < H ? tw[k] : make_double2(-1.0, 0.0);
        const double xr = er + (wk.x * orr - wk.y * oi);
        const double xi = ei + (wk.x * oi + wk.y * orr);
        put_bin<OUT>(out, nw, wi, M, m, k - bin_lo, xr, xi, R, KC, lo_elems);
    }
}

// ------------------------------------------------------------------------------------------------
// Welch Gram accumulation in complex64, upper-triangular T x T tiles (64, or 32: gram_c64_narrow); thread (tx, ty) of 16
// x 8 owns rows ty + 8 i and columns tx + 16 j of the tile.  An element's (re, im) is one packed pair of FP32 accumulators, so that the
// reference's two chained FMAs per component are two packed FMAs, (x_c, -y_c) x_r and then (y_c, x_c) y_r.  In a
// diagonal tile the 8 x 16 blocks below the diagonal are left out.
// Bound: FP32 FMAs (0.31 ms here) and the issue slots of the operand pairs' moves.  8 x 4 elements per thread, as 4 x 4
// made it shared-memory bound (89 % of its wavefronts).  Measured (B200): 2049 bins x 113 mics x 147 windows
// 821 -> 500 us.
// With `out` the sums are not added to csm but written, scaled, as the full Hermitian complex128 matrix.
// ------------------------------------------------------------------------------------------------
constexpr int GT = 64;   // the larger tile's edge
constexpr int GKC = 16;  // windows per shared-memory stage
constexpr int GTHREADS = 128;

__device__ __forceinline__ void ffma2(float2 &acc, float ax, float ay, float b)
{
    asm("{\n\t.reg .b64 ra, rb, rc;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\tmov.b64 rc, {%0, %1};\n\t"
        "fma.rn.f32x2 rc, ra, rb, rc;\n\tmov.b64 {%0, %1}, rc;\n\t}"
        : "+f"(acc.x), "+f"(acc.y)
        : "f"(ax), "f"(ay), "f"(b));
}

// One stage of `kc` windows into the accumulators.
template <bool DIAG, int T, int RI, int CJ>
__device__ __forceinline__ void gram64_stage(const float2 *xr, const float2 *xc, int kc, float2 (&acc)[RI][CJ])
{
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 4
    for (int kk = 0; kk < kc; ++kk) {
        float2 r[RI], c[CJ];
#pragma unroll
        for (int i = 0; i < RI; ++i) r[i] = xr[kk * T + ty + 8 * i];
#pragma unroll
        for (int j = 0; j < CJ; ++j) c[j] = xc[kk * T + tx + 16 * j];
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < CJ; ++j) {
                if (DIAG && i > 2 * j + 1) continue;
                ffma2(acc[i][j], c[j].x, -c[j].y, r[i].x);
                ffma2(acc[i][j], c[j].y, c[j].x, r[i].y);
            }
    }
}

template <int T>
__global__ void __launch_bounds__(GTHREADS, 4) gram_c64_kernel(const float2 *__restrict__ spec, int M, int64_t nw,
                                                               float2 *__restrict__ csm, double2 *__restrict__ out,
                                                               double scale)
{
    constexpr int RI = T / 8, CJ = T / 16;
    __shared__ float2 g64_sm[2][2][GKC][T];   // [stage][rows | columns]
    // upper-triangular tile index -> (ti, tj), ti <= tj
    const int NT = (M + T - 1) / T;
    int t = blockIdx.x, ti = 0;
    while (t >= NT - ti) {
        t -= NT - ti;
        ++ti;
    }
    const int tj = ti + t;
    const int f = blockIdx.y;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int r0 = ti * T, c0 = tj * T;
    const bool diag = ti == tj;

    float2 acc[RI][CJ];
    float2 *base = csm + (int64_t)f * M * M;
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < CJ; ++j) {
            const int r = r0 + ty + 8 * i, c = c0 + tx + 16 * j;
            acc[i][j] = make_float2(0.f, 0.f);
            if (!out && r < M && c < M && r <= c) acc[i][j] = base[(int64_t)r * M + c];
        }

    const float2 *sp = spec + (int64_t)f * nw * M;
    const int lm = threadIdx.x & (T - 1), lk = threadIdx.x / T;   // this thread's mic and first window of a stage
    auto load = [&](int64_t k0, int buf) {
#pragma unroll
        for (int u = 0; u < GKC; u += GTHREADS / T) {
            const int64_t k = k0 + lk + u;
            const bool in = k < nw;
            const float2 *src = sp + (in ? k : 0) * M;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&g64_sm[buf][0][lk + u][lm]);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src + min(r0 + lm, M - 1)),
                         "r"(in && r0 + lm < M ? 8 : 0)
                         : "memory");
            if (!diag)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + GKC * T * 8),
                             "l"(src + min(c0 + lm, M - 1)), "r"(in && c0 + lm < M ? 8 : 0)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load(0, 0);
    int buf = 0;
    for (int64_t k0 = 0; k0 < nw; k0 += GKC, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // this stage has landed for every thread, and the other buffer is read by none any more
        if (k0 + GKC < nw) load(k0 + GKC, buf ^ 1);
        const int kc = (int)((nw - k0) < GKC ? (nw - k0) : GKC);
        const float2 *xr = &g64_sm[buf][0][0][0];
        if (diag) gram64_stage<true, T>(xr, xr, kc, acc);
        else gram64_stage<false, T>(xr, xr + GKC * T, kc, acc);
    }
    double2 *ob = out + (int64_t)f * M * M;
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < CJ; ++j) {
            const int r = r0 + ty + 8 * i, c = c0 + tx + 16 * j;
            if (r >= M || c >= M || r > c) continue;
            if (out) put_hermitian(ob, M, r, c, (double)acc[i][j].x, (double)acc[i][j].y, scale);
            else base[(int64_t)r * M + c] = acc[i][j];
        }
}

// 32 x 32 tiles for arrays of up to 32 mics, and where the 64 x 64 tiles' last round over the SMs would be so empty that
// at least 3 of 10 places stay free (up to three rounds).  Measured (B200), microseconds of the whole CSM, 64 / 32: 33
// tiles 164 / 104, 65 99 / 88, 195 219 / 173, 330 303 / 261; 129 129 / 141, 257 231 / 251, 650 470 / 476; 32 mics, 513
// bins 175 / 112; 8 mics, 65 bins 77 / 42.
static bool gram_c64_narrow(int M, int64_t tiles)
{
    const int64_t rounds = (tiles + kNumSMs - 1) / kNumSMs;
    return M <= 32 || (rounds <= 3 && 10 * rounds * kNumSMs >= 13 * tiles);
}

static int gram_c64_launch(const void *spec, int M, int64_t nw, int nbins, void *csm, void *out, double scale,
                           cudaStream_t s)
{
    const int T = (M + GT - 1) / GT;
    const bool narrow = gram_c64_narrow(M, (int64_t)T * (T + 1) / 2 * nbins);
    const auto kernel = narrow ? gram_c64_kernel<32> : gram_c64_kernel<GT>;
    const int NT = narrow ? (M + 31) / 32 : T;
    kernel<<<dim3(NT * (NT + 1) / 2, nbins), GTHREADS, 0, s>>>(reinterpret_cast<const float2 *>(spec), M, nw,
                                                               reinterpret_cast<float2 *>(csm),
                                                               reinterpret_cast<double2 *>(out), scale);
    return check_launch();
}

// ------------------------------------------------------------------------------------------------
// The complex128 Gram on the FP64 matrix instruction (mma.sync m16n8k8; tcgen05 has no FP64 kind).  With the windows'
// (re, im) pairs as the K dimension,
//     Re C[r][c] = sum_k A[r][k] B[k][c],  A[r] = (x_r, y_r, ..),  B[.][c] = (x_c, y_c, ..),
//     Im C[r][c] = sum_k A[r][k] B'[k][c],                         B'[.][c] = (-y_c, x_c, ..),
// and the instruction adds its products to an element as a chain of FMAs in ascending k (checked on 10^5 random
// elements), so this is the reference's order of two chained FMAs per window and component, bit for bit.
// CTA = 32 x 32 (small launches: 32 x 16, GF_NARROW) tile of one bin's upper triangle, 4 warps of 16 x 16 (16 x 8); 16
// windows per stage, three stages of cp.async,
// four CTAs per SM.  Rows are padded to 36 mics, so that the operand reads of 4 mics x 2 windows (A) and 8 mics x 2
// windows (B) fall on different banks.  16 x 8 blocks entirely below the diagonal or past M are skipped.  With `out`
// the sums are not added to csm but written, scaled, as the full Hermitian matrix.
// A lane's two elements of a block are two columns apart (gf_column), so that four lanes read and write whole sectors of a
// row.  Measured (B200), 513 bins added to: 256 mics, 4
// windows 164 -> 150 us, 33 windows 318 -> 270; 113 mics, 1 window 49 -> 41, 33 windows 108 -> 95 (lanes with columns 2 t and
// 2 t + 1, and 16 windows' products whatever the stage holds; the FMA form before it 133, 455, 39 and 164).  999 windows of
// 256 mics 6255 -> 6189 with the transform.
// Bound: the FP64 pipe (4 M^2 K flop per bin).  Measured (B200): 513 bins x 256 mics x 999 windows 7.84 -> 5.0 ms
// (27 TFLOP/s; 64 x 64 tiles of 32 x 16 per warp 5.2 ms, half of the diagonal tiles idle); 65 bins x 64 mics x 799
// windows 281 -> 75 us (195 CTAs where the 64 x 64 tiles of the FMA form were 65), in 32 x 16 tiles 65 us.
// ------------------------------------------------------------------------------------------------
constexpr int GF_T = 32;       // tile edge
constexpr int GF_LD = GF_T + 4;
constexpr int GF_KW = 16;      // windows per stage
constexpr int GF_STAGES = 3;
// Fewer 32 x 32 tiles than this (all bins): 32 x 16 tiles, twice as many CTAs, so that no SM holds two tiles while its
// neighbour holds one.  Measured (B200), microseconds of the whole CSM, 32 x 32 / 32 x 16: 65 tiles 61 / 45, 99 151 / 145,
// 170 227 / 209, 195 110 / 101 and 96 / 73, 198 207 / 182; 255 249 / 262, 257 139 / 145, 330 319 / 352, 387 175 / 205.
constexpr int64_t GF_NARROW = kNumSMs * 3 / 2;
constexpr int GF_SMEM = GF_STAGES * 2 * GF_KW * GF_LD * (int)sizeof(double2);

// The column of an 8-column block that the instruction's column n stands for: 0 2 1 3 4 6 5 7.  Lane t's columns 2 t and
// 2 t + 1 of the instruction are then 0, 1, 4, 5 and 2, 3, 6, 7 of the block over the four lanes (pairs fill sectors), and
// neighbouring n two apart, so that their operand reads fall on different banks.
__device__ __forceinline__ int gf_column(int n) { return ((n >> 1) & 1) + 4 * (n >> 2) + 2 * (n & 1); }

template <int NB>
__global__ void __launch_bounds__(128, 4) gram_f64_kernel(const double2 *__restrict__ spec, int M, int64_t nw,
                                                          double2 *__restrict__ csm, double2 *__restrict__ out,
                                                          double scale)
{
    constexpr int T = GF_T, TC = 16 * NB, LD = GF_LD;   // T rows x TC columns
    extern __shared__ double2 gf_sm[];   // [stage][row mics | column mics][window][LD]
    // tile index -> row tile ti and column tile tj >= ti T / TC
    const int NT = (M + TC - 1) / TC;
    int tile = blockIdx.x, ti = 0;
    while (tile >= NT - ti * (T / TC)) {
        tile -= NT - ti * (T / TC);
        ++ti;
    }
    const int tj = ti * (T / TC) + tile;
    const int f = blockIdx.y;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    // warp -> 16 x 8 NB quarter, rotated over the CTAs: in a diagonal tile the lower-left quarter has nothing to do
    const int quarter = ((threadIdx.x >> 5) + blockIdx.x + blockIdx.y) & 3;
    const int wr = quarter >> 1, wc = quarter & 1;
    const int r0 = ti * T, c0 = tj * TC;
    const int rw = r0 + wr * 16, cw = c0 + wc * 8 * NB;   // this warp's first row and column
    const bool same = c0 < r0 + T;                        // the columns are among the rows
    const double2 *sp = spec + (int64_t)f * nw * M;
    double2 *base = csm + (int64_t)f * M * M;

    auto load = [&](int64_t st) {
        double2 *d = gf_sm + (st % GF_STAGES) * (2 * GF_KW * LD);
        const int64_t k0 = st * GF_KW;
#pragma unroll
        for (int i = 0; i < GF_KW / 4; ++i) {
            const int kk = i * 4 + (int)threadIdx.x / T, m = threadIdx.x % T;
            const bool in = k0 + kk < nw;
            const double2 *src = sp + (in ? k0 + kk : 0) * M;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(d + kk * LD + m);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src + min(r0 + m, M - 1)),
                         "r"(in && r0 + m < M ? 16 : 0)
                         : "memory");
            if (!same && m < TC)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + GF_KW * LD * 16),
                             "l"(src + min(c0 + m, M - 1)), "r"(in && c0 + m < M ? 16 : 0)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    double re[NB][4], im[NB][4];
    bool use[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        const int cb = cw + 8 * j;
        use[j] = rw <= cb + 7 && rw < M && cb < M;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = rw + g + 8 * (e >> 1), c = cb + gf_column(2 * t + (e & 1));
            double2 v = make_double2(0.0, 0.0);
            if (!out && c < M && r <= c) v = base[(int64_t)r * M + c];
            re[j][e] = v.x;
            im[j][e] = v.y;
        }
    }

    const int64_t nst = (nw + GF_KW - 1) / GF_KW;
    const double *ar = nullptr;
    const double2 *bc = nullptr;
    auto arrive = [&](int64_t st, bool more) {
        if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // stage st has landed for every thread; stage st - 1 is read by none any more
        if (st + 2 < nst) load(st + 2);
        const double2 *xr = gf_sm + (st % GF_STAGES) * (2 * GF_KW * LD);
        const double2 *xc = same ? xr + (c0 - r0) : xr + GF_KW * LD;
        ar = reinterpret_cast<const double *>(xr + (t >> 1) * LD + wr * 16 + g) + (t & 1);
        bc = xc + (t >> 1) * LD + wc * 8 * NB + gf_column(g);
    };
    auto four = [&](int w) {   // windows w .. w + 3 of the stage
        double b0[NB], b1[NB], q0[NB], q1[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const double2 u = bc[w * LD + 8 * j], v = bc[(w + 2) * LD + 8 * j];
            b0[j] = t & 1 ? u.y : u.x;
            b1[j] = t & 1 ? v.y : v.x;
            q0[j] = t & 1 ? u.x : -u.y;
            q1[j] = t & 1 ? v.x : -v.y;
        }
        const double *p = ar + w * LD * 2;
        const double a[4] = {p[0], p[16], p[4 * LD], p[4 * LD + 16]};
#pragma unroll
        for (int j = 0; j < NB; ++j)
            if (use[j]) {
                mma_f64(re[j], a[0], a[1], a[2], a[3], b0[j], b1[j]);
                mma_f64(im[j], a[0], a[1], a[2], a[3], q0[j], q1[j]);
            }
    };
    load(0);
    if (nst > 1) load(1);
    for (int64_t st = 0; st < nst - 1; ++st) {
        arrive(st, true);
#pragma unroll
        for (int w = 0; w < GF_KW; w += 4) four(w);
    }
    // of the last stage only the windows that are there: sums of a few windows are one stage
    arrive(nst - 1, false);
    const int kw = (int)(nw - (nst - 1) * GF_KW);
#pragma unroll
    for (int w = 0; w < GF_KW; w += 4)
        if (w < kw) four(w);
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = rw + g + 8 * (e >> 1), c = cw + 8 * j + gf_column(2 * t + (e & 1));
            if (c >= M || r > c) continue;
            if (out) put_hermitian(out + (int64_t)f * M * M, M, r, c, re[j][e], im[j][e], scale);
            else base[(int64_t)r * M + c] = make_double2(re[j][e], im[j][e]);
        }
}

static int gram_f64_launch(const void *spec, int M, int64_t nw, int nbins, void *csm, void *out, double scale,
                           cudaStream_t s)
{
    const int T = (M + GF_T - 1) / GF_T;
    const bool narrow = (int64_t)T * (T + 1) / 2 * nbins < GF_NARROW;
    const auto kernel = narrow ? gram_f64_kernel<1> : gram_f64_kernel<2>;
    const int TC = narrow ? (M + 15) / 16 : T, per = narrow ? 2 : 1;
    int tiles = 0;
    for (int ti = 0; ti < T; ++ti) tiles += TC - per * ti;
    if (const int st = allow_smem(kernel, GF_SMEM, GF_SMEM)) return st;
    kernel<<<dim3(tiles, nbins), 128, GF_SMEM, s>>>(reinterpret_cast<const double2 *>(spec), M, nw,
                                                    reinterpret_cast<double2 *>(csm), reinterpret_cast<double2 *>(out),
                                                    scale);
    return check_launch();
}

// ------------------------------------------------------------------------------------------------
// Hermitian completion + scale, 32x32 tiles through shared memory for the transposed half.
// ------------------------------------------------------------------------------------------------
template <bool C64>
__global__ void __launch_bounds__(256) finalize_kernel(const void *__restrict__ up_, int M, double scale,
                                                       double2 *__restrict__ out)
{
    using V = typename std::conditional<C64, float2, double2>::type;
    __shared__ double2 tile[32][33];
    const V *up = reinterpret_cast<const V *>(up_);
    const int f = blockIdx.z;
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    const V *ub = up + (int64_t)f * M * M;
    double2 *ob = out + (int64_t)f * M * M;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (r0 <= c0 + 31) {
        // tile touches the upper triangle: direct read (lower part of a diagonal tile handled below)
        for (int i = ty; i < 32; i += 8) {
            const int r = r0 + i, c = c0 + tx;
            if (r < M && c < M && r <= c) {
                const V v = ub[(int64_t)r * M + c];
                ob[(int64_t)r * M + c] = make_double2((double)v.x * scale, (double)v.y * scale);
            }
        }
    }
    if (c0 <= r0 + 31) {
        // lower elements (r > c) read transposed from upper[c][r]
        for (int i = ty; i < 32; i += 8) {
            const int c = c0 + i, r = r0 + tx;  // coalesced read along r of upper[c][*]
            double2 v = make_double2(0.0, 0.0);
            if (r < M && c < M && c < r) {
                const V u = ub[(int64_t)c * M + r];
                v = make_double2((double)u.x, (double)u.y);
            }
            tile[i][tx] = v;
        }
        __syncthreads();
        for (int i = ty; i < 32; i += 8) {
            const int r = r0 + i, c = c0 + tx;
            if (r < M && c < M && r > c) {
                const double2 u = tile[tx][i];
                ob[(int64_t)r * M + c] = make_double2(u.x * scale, -u.y * scale);
            }
        }
    }
}

// Mics per CTA (a power of two) and threads: up to 74 KB of padded complex doubles and 256 threads, so that two or
// three CTAs share an SM and hide each other's barriers and FP64 latency; for blocks of FFT_WIDE_N samples and more, of
// which that would hold one or two mics and store 16 bytes of a row of complex64 spectra at a time, up to 150 KB and
// 512 threads.  At most 64 mics and no more than twice what the array has, and no more threads (64 at least) than the
// first pass has tasks: with 16 mics and 256 threads whatever the block, half the threads and more idled.  Measured
// (B200), whole complex128 CSM: 64 mics, block 128 100 -> 92 us, block 64 145 -> 122, block 32 120 -> 98, block 16 147 ->
// 118; 256 mics, block 128 1306 -> 1226; 113 mics, block 256 420 -> 410; 8 mics, block 128 45 -> 41.
constexpr size_t FFT_SMEM = 150 * 1024;   // the most of any block: 148 KB of a block of 16384
static int fft_threads(int N) { return N >= FFT_WIDE_N ? 512 : 256; }
static int fft_mics_per_block(int N, int M)
{
    const size_t most = N >= FFT_WIDE_N ? FFT_SMEM : 74 * 1024;
    int mpb = 64;
    while (mpb > 1 && (mpb >= 2 * M || (size_t)mpb * fft_stride(N / 2) * sizeof(double2) > most)) mpb >>= 1;
    return mpb;
}

// Launch the windowed FFT of `num_windows` windows in output form `out_form`.
int fft_launch(const void *samples, int sample_dtype, int out_form, int num_mics, int block_size, int hop,
               int64_t first_window, int64_t num_windows, const double *window, const double2 *tw, int bin_lo,
               int num_bins, void *out, int R, int KC, int64_t lo_elems, void *scratch, cudaStream_t s)
{
    if (block_size > FFT_MAX_N) {
        if (!scratch) return ACB_ERR_WORKSPACE;
        double2 *sc = reinterpret_cast<double2 *>(scratch);
        const dim3 gs((unsigned)num_mics, (unsigned)num_windows, (unsigned)(block_size / 2 / FFT_SUB_H));
        const size_t smem = (size_t)fft_stride(FFT_SUB_H) * sizeof(double2);
        if (sample_dtype == ACB_F32) {
            if (const int st = allow_smem(fft_sub_kernel<float>, smem, smem)) return st;
            fft_sub_kernel<float><<<gs, 256, smem, s>>>(reinterpret_cast<const float *>(samples), num_mics, block_size,
                                                        hop, first_window, window, tw, sc);
        } else {
            if (const int st = allow_smem(fft_sub_kernel<double>, smem, smem)) return st;
            fft_sub_kernel<double><<<gs, 256, smem, s>>>(reinterpret_cast<const double *>(samples), num_mics,
                                                         block_size, hop, first_window, window, tw, sc);
        }
        int st = check_launch();
        if (st) return st;
        const dim3 gc((unsigned)num_bins, (unsigned)num_windows);
        const int nt = num_mics < 256 ? (num_mics + 31) / 32 * 32 : 256;
        switch (out_form) {
        case OUT_C128: fft_combine_kernel<OUT_C128><<<gc, nt, 0, s>>>(sc, num_mics, block_size, num_windows, bin_lo,
                                                                      num_bins, tw, out, R, KC, lo_elems); break;
        case OUT_C64: fft_combine_kernel<OUT_C64><<<gc, nt, 0, s>>>(sc, num_mics, block_size, num_windows, bin_lo,
                                                                    num_bins, tw, out, R, KC, lo_elems); break;
        case OUT_TF32: fft_combine_kernel<OUT_TF32><<<gc, nt, 0, s>>>(sc, num_mics, block_size, num_windows, bin_lo,
                                                                      num_bins, tw, out, R, KC, lo_elems); break;
        default: fft_combine_kernel<OUT_BF16><<<gc, nt, 0, s>>>(sc, num_mics, block_size, num_windows, bin_lo,
                                                                num_bins, tw, out, R, KC, lo_elems); break;
        }
        return check_launch();
    }
    if (out_form >= OUT_TF32) {
        const int mpb4 = fft4_mics_per_block(block_size);
        if (mpb4 > 0) {
            // every tile row (16 R padded mics) and column (32 KC padded windows) is written
            const dim3 g4((unsigned)(R * 16 / mpb4), (unsigned)(KC * 32 / FFT4_WIN));
            const size_t smem4 = fft4_smem_bytes(block_size, mpb4);
            // vector width of the sample loads: V mics of a row at once where M and the base allow it; 16 bytes at
            // most for blocks of 128, whose tasks at 4 doubles would leave half the threads idle (64 mics: 229 us
            // for 300,000 samples, 210 at 2)
            const size_t es = sample_dtype == ACB_F32 ? 4 : 8;
            int vw = 1;
            for (int v = 4; v >= 2 && vw == 1; v >>= 1)
                if (v <= mpb4 && num_mics % v == 0 && (v * es <= 16 || block_size >= 256) &&
                    reinterpret_cast<uintptr_t>(samples) % (v * es < 16 ? v * es : 16) == 0)
                    vw = v;
#define ACB_FFT4_LAUNCH(TS, OF)                                                                                     \
    do {                                                                                                            \
        auto kern = fft4_tc_kernel<TS, OF>;                                                                         \
        if (const int st_ = allow_smem(kern, smem4, 200 * 1024)) return st_;                                        \
        kern<<<g4, fft4_threads(block_size), smem4, s>>>(reinterpret_cast<const TS *>(samples), num_mics, block_size,   \
                                    hop, first_window, num_windows, mpb4, vw, window, tw, bin_lo, num_bins, out, R, KC, lo_elems);    \
    } while (0)
            if (sample_dtype == ACB_F32) {
                if (out_form == OUT_TF32) ACB_FFT4_LAUNCH(float, OUT_TF32);
                else ACB_FFT4_LAUNCH(float, OUT_BF16);
            } else {
                if (out_form == OUT_TF32) ACB_FFT4_LAUNCH(double, OUT_TF32);
                else ACB_FFT4_LAUNCH(double, OUT_BF16);
            }
#undef ACB_FFT4_LAUNCH
            return check_launch();
        }
    }
    const int mpb = fft_mics_per_block(block_size, num_mics);
    const dim3 g1((num_mics + mpb - 1) / mpb, (unsigned)num_windows);
    const size_t smem = (size_t)mpb * fft_stride(block_size / 2) * sizeof(double2);
#define ACB_FFT_LAUNCH(TS, OF)                                                                                    \
    do {                                                                                                          \
        auto kern = fft_window_kernel<TS, OF>;                                                                    \
        if (const int st_ = allow_smem(kern, smem, FFT_SMEM)) return st_;                                         \
        const int nt = max(64, min(fft_threads(block_size), mpb * (block_size / 16)));                             \
        kern<<<g1, nt, smem, s>>>(reinterpret_cast<const TS *>(samples), num_mics, block_size, hop, \
                                   first_window, num_windows, mpb, window, tw, bin_lo, num_bins, out, R, KC, lo_elems);        \
    } while (0)
#define ACB_FFT_FORMS(TS)                                                \
    switch (out_form) {                                                  \
    case OUT_C128: ACB_FFT_LAUNCH(TS, OUT_C128); break;                  \
    case OUT_C64: ACB_FFT_LAUNCH(TS, OUT_C64); break;                    \
    case OUT_TF32: ACB_FFT_LAUNCH(TS, OUT_TF32); break;                  \
    default: ACB_FFT_LAUNCH(TS, OUT_BF16); break;                        \
    }
    if (sample_dtype == ACB_F32) { ACB_FFT_FORMS(float) }
    else { ACB_FFT_FORMS(double) }
#undef ACB_FFT_FORMS
#undef ACB_FFT_LAUNCH
    return check_launch();
}

}  // namespace acb

using namespace acb;

extern "C" {

const char *acb_status_string(int s)
{
    switch (s) {
    case ACB_OK: return "ok";
    case ACB_ERR_SHAPE: return "size or shape out of range";
    case ACB_ERR_ARG: return "invalid argument";
    case ACB_ERR_CUDA: return "CUDA error";
    case ACB_ERR_UNSUPPORTED: return "unsupported by this build";
    case ACB_ERR_WORKSPACE: return "workspace missing or too small";
    case ACB_ERR_TIMEOUT: return "device-side wait timed out";
    default: return "unknown status";
    }
}

int acb_abi_version(void) { return 2; }   // 2: tensor-core tuning fields, TC CSM forms, eigenvalue maps

const char *acb_last_cuda_error(void) { return g_last_cuda_error.c_str(); }

int acb_calc_csm_c128(void *csm, const void *spec, int num_freqs, int num_mics, void *stream)
{
    if (!csm || !spec) return ACB_ERR_ARG;
    if (num_freqs <= 0 || num_mics <= 0) return ACB_ERR_SHAPE;
    return gram_f64_launch(spec, num_mics, 1, num_freqs, csm, nullptr, 1.0, as_stream(stream));
}

int acb_calc_csm_c64(void *csm, const void *spec, int num_freqs, int num_mics, void *stream)
{
    if (!csm || !spec) return ACB_ERR_ARG;
    if (num_freqs <= 0 || num_mics <= 0) return ACB_ERR_SHAPE;
    return gram_c64_launch(spec, num_mics, 1, num_freqs, csm, nullptr, 1.0, as_stream(stream));
}

size_t acb_csm_workspace_bytes(int num_mics, int num_bins, int64_t num_windows, int precision)
{
    if (num_mics <= 0 || num_bins <= 0 || num_windows <= 0) return 0;
    if (precision == ACB_CSM_TC_TF32 || precision == ACB_CSM_TC_BF16X3)
        return csm_tc_workspace_bytes(num_mics, num_bins, num_windows);
    const size_t es = precision == ACB_C64 ? 8 : 16;
    return (size_t)num_mics * (size_t)num_bins * (size_t)num_windows * es;
}

size_t acb_csm_workspace_bytes_block(int num_mics, int num_bins, int64_t num_windows, int precision, int block_size)
{
    const size_t base = acb_csm_workspace_bytes(num_mics, num_bins, num_windows, precision);
    if (base == 0) return 0;
    const size_t sc = fft_scratch_bytes(num_mics, block_size, num_windows);
    return sc ? (base + 255) / 256 * 256 + sc : base;
}

// Windows into sums: added to csm_upper, or, with csm_out, written as the finished matrix (scale applied, Hermitian).
static int csm_windows(const void *samples, int sample_dtype, int64_t num_samples, int num_mics, int block_size,
                       int hop, int64_t first_window, int64_t num_windows, const double *window, const void *twiddle,
                       int bin_lo, int num_bins, int precision, void *csm_upper, double scale, void *csm_out,
                       void *workspace, size_t workspace_bytes, void *stream)
{
    if (!samples || !window || !twiddle || (!csm_upper && !csm_out)) return ACB_ERR_ARG;
    if (sample_dtype != ACB_F32 && sample_dtype != ACB_F64) return ACB_ERR_ARG;
    const bool tc = precision == ACB_CSM_TC_TF32 || precision == ACB_CSM_TC_BF16X3;
    if (precision != ACB_C128 && precision != ACB_C64 && !tc) return ACB_ERR_ARG;
    if (num_mics <= 0 || num_windows < 0 || first_window < 0 || hop <= 0) return ACB_ERR_SHAPE;
    if (tc && csm_tc_row_tiles(num_mics) > 252) return ACB_ERR_UNSUPPORTED;
    if (block_size < 16 || (block_size & (block_size - 1))) return ACB_ERR_SHAPE;
    if (block_size > 4 * FFT_MAX_N) return ACB_ERR_UNSUPPORTED;
    if (bin_lo < 0 || num_bins <= 0 || bin_lo + num_bins > block_size / 2 + 1) return ACB_ERR_SHAPE;
    if (num_windows == 0) return csm_out ? ACB_ERR_SHAPE : ACB_OK;
    if ((first_window + num_windows - 1) * (int64_t)hop + block_size > num_samples) return ACB_ERR_SHAPE;
    if (num_windows > 65535) return ACB_ERR_SHAPE;  // one grid row per window
    const size_t need = acb_csm_workspace_bytes_block(num_mics, num_bins, num_windows, precision, block_size);
    if (!workspace || workspace_bytes < need) return ACB_ERR_WORKSPACE;
    // blocks above 16384 samples: the FFT's sub-spectra go to a scratch region after the spectra
    void *scratch = nullptr;
    if (block_size > FFT_MAX_N)
        scratch = reinterpret_cast<uint8_t *>(workspace) +
                  (acb_csm_workspace_bytes(num_mics, num_bins, num_windows, precision) + 255) / 256 * 256;
    cudaStream_t s = as_stream(stream);
    const double2 *tw = reinterpret_cast<const double2 *>(twiddle);
    if (tc)
        return csm_tc_accumulate(samples, sample_dtype, num_mics, block_size, hop, first_window, num_windows, window,
                                 tw, bin_lo, num_bins, precision == ACB_CSM_TC_TF32, csm_upper, csm_out, scale,
                                 workspace, scratch, s);
    int st = fft_launch(samples, sample_dtype, precision == ACB_C64 ? OUT_C64 : OUT_C128, num_mics, block_size, hop,
                        first_window, num_windows, window, tw, bin_lo, num_bins, workspace, 0, 0, 0, scratch, s);
    if (st) return st;
    auto gram = precision == ACB_C64 ? gram_c64_launch : gram_f64_launch;
    return gram(workspace, num_mics, num_windows, num_bins, csm_upper, csm_out, scale, s);
}

int acb_csm_accumulate(const void *samples, int sample_dtype, int64_t num_samples, int num_mics, int block_size,
                       int hop, int64_t first_window, int64_t num_windows, const double *window,
                       const void *twiddle, int bin_lo, int num_bins, int precision, void *csm_upper,
                       void *workspace, size_t workspace_bytes, void *stream)
{
    if (!csm_upper) return ACB_ERR_ARG;
    return csm_windows(samples, sample_dtype, num_samples, num_mics, block_size, hop, first_window, num_windows, window,
                       twiddle, bin_lo, num_bins, precision, csm_upper, 1.0, nullptr, workspace, workspace_bytes,
                       stream);
}

int acb_csm_finished(const void *samples, int sample_dtype, int64_t num_samples, int num_mics, int block_size,
                     int hop, int64_t first_window, int64_t num_windows, const double *window, const void *twiddle,
                     int bin_lo, int num_bins, int precision, double scale, void *csm_out, void *workspace,
                     size_t workspace_bytes, void *stream)
{
    if (!csm_out) return ACB_ERR_ARG;
    return csm_windows(samples, sample_dtype, num_samples, num_mics, block_size, hop, first_window, num_windows, window,
                       twiddle, bin_lo, num_bins, precision, nullptr, scale, csm_out, workspace, workspace_bytes,
                       stream);
}

int acb_csm_finalize(const void *csm_upper, int num_bins, int num_mics, int precision, double scale, void *csm_out,
                     void *stream)
{
    if (!csm_upper || !csm_out) return ACB_ERR_ARG;
    if (precision != ACB_C128 && precision != ACB_C64) return ACB_ERR_ARG;
    if (num_bins <= 0 || num_mics <= 0 || num_bins > 65535) return ACB_ERR_SHAPE;
    const int T = (num_mics + 31) / 32;
    const dim3 g(T, T, num_bins);
    if (precision == ACB_C64)
        finalize_kernel<true><<<g, 256, 0, as_stream(stream)>>>(csm_upper, num_mics, scale, (double2 *)csm_out);
    else
        finalize_kernel<false><<<g, 256, 0, as_stream(stream)>>>(csm_upper, num_mics, scale, (double2 *)csm_out);
    return check_launch();
}

}  // extern "C"
