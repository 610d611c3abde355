// CLEAN-SC (BeamformerCleansc._calc, acoular/fbeamform.py:1424-1490) on the device, all bins of a request
// at once, with no host synchronisation inside the iterations.
//
// Per bin the reference iterates j = 0 .. J-1 on the conventional map h (full-CSM form, no clipping):
//   xi = argmax h (first index), hmax = h[xi], powers[j] = hmax, result[xi] += damp hmax (float32 result);
//   stop when j > stopn and hmax > powers[j - stopn];
//   w = conj(steer_vector(f, xi) sqrt(norm)) (the transfer of calcTransfer, fastFuncs.py:857-897, and the
//   steering formulas of SteeringVector._steer_funcs_freq, fbeamform.py:145-153);
//   D1 = (C^T - diag C) w / hmax; 20 fixed-point steps hh = (D1 + |hh|^2 w) / sqrt(1 + sum |w|^2 |hh|^2);
//   h -= damp * map of the single component (hmax, conj(hh)); C -= damp hmax (hh hh^H)^T.
//
// Device schedule (arrays and grids that fit run all iterations of a bin in one cluster, cleansc_cluster_kernel; this is
// the one for the others): the steering vectors of every grid point are synthesised once per bin (normalised for
// the steering type, cleansc_steer_kernel); then per iteration cleansc_step_kernel (one CTA per bin: the
// map update h -= damp h1 fused with the argmax, then the peak's steering vector, D1, the fixed point and
// the CSM update) and the eigenvalue-form map of the new component on the cached steering vectors
// (map_eig_custom_launch, E = 1), both over all bins; a bin that has stopped clears its active flag and
// both kernels skip it.  The scalar arithmetic of the steering
// formulas and of the divisions follows numpy's complex arithmetic (x / y for a real y is x * (1 / y));
// sums (einsum, BLAS dot products) are formed in mic order.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <cooperative_groups.h>

#include "common.cuh"
#include "map_internal.h"

namespace cg = cooperative_groups;

namespace acb {

constexpr int kCscThreads = 512;
constexpr int kCscWarps = kCscThreads / 32;

struct CscArgs {
    int M;
    int64_t G;
    int J;
    int stopn;
    double damp;
    double sqrt_norm;
    int steer_type;
    const double *k;
    const double *r0;   // given distances (non-Euclidean environments), else nullptr
    const double *rm;
    const double *mpos;
    const double *gpos;
    int ref_mode;
    double ref0, ref1, ref2, ref_dist;
    int faithful;
    const uint64_t *table;
    uint64_t mask;
    double2 *csm;      // (B, M, M) working copy, updated
    double *h;         // (B, G) map, updated
    const double *h1;  // (B, G) map of the previous iteration's component
    double *powers;    // (B, J)
    float *result;     // (B, G)
    int *active;       // (B)
    double *lam;       // (B) component eigenvalue (hmax)
    double2 *vec;      // (B, M) component vector conj(hh)
    const double2 *given;   // (B, G, M) a steering object's own vectors (custom steering), else nullptr
};

// numpy's complex division (Smith's method with a reciprocal scale), for a real divisor y = (yr, 0).
__device__ __forceinline__ double2 cdiv_real(double2 x, double yr)
{
    const double rat = __ddiv_rn(0.0, yr);
    const double scl = __ddiv_rn(1.0, __dadd_rn(yr, __dmul_rn(0.0, rat)));
    return make_double2(__dmul_rn(__dadd_rn(x.x, __dmul_rn(x.y, rat)), scl),
                        __dmul_rn(__dsub_rn(x.y, __dmul_rn(x.x, rat)), scl));
}

// numpy's complex division x / y for a general y.
__device__ __forceinline__ double2 cdiv(double2 x, double2 y)
{
    if (fabs(y.x) >= fabs(y.y)) {
        const double rat = __ddiv_rn(y.y, y.x);
        const double scl = __ddiv_rn(1.0, __dadd_rn(y.x, __dmul_rn(y.y, rat)));
        return make_double2(__dmul_rn(__dadd_rn(x.x, __dmul_rn(x.y, rat)), scl),
                            __dmul_rn(__dsub_rn(x.y, __dmul_rn(x.x, rat)), scl));
    }
    const double rat = __ddiv_rn(y.x, y.y);
    const double scl = __ddiv_rn(1.0, __dadd_rn(y.y, __dmul_rn(y.x, rat)));
    return make_double2(__dmul_rn(__dadd_rn(__dmul_rn(x.x, rat), x.y), scl),
                        __dmul_rn(__dsub_rn(__dmul_rn(x.y, rat), x.x), scl));
}

// Steering vectors of every grid point for the component maps, normalised so that the custom-steering
// quadratic form equals the steering type's map: v_m = e^{-i fl32(k r_m)} (times r_m for 'inverse',
// over r_m for 'true level' / 'true location'; the map kernel's synthesis), divided by M (classic),
// M r0 (inverse), r0 S (true level) or sqrt(M S) (true location), S = sum r^2 or sum 1/r^2.
// One warp per grid point, lanes over the mics; out (B, G, M), or with MIC_MAJOR (B, M, G): a warp then takes four of
// its CTA's 32 points, which go out through a shared-memory tile [M][33].
template <bool MIC_MAJOR>
__global__ void __launch_bounds__(256) cleansc_steer_kernel(CscArgs a, double2 *__restrict__ out)
{
    extern __shared__ double2 st_sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b = blockIdx.y;
    const int M = a.M;
    const double k = a.k[b];
    const SincosTable sct = sincos_table(a.table, a.mask, a.faithful != 0);
    constexpr int kPer = MIC_MAJOR ? 4 : 1;   // points per warp
    const int64_t gb = (int64_t)blockIdx.x * 8 * kPer;
    for (int i = 0; i < kPer; ++i) {
        const int pt = warp * kPer + i;
        const int64_t g = gb + pt;
        if (g >= a.G) break;
        double gx = 0, gy = 0, gz = 0, r0;
        if (a.rm) {
            r0 = a.r0[g];
        } else {
            gx = a.gpos[g];
            gy = a.gpos[a.G + g];
            gz = a.gpos[2 * a.G + g];
            r0 = a.ref_mode == 1 ? a.ref_dist : dist3(gx, gy, gz, a.ref0, a.ref1, a.ref2);
        }
        double2 *o = MIC_MAJOR ? st_sm + pt : out + ((int64_t)b * a.G + g) * M;
        const int64_t step = MIC_MAJOR ? 33 : 1;
        double S = 0.0;
        for (int m = lane; m < M; m += 32) {
            const double r = a.rm ? a.rm[g * M + m] : dist3(gx, gy, gz, a.mpos[m], a.mpos[M + m], a.mpos[2 * M + m]);
            const float arg = __double2float_rn(__dmul_rn(k, r));
            float c, sn;
            sincos_f32_arg(arg, sct, c, sn);
            double2 v = make_double2((double)c, -(double)sn);
            if (a.steer_type == 2) {
                v.x = __dmul_rn(v.x, r);
                v.y = __dmul_rn(v.y, r);
                S += r * r;
            } else if (a.steer_type >= 3) {
                v.x = __ddiv_rn(v.x, r);
                v.y = __ddiv_rn(v.y, r);
                S += 1.0 / (r * r);
            }
            o[m * step] = v;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) S += __shfl_xor_sync(0xffffffffu, S, off);
        const double Md = (double)M;
        const double nf =
            a.steer_type == 1 ? Md : a.steer_type == 2 ? Md * r0 : a.steer_type == 3 ? r0 * S : sqrt(Md * S);
        const double inv = 1.0 / nf;
        __syncwarp();
        for (int m = lane; m < M; m += 32) {
            const double2 v = o[m * step];
            o[m * step] = make_double2(v.x * inv, v.y * inv);
        }
    }
    if (!MIC_MAJOR) return;
    __syncthreads();
    for (int m = warp; m < M; m += 8)
        if (gb + lane < a.G) out[((int64_t)b * M + m) * a.G + gb + lane] = st_sm[m * 33 + lane];
}

__global__ void cleansc_init_kernel(int *active, float *result, int64_t n_result, int B)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < B) active[i] = 1;
    if (i < n_result) result[i] = 0.0f;
}

__global__ void __launch_bounds__(kCscThreads) cleansc_step_kernel(CscArgs a, int j)
{
    extern __shared__ double sm[];
    const int b = blockIdx.x;
    if (!a.active[b]) return;
    const int M = a.M;
    const int64_t G = a.G;
    double2 *w = reinterpret_cast<double2 *>(sm);   // [M] steering of the peak, then its conjugate
    double2 *d1 = w + M;                              // [M]
    double2 *hh = d1 + M;                             // [M]
    double *ww = reinterpret_cast<double *>(hh + M);  // [M] |w|^2
    __shared__ double red_v[kCscWarps];
    __shared__ int64_t red_i[kCscWarps];
    __shared__ double scratch[kCscWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *h = a.h + (int64_t)b * G;
    const double *h1 = a.h1 + (int64_t)b * G;

    // 1. h -= damp h1 (the previous iteration's component), fused with the argmax (first index of the max)
    double best = -INFINITY;
    int64_t bi = G;
    for (int64_t g = threadIdx.x; g < G; g += kCscThreads) {
        double v = h[g];
        if (j > 0) {
            v = __dsub_rn(v, __dmul_rn(a.damp, h1[g]));
            h[g] = v;
        }
        if (v > best || (v == best && g < bi)) {
            best = v;
            bi = g;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int64_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) {
            best = ov;
            bi = oi;
        }
    }
    if (lane == 0) {
        red_v[warp] = best;
        red_i[warp] = bi;
    }
    __syncthreads();
    best = red_v[0];
    bi = red_i[0];
    for (int wv = 1; wv < kCscWarps; ++wv)
        if (red_v[wv] > best || (red_v[wv] == best && red_i[wv] < bi)) {
            best = red_v[wv];
            bi = red_i[wv];
        }
    if (bi >= G) {   // no comparable value (NaN map): stop this bin
        if (threadIdx.x == 0) a.active[b] = 0;
        return;
    }
    const int64_t xi = bi;
    const double hmax = best;
    const bool stop = j > a.stopn && hmax > a.powers[(int64_t)b * a.J + j - a.stopn];
    __syncthreads();   // every thread has read powers before thread 0 writes this iteration's entry
    if (threadIdx.x == 0) {
        a.powers[(int64_t)b * a.J + j] = hmax;
        float *r = a.result + (int64_t)b * G + xi;
        *r = __double2float_rn(__dadd_rn((double)*r, __dmul_rn(a.damp, hmax)));
        if (stop) a.active[b] = 0;
    }
    if (stop) return;

    if (a.given) {
        // 2'. custom steering: the object's own steering vector of the peak, w = conj(v sqrt(norm))
        const double2 *v = a.given + ((int64_t)b * G + xi) * M;
        for (int m = threadIdx.x; m < M; m += kCscThreads) {
            const double2 x = v[m];
            const double2 c = make_double2(__dmul_rn(x.x, a.sqrt_norm), -__dmul_rn(x.y, a.sqrt_norm));
            w[m] = c;
            ww[m] = __dadd_rn(__dmul_rn(c.x, c.x), __dmul_rn(c.y, c.y));
            hh[m] = c;
        }
        __syncthreads();
    } else {
    // 2. steering vector of the peak: transfer x_m = (cos p - i sin p) r0 / rm, p = fl32(k (rm - r0))
    const double k = a.k[b];
    const SincosTable sct = sincos_table(a.table, a.mask, a.faithful != 0);
    double gx = 0, gy = 0, gz = 0, r0x;
    if (a.rm) {
        r0x = a.r0[xi];
    } else {
        gx = a.gpos[xi];
        gy = a.gpos[G + xi];
        gz = a.gpos[2 * G + xi];
        r0x = a.ref_mode == 1 ? a.ref_dist : dist3(gx, gy, gz, a.ref0, a.ref1, a.ref2);
    }
    for (int m = threadIdx.x; m < M; m += kCscThreads) {
        const double rmm = a.rm ? a.rm[xi * M + m] : dist3(gx, gy, gz, a.mpos[m], a.mpos[M + m], a.mpos[2 * M + m]);
        const float arg = __double2float_rn(__dmul_rn(k, __dsub_rn(rmm, r0x)));
        float c, s;
        sincos_f32_arg(arg, sct, c, s);
        const double xr = __ddiv_rn(__dmul_rn((double)c, r0x), rmm);
        const double xim = __ddiv_rn(__dmul_rn(-(double)s, r0x), rmm);
        w[m] = make_double2(xr, xim);
        ww[m] = __dadd_rn(__dmul_rn(xr, xr), __dmul_rn(xim, xim));   // Re x conj(x)
    }
    __syncthreads();
    double nrm = 0.0;
    if (a.steer_type >= 3) {   // einsum('ij,ij->i', x, x.conj()), in mic order
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int m = 0; m < M; ++m) t = __dadd_rn(t, ww[m]);
            scratch[0] = t;
        }
        __syncthreads();
        nrm = scratch[0];
        if (a.steer_type == 4) nrm = __dsqrt_rn(__dmul_rn(nrm, (double)M));
        __syncthreads();
    }
    for (int m = threadIdx.x; m < M; m += kCscThreads) {
        double2 x = w[m];
        if (a.steer_type == 1) {   // x / |x| / M
            x = cdiv_real(cdiv_real(x, hypot(x.x, x.y)), (double)M);
        } else if (a.steer_type == 2) {   // 1 / conj(x) / M
            x = cdiv_real(cdiv(make_double2(1.0, 0.0), make_double2(x.x, -x.y)), (double)M);
        } else {   // x / sum |x|^2  |  x / sqrt(sum |x|^2 M)
            x = cdiv_real(x, nrm);
        }
        // * sqrt(normfactor), then the conjugate
        const double2 v = make_double2(__dmul_rn(x.x, a.sqrt_norm), -__dmul_rn(x.y, a.sqrt_norm));
        w[m] = v;
        ww[m] = __dadd_rn(__dmul_rn(v.x, v.x), __dmul_rn(v.y, v.y));   // conj(w) w
        hh[m] = v;
    }
    __syncthreads();
    }

    // 3. D1 = (C^T - diag C) w / hmax: D1_a = sum_{m != a} C[m][a] w_m, a warp per row a
    const double2 *C = a.csm + (int64_t)b * M * M;
    for (int r = warp; r < M; r += kCscWarps) {
        double sr = 0.0, si = 0.0;
        for (int m = lane; m < M; m += 32) {
            if (m == r) continue;
            const double2 c = C[(int64_t)m * M + r];
            const double2 v = w[m];
            sr = fma(c.x, v.x, fma(-c.y, v.y, sr));
            si = fma(c.x, v.y, fma(c.y, v.x, si));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sr += __shfl_xor_sync(0xffffffffu, sr, o);
            si += __shfl_xor_sync(0xffffffffu, si, o);
        }
        if (lane == 0) d1[r] = cdiv_real(make_double2(sr, si), hmax);
    }
    __syncthreads();

    // 4. 20 fixed-point steps: hh = (D1 + |hh|^2 w) / sqrt(1 + sum_m |w_m|^2 |hh_m|^2), in warp 0 alone
    //    (each lane owns mics lane, lane + 32, ...; the sum is a shuffle reduction, no block barrier)
    if (warp == 0) {
        for (int it = 0; it < 20; ++it) {
            double part = 0.0;
            for (int m = lane; m < M; m += 32) {
                const double2 q = hh[m];
                part = fma(ww[m], __dadd_rn(__dmul_rn(q.x, q.x), __dmul_rn(q.y, q.y)), part);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            const double den = __dsqrt_rn(__dadd_rn(1.0, part));
            for (int m = lane; m < M; m += 32) {
                const double2 q = hh[m];
                const double H = __dadd_rn(__dmul_rn(q.x, q.x), __dmul_rn(q.y, q.y));
                const double2 v = w[m], d = d1[m];
                hh[m] = cdiv_real(make_double2(__dadd_rn(d.x, __dmul_rn(H, v.x)), __dadd_rn(d.y, __dmul_rn(H, v.y))),
                                  den);
            }
            __syncwarp();
        }
    }
    __syncthreads();

    // 5. C[r][c] -= damp (hmax (hh_c conj(hh_r))); 6. the component for the map: (hmax, conj(hh))
    double2 *Cw = a.csm + (int64_t)b * M * M;
    for (int64_t e = threadIdx.x; e < (int64_t)M * M; e += kCscThreads) {
        const int r = (int)(e / M), c = (int)(e % M);
        const double2 x = hh[c], y = hh[r];
        const double pr = __dsub_rn(__dmul_rn(x.x, y.x), __dmul_rn(x.y, -y.y));
        const double pi = __dadd_rn(__dmul_rn(x.x, -y.y), __dmul_rn(x.y, y.x));
        double2 v = Cw[e];
        v.x = __dsub_rn(v.x, __dmul_rn(a.damp, __dmul_rn(hmax, pr)));
        v.y = __dsub_rn(v.y, __dmul_rn(a.damp, __dmul_rn(hmax, pi)));
        Cw[e] = v;
    }
    for (int m = threadIdx.x; m < M; m += kCscThreads) a.vec[(int64_t)b * M + m] = make_double2(hh[m].x, -hh[m].y);
    if (threadIdx.x == 0) a.lam[b] = hmax;
}

// ------------------------------------------------------------------------------------------------
// All iterations of a bin in one cluster of one to eight CTAs (csc_ctas), for arrays whose CSM fits each CTA's shared memory and grids
// whose map fits the cluster's registers (csc_cluster_fits).  Every CTA keeps the whole CSM and does the step's small
// work for itself, the same bits in each; the grid points are split over the CTAs (a thread keeps the map values of up
// to four), and the argmax is the one exchange: each CTA stores its candidate into every CTA's slots (two sets, used
// alternately, so that one cluster barrier per iteration suffices) and picks the best of them.  The component's
// map reads the steering vectors mic-major, lanes along the grid.  A bin's result has the same bits whatever the cluster.
// Bound: the serial chain of an iteration (the fixed point's sums and reciprocal square roots at the latency of FP64
// instructions).  Two launches per iteration cost more than that: 5 bins x 1681 points x 64 mics, 128 iterations
// 3.1 -> 1.07 ms (B200);
// 8 bins x 3600 points x 112 mics, 60 iterations 4.3 -> 2.1; 3 bins x 8099 points x 33 mics 2.3 -> 1.17.
// The fixed point stops when a step leaves every value as it was: the remaining ones would change nothing.
// ------------------------------------------------------------------------------------------------
constexpr int kCscMaxCtas = 8, kCscClThreads = 256, kCscPoints = 4, kCscHistory = 64;
constexpr int kCscClMics = 112;

constexpr size_t kCscStepSmem = 2048 * (3 * sizeof(double2) + sizeof(double));   // cleansc_step_kernel's at the most mics

struct CscPeak {
    double v;
    long long g;
};

static __host__ __device__ size_t csc_cluster_smem(int M)
{
    return ((size_t)M * M + 3 * M + kCscClThreads) * sizeof(double2) + (size_t)M * sizeof(double);
}

__device__ __forceinline__ void better(double &v, int64_t &g, double ov, int64_t og)
{
    if (ov > v || (ov == v && og < g)) {   // the first index of the maximum
        v = ov;
        g = og;
    }
}

// NC: the cluster's CTAs, 0 where they are known at run time only (eight of them 1 to 2 % slower).
template <int NP, int AHEAD, int MINB, int NC>
__global__ void __launch_bounds__(kCscClThreads, MINB) cleansc_cluster_kernel(CscArgs a, const double2 *__restrict__ steer,
                                                                        int r_diag, double norm)
{
    extern __shared__ double2 cl_sm[];
    __shared__ CscPeak peaks[2][kCscMaxCtas], wpeak[kCscClThreads / 32];
    __shared__ double powers[kCscHistory];   // the last peaks, by iteration modulo its length
    cg::cluster_group cluster = cg::this_cluster();
    const int nctas = NC ? NC : (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int b = blockIdx.x / nctas;
    const int M = a.M, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t G = a.G;
    double2 *C = cl_sm, *w = C + M * M, *d1 = w + M, *hh = d1 + M, *part = hh + M;
    double *ww = reinterpret_cast<double *>(part + kCscClThreads);
    double2 *Cg = a.csm + (int64_t)b * M * M;
    for (int e = tid; e < M * M; e += kCscClThreads) C[e] = Cg[e];
    // this thread's grid points and their map values
    double h[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        const int64_t g = (int64_t)q * nctas * kCscClThreads + rank * kCscClThreads + tid;
        h[q] = g < G ? a.h[(int64_t)b * G + g] : -INFINITY;
    }
    const double k = a.k[b];
    const SincosTable sct = sincos_table(a.table, a.mask, a.faithful != 0);
    const double2 *sv = steer + (int64_t)b * M * G;
    const int Mp = (M + 31) & ~31, ngrp = kCscClThreads / Mp;   // matvec: ngrp threads per row
    cluster.sync();   // every CTA runs before the first remote store

    for (int j = 0; j < a.J; ++j) {
        // 1. the peak (and, after the first iteration, nothing else: h was updated at the end of the last one)
        double best = -INFINITY;
        int64_t bi = G;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const int64_t g = (int64_t)q * nctas * kCscClThreads + rank * kCscClThreads + tid;
            if (g < G) better(best, bi, h[q], g);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int64_t og = __shfl_xor_sync(0xffffffffu, bi, o);
            better(best, bi, ov, og);
        }
        if (lane == 0) wpeak[warp] = CscPeak{best, bi};
        __syncthreads();
        if (tid < nctas) {
            for (int u = 0; u < kCscClThreads / 32; ++u) better(best, bi, wpeak[u].v, wpeak[u].g);
            *cluster.map_shared_rank(&peaks[j & 1][rank], tid) = CscPeak{best, bi};
        }
        cluster.sync();
        best = -INFINITY;
        bi = G;
#pragma unroll
        for (int u = 0; u < kCscMaxCtas; ++u)
            if (u < nctas) better(best, bi, peaks[j & 1][u].v, peaks[j & 1][u].g);
        if (bi >= G) break;   // no comparable value (NaN map)
        const int64_t xi = bi;
        const double hmax = best;
        const bool stop = j > a.stopn && hmax > powers[(j - a.stopn) % kCscHistory];
        if (rank == 0 && tid == kCscClThreads - 1) {
            float *r = a.result + (int64_t)b * G + xi;
            *r = __double2float_rn(__dadd_rn((double)*r, __dmul_rn(a.damp, hmax)));
        }
        if (stop) break;   // the same decision in every CTA

        // 2. steering vector of the peak: transfer x_m = (cos p - i sin p) r0 / rm, p = fl32(k (rm - r0))
        double2 x = make_double2(0.0, 0.0);
        if (tid < M) {
            double gx = 0, gy = 0, gz = 0, r0x;
            if (a.rm) {
                r0x = a.r0[xi];
            } else {
                gx = a.gpos[xi];
                gy = a.gpos[G + xi];
                gz = a.gpos[2 * G + xi];
                r0x = a.ref_mode == 1 ? a.ref_dist : dist3(gx, gy, gz, a.ref0, a.ref1, a.ref2);
            }
            const double rmm =
                a.rm ? a.rm[xi * M + tid] : dist3(gx, gy, gz, a.mpos[tid], a.mpos[M + tid], a.mpos[2 * M + tid]);
            const float arg = __double2float_rn(__dmul_rn(k, __dsub_rn(rmm, r0x)));
            float c, s;
            sincos_f32_arg(arg, sct, c, s);
            x = make_double2(__ddiv_rn(__dmul_rn((double)c, r0x), rmm), __ddiv_rn(__dmul_rn(-(double)s, r0x), rmm));
            ww[tid] = __dadd_rn(__dmul_rn(x.x, x.x), __dmul_rn(x.y, x.y));   // Re x conj(x)
        }
        __syncthreads();
        if (tid == 0) powers[j % kCscHistory] = hmax;   // read again after more barriers only
        double nrm = 0.0;
        if (a.steer_type >= 3) {   // einsum('ij,ij->i', x, x.conj())
            for (int m = lane; m < M; m += 32) nrm += ww[m];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
            if (a.steer_type == 4) nrm = __dsqrt_rn(__dmul_rn(nrm, (double)M));
        }
        if (tid < M) {
            if (a.steer_type == 1) {   // x / |x| / M
                x = cdiv_real(cdiv_real(x, hypot(x.x, x.y)), (double)M);
            } else if (a.steer_type == 2) {   // 1 / conj(x) / M
                x = cdiv_real(cdiv(make_double2(1.0, 0.0), make_double2(x.x, -x.y)), (double)M);
            } else {   // x / sum |x|^2  |  x / sqrt(sum |x|^2 M)
                x = cdiv_real(x, nrm);
            }
            // * sqrt(normfactor), then the conjugate
            w[tid] = make_double2(__dmul_rn(x.x, a.sqrt_norm), -__dmul_rn(x.y, a.sqrt_norm));
        }
        __syncthreads();

        // 3. D1 = (C^T - diag C) w / hmax: D1_a = sum_{m != a} C[m][a] w_m, the mics m split over ngrp threads per a
        {
            const int r = tid % Mp, grp = tid / Mp;
            double sr[2] = {0.0, 0.0}, si[2] = {0.0, 0.0};
            if (r < M && grp < ngrp) {
                const int per = (M + ngrp - 1) / ngrp, m1 = min(M, (grp + 1) * per);
                for (int m = grp * per; m < m1; m += 2) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        if (m + u >= m1 || m + u == r) continue;
                        const double2 c = C[(m + u) * M + r], v = w[m + u];
                        sr[u] = fma(c.x, v.x, fma(-c.y, v.y, sr[u]));
                        si[u] = fma(c.x, v.y, fma(c.y, v.x, si[u]));
                    }
                }
                part[grp * Mp + r] = make_double2(sr[0] + sr[1], si[0] + si[1]);
            }
        }
        __syncthreads();

        // the first steering values of step 6 go out now: they land while warp 0 iterates
        double2 pre[AHEAD];
        auto fetch = [&](int64_t g, int m0) {
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
                pre[u] = __ldg(sv + (int64_t)min(m0 + u, M - 1) * G + min(g, G - 1));
        };
        fetch((int64_t)rank * kCscClThreads + tid, 0);

        // 4. 20 fixed-point steps: hh = (D1 + |hh|^2 w) / sqrt(1 + sum_m |w_m|^2 |hh_m|^2), from hh = w, in warp 0
        if (warp == 0) {
            double2 q[kCscClMics / 32 + 1], v[kCscClMics / 32 + 1], d[kCscClMics / 32 + 1];
            double wv[kCscClMics / 32 + 1];
            const double inv = cdiv_real(make_double2(1.0, 0.0), hmax).x;
#pragma unroll
            for (int u = 0; u <= kCscClMics / 32; ++u) {
                const int m = lane + 32 * u;
                v[u] = d[u] = make_double2(0.0, 0.0);
                if (m < M) {
                    v[u] = w[m];
                    double2 t = part[m];
                    for (int e = 1; e < ngrp; ++e) t = make_double2(t.x + part[e * Mp + m].x, t.y + part[e * Mp + m].y);
                    d[u] = make_double2(t.x * inv, t.y * inv);
                }
                q[u] = v[u];
                wv[u] = v[u].x * v[u].x + v[u].y * v[u].y;
            }
            for (int it = 0; it < 20; ++it) {
                double sum = 0.0, H[kCscClMics / 32 + 1];
#pragma unroll
                for (int u = 0; u <= kCscClMics / 32; ++u) {
                    H[u] = fma(q[u].x, q[u].x, q[u].y * q[u].y);
                    sum = fma(wv[u], H[u], sum);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                const double scl = rsqrt(1.0 + sum);
                bool same = true;
#pragma unroll
                for (int u = 0; u <= kCscClMics / 32; ++u) {
                    const double2 n = make_double2(fma(H[u], v[u].x, d[u].x) * scl, fma(H[u], v[u].y, d[u].y) * scl);
                    same = same && n.x == q[u].x && n.y == q[u].y;
                    q[u] = n;
                }
                if (__all_sync(0xffffffffu, same)) break;
            }
#pragma unroll
            for (int u = 0; u <= kCscClMics / 32; ++u)
                if (lane + 32 * u < M) hh[lane + 32 * u] = q[u];
        }
        __syncthreads();

        // 5. C[r][c] -= damp (hmax (hh_c conj(hh_r)))
        for (int r = warp; r < M; r += kCscClThreads / 32) {
            const double2 y = hh[r];
            for (int c = lane; c < M; c += 32) {
                const double2 u = hh[c];
                const double pr = __dsub_rn(__dmul_rn(u.x, y.x), __dmul_rn(u.y, -y.y));
                const double pi = __dadd_rn(__dmul_rn(u.x, -y.y), __dmul_rn(u.y, y.x));
                double2 e = C[r * M + c];
                e.x = __dsub_rn(e.x, __dmul_rn(a.damp, __dmul_rn(hmax, pr)));
                e.y = __dsub_rn(e.y, __dmul_rn(a.damp, __dmul_rn(hmax, pi)));
                C[r * M + c] = e;
            }
        }
        // 6. h -= damp times the map of the component (hmax, conj(hh)): t_m = hh_m v_m
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int64_t g = (int64_t)p * nctas * kCscClThreads + rank * kCscClThreads + tid;
            if (g >= G) break;
            double fr[4] = {0, 0, 0, 0}, fi[4] = {0, 0, 0, 0}, dg[4] = {0, 0, 0, 0};
            for (int m = 0; m < M; m += AHEAD) {
                if (p || m) fetch(g, m);
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    if (m + u >= M) break;
                    const double2 s = pre[u], q = hh[m + u];
                    const double tr = q.x * s.x - q.y * s.y, ti = q.x * s.y + q.y * s.x;
                    fr[u & 3] += tr;
                    fi[u & 3] += ti;
                    if (r_diag) dg[u & 3] += tr * tr + ti * ti;
                }
            }
            const double sr = (fr[0] + fr[1]) + (fr[2] + fr[3]), si = (fi[0] + fi[1]) + (fi[2] + fi[3]);
            double full = sr * sr + si * si;
            if (r_diag) full -= (dg[0] + dg[1]) + (dg[2] + dg[3]);
            h[p] = __dsub_rn(h[p], __dmul_rn(a.damp, full * hmax * norm));
        }
    }
    __syncthreads();
    if (rank == 0)
        for (int e = tid; e < M * M; e += kCscClThreads) Cg[e] = C[e];   // the cleaned matrix
}

static bool csc_cluster_fits(int M, int64_t G, int stopn)
{
    return M <= kCscClMics && G <= (int64_t)kCscPoints * kCscMaxCtas * kCscClThreads && stopn >= 1 && stopn < kCscHistory;
}

// CTAs of a bin's cluster, for B bins of G points whose CTAs fit `per_sm` to an SM.  Eight finish a bin soonest, but only 15
// such clusters are resident per CTA of an SM, and the other bins wait for their turn: the size that makes the least of
// rounds times a round's length, a round being about as long as the map of three points per thread and its own points.
// Measured (B200), microseconds of 20 iterations, always eight CTAs / this rule / two launches per iteration: 64 mics x 100
// points: 60 bins 784 / 423 / 844, 120 1495 / 443 / 861, 513 5894 / 917 / 1778; x 1681 points: 60 1093 / 939 / 1611, 513 8279 /
// 6277 / 7896; 112 mics x 400 points: 60 2359 / 724 / 1569, 513 20,017 / 4680 / 6203; x 4000 points, 513: 43,201 / 34,568 /
// 29,652 (the launches skip bins that stop early, which evens that out); 16 mics x 1681 points, 300: 2991 / 1537 / 2409.
static int csc_ctas(int64_t G, int B, int per_sm)
{
    int best = kCscMaxCtas;
    int64_t cost = INT64_MAX;
    for (int c = kCscMaxCtas; c >= 1 && G <= (int64_t)kCscPoints * c * kCscClThreads; c >>= 1) {
        const int64_t resident = per_sm * (c == 8 ? 15 : c == 4 ? 33 : kNumSMs / c);
        const int64_t points = (G + c * kCscClThreads - 1) / (c * kCscClThreads);
        const int64_t t = (B + resident - 1) / resident * (3 + points);
        if (t < cost) {
            cost = t;
            best = c;
        }
    }
    return best;
}

struct CscWorkspace {
    size_t h, h1, powers, lam, vec, active, steer, total;
};

static CscWorkspace csc_layout(int M, int64_t G, int B, int J)
{
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    CscWorkspace w;
    size_t off = 0;
    w.h = off;
    off += up((size_t)B * G * sizeof(double));
    w.h1 = off;
    off += up((size_t)B * G * sizeof(double));
    w.powers = off;
    off += up((size_t)B * J * sizeof(double));
    w.lam = off;
    off += up((size_t)B * sizeof(double));
    w.vec = off;
    off += up((size_t)B * M * sizeof(double2));
    w.active = off;
    off += up((size_t)B * sizeof(int));
    w.steer = off;
    off += up((size_t)B * G * M * sizeof(double2));
    w.total = off;
    return w;
}

}  // namespace acb

using namespace acb;

extern "C" {

size_t acb_cleansc_workspace_bytes(int num_mics, int64_t num_grid, int num_bins, int n_iter)
{
    if (num_mics < 2 || num_grid <= 0 || num_bins <= 0 || n_iter < 0) return 0;
    const int J = n_iter > 0 ? n_iter : 2 * num_mics;
    return csc_layout(num_mics, num_grid, num_bins, J).total;
}

int acb_cleansc_f64(const acb_map_params *p, void *csm, const double *wavenumber, const double *mpos,
                    const double *gpos, const double *r0, const double *rm, int n_iter, double damp, int stopn,
                    float *result, void *workspace, size_t workspace_bytes, void *stream)
{
    if (!p || !csm || !wavenumber || !result || !workspace) return ACB_ERR_ARG;
    if (!rm && (!mpos || !gpos)) return ACB_ERR_ARG;
    if (rm && !r0) return ACB_ERR_ARG;
    if (p->steer_type < 1 || p->steer_type > 4) return ACB_ERR_ARG;
    const int M = p->num_mics, B = p->num_bins;
    const int64_t G = p->num_grid;
    if (M < 2 || M > 2048 || G <= 0 || B <= 0 || B > 65535 || n_iter < 0) return ACB_ERR_SHAPE;
    if (p->glibc_faithful && (!p->sincos_table || p->sincos_table_slots <= 0 ||
                              (p->sincos_table_slots & (p->sincos_table_slots - 1))))
        return ACB_ERR_ARG;
    const int J = n_iter > 0 ? n_iter : 2 * M;
    const CscWorkspace lay = csc_layout(M, G, B, J);
    if (workspace_bytes < lay.total) return ACB_ERR_WORKSPACE;
    cudaStream_t s = as_stream(stream);
    char *ws = static_cast<char *>(workspace);

    acb_map_params q = *p;
    q.clip_negative = 0;   // CLEAN-SC works on the unclipped map
    CscArgs a;
    a.M = M;
    a.G = G;
    a.J = J;
    a.stopn = stopn;
    a.damp = damp;
    a.sqrt_norm = sqrt(p->norm);
    a.steer_type = p->steer_type;
    a.k = wavenumber;
    a.r0 = rm ? r0 : nullptr;
    a.rm = rm;
    a.mpos = mpos;
    a.gpos = gpos;
    a.ref_mode = p->ref_mode;
    a.ref0 = p->ref_point[0];
    a.ref1 = p->ref_point[1];
    a.ref2 = p->ref_point[2];
    a.ref_dist = p->ref_distance;
    a.faithful = p->glibc_faithful;
    a.table = p->sincos_table;
    a.mask = p->glibc_faithful ? (uint64_t)p->sincos_table_slots - 1 : 0;
    a.csm = static_cast<double2 *>(csm);
    a.h = reinterpret_cast<double *>(ws + lay.h);
    a.h1 = reinterpret_cast<const double *>(ws + lay.h1);
    a.powers = reinterpret_cast<double *>(ws + lay.powers);
    a.result = result;
    a.active = reinterpret_cast<int *>(ws + lay.active);
    a.lam = reinterpret_cast<double *>(ws + lay.lam);
    a.vec = reinterpret_cast<double2 *>(ws + lay.vec);
    a.given = nullptr;

    const int64_t n_init = (int64_t)B * G > B ? (int64_t)B * G : B;
    cleansc_init_kernel<<<(unsigned)((n_init + 255) / 256), 256, 0, s>>>(a.active, result, (int64_t)B * G, B);
    int st = check_launch();
    if (st) return st;
    st = map_plain_launch(&q, B, csm, wavenumber, mpos, gpos, r0, rm, a.h, s);
    if (st) return st;
    double2 *steer = reinterpret_cast<double2 *>(ws + lay.steer);
    if (csc_cluster_fits(M, G, stopn)) {
        const size_t tile = (size_t)M * 33 * sizeof(double2), smem = csc_cluster_smem(M);
        const int per_sm = 2 * (smem + 2048) <= 228 * 1024 ? 2 : 1, C = csc_ctas(G, B, per_sm);
        // few bins: 16 steering values in flight per thread and all the registers that takes; more bins than one CTA per
        // SM holds: 8, and 128 registers for two (60 bins of 64 mics in clusters of eight: 2.14 against 3.43 ms)
        const bool few = B * C <= 120, small = G <= C * kCscClThreads;
        auto kern = few && C == 8 ? (small ? cleansc_cluster_kernel<1, 16, 1, 8> : cleansc_cluster_kernel<kCscPoints, 16, 1, 8>)
                    : few         ? (small ? cleansc_cluster_kernel<1, 16, 1, 0> : cleansc_cluster_kernel<kCscPoints, 16, 1, 0>)
                                  : (small ? cleansc_cluster_kernel<1, 8, 2, 0> : cleansc_cluster_kernel<kCscPoints, 8, 2, 0>);
        st = allow_smem(cleansc_steer_kernel<true>, tile, (size_t)kCscClMics * 33 * sizeof(double2));
        if (!st) st = allow_smem(kern, smem, csc_cluster_smem(kCscClMics));
        if (st) return st;
        cleansc_steer_kernel<true><<<dim3((unsigned)((G + 31) / 32), B), 256, tile, s>>>(a, steer);
        st = check_launch();
        if (st) return st;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(B * C));
        cfg.blockDim = dim3(kCscClThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)C;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaLaunchKernelEx(&cfg, kern, a, static_cast<const double2 *>(steer), p->r_diag, p->norm) != cudaSuccess)
            return ACB_ERR_CUDA;
        return check_launch();
    }
    cleansc_steer_kernel<false><<<dim3((unsigned)((G + 7) / 8), B), 256, 0, s>>>(a, steer);
    st = check_launch();
    if (st) return st;
    const size_t smem = (size_t)M * (3 * sizeof(double2) + sizeof(double));
    st = allow_smem(cleansc_step_kernel, smem, kCscStepSmem);
    if (st) return st;
    for (int j = 0; j < J; ++j) {
        cleansc_step_kernel<<<B, kCscThreads, smem, s>>>(a, j);
        st = check_launch();
        if (st) return st;
        if (j + 1 < J) {
            st = map_eig_custom_launch(&q, B, 1, a.lam, a.vec, steer, reinterpret_cast<double *>(ws + lay.h1),
                                       a.active, s);
            if (st) return st;
        }
    }
    return ACB_OK;
}

int acb_cleansc_custom_f64(const acb_map_params *p, void *csm, const void *steer, int n_iter, double damp, int stopn,
                           float *result, void *workspace, size_t workspace_bytes, void *stream)
{
    if (!p || !csm || !steer || !result || !workspace) return ACB_ERR_ARG;
    const int M = p->num_mics, B = p->num_bins;
    const int64_t G = p->num_grid;
    if (M < 2 || M > 2048 || G <= 0 || B <= 0 || B > 65535 || n_iter < 0) return ACB_ERR_SHAPE;
    const int J = n_iter > 0 ? n_iter : 2 * M;
    const CscWorkspace lay = csc_layout(M, G, B, J);
    if (workspace_bytes < lay.steer) return ACB_ERR_WORKSPACE;   // the steering region is not needed
    cudaStream_t s = as_stream(stream);
    char *ws = static_cast<char *>(workspace);

    acb_map_params q = *p;
    q.clip_negative = 0;   // CLEAN-SC works on the unclipped map
    q.glibc_faithful = 0;  // no phase synthesis: the vectors are given
    CscArgs a = {};
    a.M = M;
    a.G = G;
    a.J = J;
    a.stopn = stopn;
    a.damp = damp;
    a.sqrt_norm = sqrt(p->norm);
    a.steer_type = 0;
    a.csm = static_cast<double2 *>(csm);
    a.h = reinterpret_cast<double *>(ws + lay.h);
    a.h1 = reinterpret_cast<const double *>(ws + lay.h1);
    a.powers = reinterpret_cast<double *>(ws + lay.powers);
    a.result = result;
    a.active = reinterpret_cast<int *>(ws + lay.active);
    a.lam = reinterpret_cast<double *>(ws + lay.lam);
    a.vec = reinterpret_cast<double2 *>(ws + lay.vec);
    a.given = static_cast<const double2 *>(steer);

    const int64_t n_init = (int64_t)B * G > B ? (int64_t)B * G : B;
    cleansc_init_kernel<<<(unsigned)((n_init + 255) / 256), 256, 0, s>>>(a.active, result, (int64_t)B * G, B);
    int st = check_launch();
    if (st) return st;
    st = acb_map_custom_f64(&q, csm, steer, a.h, nullptr, stream);
    if (st) return st;
    const size_t smem = (size_t)M * (3 * sizeof(double2) + sizeof(double));
    st = allow_smem(cleansc_step_kernel, smem, kCscStepSmem);
    if (st) return st;
    for (int j = 0; j < J; ++j) {
        cleansc_step_kernel<<<B, kCscThreads, smem, s>>>(a, j);
        st = check_launch();
        if (st) return st;
        if (j + 1 < J) {
            st = map_eig_custom_launch(&q, B, 1, a.lam, a.vec, steer, reinterpret_cast<double *>(ws + lay.h1),
                                       a.active, s);
            if (st) return st;
        }
    }
    return ACB_OK;
}

}  // extern "C"
