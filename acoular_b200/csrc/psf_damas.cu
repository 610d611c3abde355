// Point-spread functions (calcPointSpreadFunction, acoular/fastFuncs.py:563-801, as
// PointSpreadFunction._psf_call uses it, acoular/fbeamform.py:1093-1125) and the DAMAS Gauss-Seidel
// solver (damasSolverGaussSeidel, acoular/fastFuncs.py:804-855, as BeamformerDamas._calc uses it,
// acoular/fbeamform.py:1167-1208), plain FP64.
//
// PSF: for grid point g and source (grid point) s,
//     P = |sum_m e^{-i fl32(k (rm[g,m] - rm[s,m]))} w_m|^2 * n^2,
// the four steering types weighting w_m and n as the reference does; the phase is rounded to float32
// and its cos/sin are the C library's float32 ones (the exception table of the plain map).
// CTA = 32 grid points x 32 sources; their distance rows and reciprocals are staged in shared memory.
//
// DAMAS: per bin, n_iter sweeps over g = 0 .. G-1 in order, each x[g] = max(0, (1 - relax) x[g] +
// relax (y[g] - sum_{h != g} A[g][h] x[h])) with the latest x.  The sweep is sequential by
// definition; a cluster of 1-8 CTAs per bin keeps x in every CTA's shared memory, splits the bulk of
// each row's dot product over its CTAs' column slices one block of rows ahead, and one warp solves
// each block of 32 rows in order (damas_kernel).
#include <cuda_runtime.h>
#include <stdint.h>

#include <cooperative_groups.h>

#include "common.cuh"
#include "tc_common.cuh"

namespace cg = cooperative_groups;

namespace acb {

constexpr int kPsfTile = 32;      // grid points per CTA, and its most sources
constexpr int kPsfWarps = 8;
constexpr int kPsfMics = 32;      // mics per shared-memory chunk: 33 KB, four CTAs per SM (64: 0.67 ms below)

// Distances and their reciprocals of a tile's 32 grid points, mic-major, and of its 32 sources, source-major.
constexpr int kPsfG = kPsfMics * (kPsfTile + 1), kPsfS = kPsfTile * (kPsfMics + 1);
constexpr int kPsfSmem = 2 * (kPsfG + kPsfS) * (int)sizeof(double);

// CTA = 32 grid points (lanes) x 8 PER sources (PER per warp, whose phases a lane evaluates together): 32 where there are
// CTAs enough, fewer for a few sources, whose chains of phases are what takes the time then (psf_per).
// MIRROR (as many sources as points, PER = 4): the phase of (g, s) is minus that of (s, g), so that where the sources are
// the grid itself (checked on the tile's own indices), a tile right of the diagonal also gives its mirror image, whose
// CTA then has nothing to do.  The mirrored sums differ in their weights only: w for P(g; s), wm for P(s; g), the same
// for 'true level' and 'true location'.
// Bound: issue slots (62 %; 108 instructions per phase, its sums included).  Measured (B200): 1681 x 1681 x 64 mics
// 1.03 -> 0.48 ms.
template <int ST, int PER, bool MIRROR>
__global__ void __launch_bounds__(256, 4) psf_kernel(int M, int64_t G, int S, const int64_t *__restrict__ src,
                                                     const double *__restrict__ r0, const double *__restrict__ rm,
                                                     double k, const uint64_t *__restrict__ table, uint64_t mask,
                                                     int faithful, int round_f32, double *__restrict__ out)
{
    extern __shared__ double psf_sm[];
    double *rg_s = psf_sm, *ig_s = rg_s + kPsfG;        // [mic][point, 33]
    double *rs_s = ig_s + kPsfG, *is_s = rs_s + kPsfS;   // [source][mic, 33]
    __shared__ int64_t src_s[kPsfTile];
    __shared__ double help_s[2 * kPsfTile];              // sums of 1 / r^2: points, sources
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NS = kPsfWarps * PER;                  // the tile's sources
    static_assert(!MIRROR || NS == kPsfTile, "a mirrored tile is square");
    const int64_t gb = (int64_t)blockIdx.x * kPsfTile;
    const int sb = blockIdx.y * NS;
    const int64_t g = gb + lane;
    bool own = MIRROR;   // this tile's points and sources are the grid's in order
    if (threadIdx.x < NS) {
        const int i = sb + threadIdx.x;
        const int64_t s = i < S ? src[i] : 0;
        src_s[threadIdx.x] = s;
        if (MIRROR) own = i >= S || s == i;
    } else if (MIRROR && threadIdx.x < 2 * kPsfTile) {
        const int64_t i = gb + threadIdx.x - kPsfTile;
        own = i >= S || src[i] == i;
    }
    const bool sym = __syncthreads_and(own) && gb != sb;
    if (sym && gb > sb) return;   // the tile on the other side of the diagonal writes this one
    const SincosTable sct = sincos_table(table, mask, faithful != 0);
    double re[PER], im[PER], rem[PER], imm[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) re[j] = im[j] = rem[j] = imm[j] = 0.0;
    if (threadIdx.x < 2 * kPsfTile) help_s[threadIdx.x] = 0.0;
    for (int m0 = 0; m0 < M; m0 += kPsfMics) {
        const int n = min(kPsfMics, M - m0);
        __syncthreads();
        for (int i = threadIdx.x; i < kPsfTile * kPsfMics; i += blockDim.x) {
            const int p = i / kPsfMics, m = i % kPsfMics;
            if (m >= n) continue;
            const double a = gb + p < G ? rm[(gb + p) * M + m0 + m] : 1.0;
            rg_s[m * (kPsfTile + 1) + p] = a;
            if (ST >= 3 || MIRROR) ig_s[m * (kPsfTile + 1) + p] = 1.0 / a;
            if (p >= NS) continue;
            int64_t s = src_s[p];
            s = s >= 0 && s < G ? s : 0;   // an index outside the grid yields NaN, never a stray read
            const double b = rm[s * M + m0 + m];
            rs_s[p * (kPsfMics + 1) + m] = b;
            is_s[p * (kPsfMics + 1) + m] = 1.0 / b;
        }
        __syncthreads();
        if (ST >= 3 && threadIdx.x < (MIRROR ? 2 * kPsfTile : kPsfTile)) {
            double h = help_s[threadIdx.x];
            for (int m = 0; m < n; ++m) {
                const double q = threadIdx.x < kPsfTile ? ig_s[m * (kPsfTile + 1) + threadIdx.x]
                                                        : is_s[(threadIdx.x - kPsfTile) * (kPsfMics + 1) + m];
                h = fma(q, q, h);
            }
            help_s[threadIdx.x] = h;
        }
        if (sb + warp * PER >= S) continue;   // no such sources
        const double *rsw = rs_s + warp * PER * (kPsfMics + 1), *isw = is_s + warp * PER * (kPsfMics + 1);
        for (int m = 0; m < n; ++m) {
            const double rg = rg_s[m * (kPsfTile + 1) + lane];
            const double ig = ST >= 3 || MIRROR ? ig_s[m * (kPsfTile + 1) + lane] : 0.0;
            SincosPending<PER> pend;
#pragma unroll
            for (int j = 0; j < PER; ++j)
                pend.x[j] = __double2float_rn(__dmul_rn(k, __dsub_rn(rg, rsw[j * (kPsfMics + 1) + m])));
            sincos_begin(pend, sct);
            sincos_finish(pend, sct);
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const double c = (double)pend.c[j], sn = -(double)pend.s[j];
                // (cos - i sin) / rs  [* rg (inverse) | / rg (true level, true location)]; the divisions as
                // products with reciprocals (within an ulp of the quotients); the mirror image's sine is negated
                const double is = isw[j * (kPsfMics + 1) + m];
                const double w = ST == 1 ? is : ST == 2 ? is * rg : is * ig;
                re[j] = fma(c, w, re[j]);
                im[j] = fma(sn, w, im[j]);
                if (MIRROR && ST < 3 && sym) {
                    const double wm = ST == 1 ? ig : ig * rsw[j * (kPsfMics + 1) + m];
                    rem[j] = fma(c, wm, rem[j]);
                    imm[j] = fma(sn, wm, imm[j]);
                }
            }
        }
    }
    __syncthreads();
    double *tile = psf_sm;   // [point][source, 33]
    const double Md = (double)M;
    // P(a; b) from the sum's squared magnitude, the reference distances and a's sum of 1 / r^2
    auto value = [&](double a2, double ra, double rb, double help) {
        double nf, res;
        if (ST == 1) {
            nf = rb / Md;
            res = a2 * (nf * nf);
        } else if (ST == 2) {
            nf = rb / ra / Md;
            res = a2 * (nf * nf);
        } else if (ST == 3) {
            nf = rb / ra / help;
            res = a2 * (nf * nf);
        } else {
            res = a2 * (rb * rb) / Md / help;
        }
        return round_f32 ? (double)__double2float_rn(res) : res;
    };
    const double ra = g < G ? r0[g] : 1.0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int q = warp * PER + j;
        const int64_t s = src_s[q];
        const bool ok = s >= 0 && s < G;
        const double rb = r0[ok ? s : 0];
        const double a2 = re[j] * re[j] + im[j] * im[j];
        tile[lane * (kPsfTile + 1) + q] =
            ok ? value(a2, ra, rb, help_s[lane]) : __longlong_as_double(0x7ff8000000000000ll);
        if (MIRROR && sym && sb + q < S && g < G) {
            const double m2 = ST < 3 ? rem[j] * rem[j] + imm[j] * imm[j] : a2;
            out[(int64_t)(sb + q) * S + g] = value(m2, rb, ra, help_s[kPsfTile + q]);
        }
    }
    __syncthreads();
    for (int p = warp; p < kPsfTile; p += kPsfWarps)
        if (gb + p < G && lane < NS && sb + lane < S) out[(gb + p) * S + sb + lane] = tile[p * (kPsfTile + 1) + lane];
}

// Sources per warp: the most whose tiles are filled (at most a quarter of padding) and are CTAs enough.  Measured (B200),
// microseconds at 4 / 2 / 1 per warp, 'true level': 64 mics x 1681 points: 1 source 87 / 55 / 42, 33 103 / 63 / 51, 200 (371
// CTAs / 689 / 1325) 162 / 159 / 135, 400 (689 / 1325 / 2650) 294 / 246 / 242, 1000 (1696 / 3339) 537 / 527; x 10,201 points:
// 64 (638 / 1276 / 2552) 281 / 246 / 247, 200 (2233 / 4147) 662 / 659 / 699, 1000 2951 / 3067 / 3356; 32 mics x 40,000 points:
// 24 (1250 / 2500 / 3750) 212 / 210 / 193, 64 (2500 / 5000) 405 / 415 / 468.  The mirrored form: 1681 points 472 where they take
// 857 / 926; 441 points (105 CTAs with anything to do) 124 / 86 / 103.  Before (8 sources per CTA, one per warp, whatever
// their number) 1681 points: 1 source 96, 33 124, 200 264, 1000 1032, all 1697.
constexpr int64_t kPsfManyCtas4 = 15 * kNumSMs, kPsfManyCtas2 = 17 * kNumSMs / 2;

static int psf_per(int64_t G, int S)
{
    const int64_t tiles = (G + kPsfTile - 1) / kPsfTile;
    for (int per = 4; per > 1; per >>= 1) {
        const int64_t ns = kPsfWarps * per, cols = (S + ns - 1) / ns;
        if (4 * cols * ns <= 5 * (int64_t)S && tiles * cols >= (per == 4 ? kPsfManyCtas4 : kPsfManyCtas2)) return per;
    }
    return 1;
}

constexpr int kDamasThreads = 512;
constexpr int kDamasWarps = kDamasThreads / 32;
constexpr int kDamasRows = 32;        // rows solved per step (one per lane of the solving warp)
constexpr int kDamasMaxCta = 8;       // CTAs per bin (a portable cluster)
constexpr int kDamasPad = kDamasRows + 1;

// Shared memory of one CTA, in doubles: x[G] | partials[2][8][32] | diagonal tile^T[2][32][33] |
// previous-block tile^T[2][32][33] | y[2][32]
__host__ __device__ inline int64_t damas_smem_doubles(int64_t G)
{
    return G + 2 * kDamasMaxCta * kDamasRows + 4 * kDamasRows * kDamasPad + 2 * kDamasRows;
}

// Blocked, pipelined Gauss-Seidel.  Rows are taken in blocks of 32; step t solves block k = t mod nblk.
// Row i of block k needs sum_{h != i} A[i][h] x[h] with the latest x.  It is assembled from
//   (a) the columns outside blocks k and k-1 (final values of this sweep left of k-1, values of the
//       previous sweep right of k): computed one step AHEAD, while block k-1 is being solved, by the
//       warps of the cluster (in the first CTA only those off the solver's SM sub-partition, which
//       would otherwise take its issue slots), each CTA over its own column slice, and summed
//       through distributed shared memory into the first CTA;
//   (b) the columns of block k-1, whose new values are known at the start of step t (tile L);
//   (c) the other columns of block k (tile D), old values for the rows after each row, new ones as
//       they are solved.
// The solving warp (warp 0 of the first CTA) takes (b), (c) and the rows of block k in order, lane i
// owning row i: row j's new value is broadcast with a shuffle and every later lane subtracts its
// contribution.  One cluster barrier per step publishes block k's values to every CTA and the
// partial sums of block k+1 to the solver.  An L2 prefetch of block k+2's rows runs a step ahead
// of their loads.  Sweeps continue across the wrap-around (block 0 follows block nblk-1).
__global__ void __launch_bounds__(kDamasThreads) damas_kernel(const double *__restrict__ A, int64_t G,
                                                             const double *__restrict__ y, double *__restrict__ x,
                                                             int n_iter, double relax)
{
    extern __shared__ double sm[];
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks();
    const int crank = (int)cluster.block_rank();
    const int64_t bin = blockIdx.x / C;
    double *xs = sm;
    double *red = xs + G;
    double *dT = red + 2 * kDamasMaxCta * kDamasRows;
    double *lT = dT + 2 * kDamasRows * kDamasPad;
    double *ys = lT + 2 * kDamasRows * kDamasPad;
    const double *Ab = A + bin * G * G;
    const double *yg = y + bin * G;
    double *xg = x + bin * G;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nblk = (int)((G + kDamasRows - 1) / kDamasRows);
    const int64_t W = ((G + C - 1) / C + 31) / 32 * 32;
    const int64_t c0 = min((int64_t)crank * W, G), c1 = min(c0 + W, G);
    double *red0 = cluster.map_shared_rank(red, 0);
    double *dT0 = cluster.map_shared_rank(dT, 0);
    double *lT0 = cluster.map_shared_rank(lT, 0);

    for (int64_t i = threadIdx.x; i < G; i += kDamasThreads) xs[i] = xg[i];
    // tiles start zeroed: entries outside a short last block are then finite (0 or an earlier value)
    for (int i = threadIdx.x; i < 4 * kDamasRows * kDamasPad; i += kDamasThreads) dT[i] = 0.0;
    __syncthreads();

    // Partial sums of block k (columns of blocks k and prev excluded) into buffer buf of the first
    // CTA.  The same pass routes the columns of block k (tile D) and of block prev (tile L) to the
    // first CTA's tiles instead of summing them; a warp takes up to three rows at once so that all
    // of its loads of a step are in flight together.
    auto prepare = [&](int k, int prev, int buf, bool spare) {
        if (spare && (warp & 3) == 0) return;
        const int w = spare ? warp - (warp >> 2) - 1 : warp;
        const int nw = spare ? kDamasWarps - kDamasWarps / 4 : kDamasWarps;
        const int64_t g0 = (int64_t)k * kDamasRows, p0 = (int64_t)prev * kDamasRows;
        const int nb = (int)min((int64_t)kDamasRows, G - g0);
        const int np = prev == k ? 0 : (int)min((int64_t)kDamasRows, G - p0);
        if (crank == 0 && w == 0) ys[buf * kDamasRows + lane] = lane < nb ? yg[g0 + lane] : 0.0;
        double *dt0 = dT0 + buf * kDamasRows * kDamasPad;
        double *lt0 = lT0 + buf * kDamasRows * kDamasPad;
        for (int rb = w; rb < nb; rb += 3 * nw) {
            const int r1 = rb + nw, r2 = rb + 2 * nw;
            const bool v1ok = r1 < nb, v2ok = r2 < nb;
            const double *row0 = Ab + (g0 + rb) * G;
            const double *row1 = Ab + (g0 + (v1ok ? r1 : rb)) * G;
            const double *row2 = Ab + (g0 + (v2ok ? r2 : rb)) * G;
            double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0;
            // chunks of 8 columns per lane: all loads of a chunk are issued before any use
            for (int64_t base = c0 + lane; base < c1; base += 8 * 32) {
                double v0[8], v1[8], v2[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int64_t h = base + u * 32;
                    const bool in = h < c1;
                    v0[u] = in ? __ldg(row0 + h) : 0.0;
                    v1[u] = (in && v1ok) ? __ldg(row1 + h) : 0.0;
                    v2[u] = (in && v2ok) ? __ldg(row2 + h) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int64_t h = base + u * 32;
                    if (h >= c1) break;
                    if (h >= g0 && h < g0 + nb) {
                        double *t = dt0 + (h - g0) * kDamasPad;
                        t[rb] = v0[u];
                        if (v1ok) t[r1] = v1[u];
                        if (v2ok) t[r2] = v2[u];
                    } else if (h >= p0 && h < p0 + np) {
                        double *t = lt0 + (h - p0) * kDamasPad;
                        t[rb] = v0[u];
                        if (v1ok) t[r1] = v1[u];
                        if (v2ok) t[r2] = v2[u];
                    } else {
                        const double xh = xs[h];
                        acc0 = fma(v0[u], xh, acc0);
                        acc1 = fma(v1[u], xh, acc1);
                        acc2 = fma(v2[u], xh, acc2);
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                acc0 += __shfl_xor_sync(0xffffffffu, acc0, o);
                acc1 += __shfl_xor_sync(0xffffffffu, acc1, o);
                acc2 += __shfl_xor_sync(0xffffffffu, acc2, o);
            }
            if (lane == 0) {
                double *rp = red0 + buf * kDamasMaxCta * kDamasRows + crank * kDamasRows;
                rp[rb] = acc0;
                if (v1ok) rp[r1] = acc1;
                if (v2ok) rp[r2] = acc2;
            }
        }
    };

    // Solve the rows of block k in order (warp 0 of the first CTA) and publish them to every CTA.
    // Lane i keeps u_i = c_i - relax (s_i + sum_{l > i} A[i][l] x_l), c_i = (1 - relax) x_i + relax y_i
    // and s_i the sum over the columns outside the block; row j's new value is max(0, u_j), and
    // every lane then subtracts relax A[i][j] times it.  The chain per row is one FMA, one max and
    // one shuffle; the sums feeding it use independent accumulators.
    auto solve = [&](int k, int prev, int buf) {
        const int64_t g0 = (int64_t)k * kDamasRows, p0 = (int64_t)prev * kDamasRows;
        const int nb = (int)min((int64_t)kDamasRows, G - g0);
        const int np = prev == k ? 0 : (int)min((int64_t)kDamasRows, G - p0);
        const int i = lane;
        const double *dt = dT + buf * kDamasRows * kDamasPad;
        const double *lt = lT + buf * kDamasRows * kDamasPad;
        const double *rp = red + buf * kDamasMaxCta * kDamasRows + i;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int c = 0; c < kDamasMaxCta; ++c)
            if (c < C) acc[c & 3] += rp[c * kDamasRows];
#pragma unroll
        for (int j = 0; j < kDamasRows; ++j)
            if (j < np) acc[j & 3] = fma(lt[j * kDamasPad + i], xs[p0 + j], acc[j & 3]);
        double b[kDamasRows];
#pragma unroll
        for (int j = 0; j < kDamasRows; ++j) b[j] = dt[j * kDamasPad + i];
        const double xold = i < nb ? xs[g0 + i] : 0.0;
#pragma unroll
        for (int j = 0; j < kDamasRows; ++j) {
            const double xj = __shfl_sync(0xffffffffu, xold, j);
            if (j > i) acc[j & 3] = fma(b[j], xj, acc[j & 3]);
        }
        const double s = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        double u = (1.0 - relax) * xold + relax * (ys[buf * kDamasRows + i] - s);
#pragma unroll
        for (int j = 0; j < kDamasRows; ++j) b[j] = j < i ? relax * b[j] : 0.0;
        double xv = 0.0;
#pragma unroll
        for (int j = 0; j < kDamasRows; ++j) {
            if (j >= nb) break;
            const double xn = __shfl_sync(0xffffffffu, fmax(u, 0.0), j);
            u = fma(-b[j], xn, u);
            xv = i == j ? xn : xv;
        }
        if (i < nb)
            for (int r = 0; r < C; ++r) cluster.map_shared_rank(xs, r)[g0 + i] = xv;
    };

    // L2 prefetch of this CTA's column slice of the rows of block k (read two steps later).
    auto prefetch = [&](int k, bool spare) {
        if (spare && (warp & 3) == 0) return;
        const int w = spare ? warp - (warp >> 2) - 1 : warp;
        const int64_t g0 = (int64_t)k * kDamasRows;
        const int nb = (int)min((int64_t)kDamasRows, G - g0);
        const int64_t nlines = (c1 - c0 + 15) / 16;     // 128-byte lines of 16 doubles
        const int nthr = (spare ? kDamasWarps - kDamasWarps / 4 : kDamasWarps) * 32;
        for (int64_t e = w * 32 + lane; e < nb * nlines; e += nthr) {
            const double *ptr = Ab + (g0 + e / nlines) * G + c0 + (e % nlines) * 16;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr));
        }
    };

    prepare(0, nblk - 1, 0, false);
    if (nblk > 1) prefetch(1, false);
    cluster.sync();
    const int64_t steps = (int64_t)n_iter * nblk;
    for (int64_t t = 0; t < steps; ++t) {
        const int k = (int)(t % nblk);
        const int buf = (int)(t & 1);
        const int kn = k + 1 == nblk ? 0 : k + 1;
        if (crank == 0 && warp == 0) solve(k, k == 0 ? nblk - 1 : k - 1, buf);
        if (t + 1 < steps) prepare(kn, k, buf ^ 1, crank == 0);
        if (t + 2 < steps) prefetch(kn + 1 == nblk ? 0 : kn + 1, crank == 0);
        cluster.sync();
    }
    if (crank == 0)
        for (int64_t i = threadIdx.x; i < G; i += kDamasThreads) xg[i] = xs[i];
}

// ------------------------------------------------------------------------------------------------
// The same sweeps with the solver fed two blocks ahead, for six or more blocks of rows and clusters of four or eight
// CTAs.  CTA 0 solves: warp 0 takes the rows of one block after another (step t: block t mod nblk), lane i owning row i,
// and three warps bring it, per step, three 32 x 32 tiles of the block's columns: of its own rows and of the next two
// blocks' rows.  As each new value x_j is broadcast, every lane also adds its contribution to its rows of the next two
// blocks, off the serial path, so that a step starts as soon as the sums over all other columns are there.  Those
// come from the other CTAs: CTA r > 0 holds a slice of the columns, and for block t it needs the values of step t - 3
// and before (the solver adds those of t - 1 and t - 2 itself; right of the block and, within it, right of each row
// the previous sweep's values count), so it has two steps' time.  New values and sums travel as asynchronous stores
// counted on mbarriers (rings of four; a ring's slot is used again only after an exchange in the other direction that
// follows its last use): no cluster barrier in a step.
// Bound: the solver's step, 2550 cycles: 60 per row (one FMA, a compare and a shuffle are 50 of them) and the rest to take
// in the sums and publish the values.  Measured (B200): 5 bins x 1681 points x 100 sweeps 21.2 -> 7.0 ms; 2 bins x 4000
// points 71 -> 29 (the form above spends 7600 cycles a step, of them 2000 in its cluster barrier).  Four rows at a time,
// every lane solving their triangle for itself, was slower (80 a row: the extra FMAs' issue slots).
// ------------------------------------------------------------------------------------------------
constexpr int kGsTile = kDamasRows * kDamasPad, kGsStages = 3, kGsRing = 4;

__host__ __device__ inline int64_t gs_smem_bytes(int64_t G)
{
    const int64_t nblk = (G + kDamasRows - 1) / kDamasRows;
    return (nblk * kDamasRows + (int64_t)kGsStages * 3 * kGsTile + kGsRing * kDamasMaxCta * kDamasRows) * 8;
}

// max(0, u), and 0 for NaN as fmax gives it, on the integer pipe (sign bit or an exponent of ones with mantissa)
__device__ __forceinline__ double gs_clamp(double u)
{
    return (uint32_t)__double2hiint(u) > 0x7ff00000u ? 0.0 : u;
}

__global__ void __launch_bounds__(kDamasThreads) damas_ahead_kernel(const double *__restrict__ A, int64_t G,
                                                                   const double *__restrict__ y,
                                                                   double *__restrict__ x, int n_iter, double relax,
                                                                   uint64_t limit_ns)
{
    extern __shared__ double sm[];
    __shared__ uint64_t xbar[kGsRing], pbar[kGsRing], tbar[kGsStages];
    __shared__ int stop_s;
    volatile int *stop = &stop_s;
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int64_t bin = blockIdx.x / C;
    const int nblk = (int)((G + kDamasRows - 1) / kDamasRows);
    double *xs = sm;                                     // [nblk * 32], zeros past G
    double *tiles = xs + (int64_t)nblk * kDamasRows;     // [stage][own rows | next | the one after][column][33]
    double *part = tiles + kGsStages * 3 * kGsTile;      // [ring][CTA][32] (CTA 0's are used)
    const double *Ab = A + bin * G * G;
    const double *yg = y + bin * G;
    double *xg = x + bin * G;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t steps = (int64_t)n_iter * nblk;

    for (int64_t i = threadIdx.x; i < (int64_t)nblk * kDamasRows; i += kDamasThreads) xs[i] = i < G ? xg[i] : 0.0;
    if (threadIdx.x == 0) {
        for (int q = 0; q < kGsRing; ++q) {
            tc::mbar_init(&xbar[q], 1);
            tc::mbar_init(&pbar[q], 1);
        }
        for (int q = 0; q < kGsStages; ++q) tc::mbar_init(&tbar[q], 96);
        stop_s = 0;
        tc::fence_mbar_init();
        for (int q = 0; q < kGsRing; ++q)   // the first round of each ring
            if (rank == 0) tc::mbar_arrive_expect_tx(&pbar[q], (uint32_t)((C - 1) * kDamasRows * 8));
            else tc::mbar_arrive_expect_tx(&xbar[q], kDamasRows * 8);
    }
    cluster.sync();

    if (rank == 0 && warp == 0) {
        // ---------------- the solver
        double acc1 = 0.0, acc2 = 0.0;   // -relax times the new values' part of row `lane` of the next two blocks
        double yv = lane < G ? yg[lane] : 0.0;
        int k = 0;
        for (int64_t t = 0; t < steps; ++t) {
            const int64_t g0 = (int64_t)k * kDamasRows;
            const bool row = g0 + lane < G;
            const int st = (int)(t % kGsStages), slot = (int)(t % kGsRing);
            const double *D = tiles + st * 3 * kGsTile + lane, *N1 = D + kGsTile, *N2 = N1 + kGsTile;
            const double xold = xs[g0 + lane];
            const double c = fma(relax, yv, fma(1.0 - relax, xold, acc1));
            const bool here = tc::cluster_wait(&tbar[st], (uint32_t)(t / kGsStages) & 1, stop, limit_ns) &&
                              tc::cluster_wait(&pbar[slot], (uint32_t)(t / kGsRing) & 1, stop, limit_ns);
            if (!__all_sync(0xffffffffu, here)) {
                tc::cluster_stop(stop, C);
                break;
            }
            double sum[2] = {0.0, 0.0};
#pragma unroll
            for (int r = 1; r < kDamasMaxCta; ++r)
                if (r < C) sum[r & 1] += part[(slot * kDamasMaxCta + r) * kDamasRows + lane];
            if (lane == 0 && t + kGsRing < steps)
                tc::mbar_arrive_expect_tx(&pbar[slot], (uint32_t)((C - 1) * kDamasRows * 8));
            double u = row ? fma(-relax, sum[0] + sum[1], c) : 0.0;
            acc1 = acc2;
            acc2 = 0.0;
            k = k + 1 == nblk ? 0 : k + 1;
            const int64_t gn = (int64_t)k * kDamasRows + lane;
            yv = gn < G ? __ldg(yg + gn) : 0.0;
            double xv = 0.0;
#pragma unroll
            for (int j = 0; j < kDamasRows; ++j) {
                const double d = j < lane ? -relax * D[j * kDamasPad] : 0.0;
                const double n1 = -relax * N1[j * kDamasPad], n2 = -relax * N2[j * kDamasPad];
                const double xn = __shfl_sync(0xffffffffu, gs_clamp(u), j);
                u = fma(d, xn, u);
                acc1 = fma(n1, xn, acc1);
                acc2 = fma(n2, xn, acc2);
                xv = lane == j ? xn : xv;
            }
            xs[g0 + lane] = xv;
            if (t + 3 < steps)   // the other CTAs wait for step t's values at step t + 3
                for (int r = 1; r < C; ++r) tc::cluster_send(r, xs + g0 + lane, xv, &xbar[slot]);
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&xbar[slot]);
        }
    } else if (rank == 0 && warp <= 3) {
        // ---------------- the solver's tiles: rows of block t (+ 1, + 2), columns of block t
        const int which = warp - 1;
        for (int64_t t = 0; t < steps; ++t) {
            // the stage was read at step t - 3
            const bool here = t < kGsStages || tc::cluster_wait(&xbar[(t - kGsStages) % kGsRing],
                                                                (uint32_t)((t - kGsStages) / kGsRing) & 1, stop,
                                                                limit_ns);
            if (!__all_sync(0xffffffffu, here)) {
                tc::cluster_stop(stop, C);
                break;
            }
            const int64_t g0 = (t % nblk) * kDamasRows, gr = ((t + which) % nblk) * kDamasRows;
            const int st = (int)(t % kGsStages);
            double *dst = tiles + (st * 3 + which) * kGsTile + lane * kDamasPad;   // column `lane`
            const bool col = g0 + lane < G;
#pragma unroll 8
            for (int i = 0; i < kDamasRows; ++i) {
                const bool in = col && gr + i < G;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(tc::smem_u32(dst + i)),
                             "l"(Ab + (in ? (gr + i) * G + g0 + lane : 0)), "r"(in ? 8 : 0)
                             : "memory");
            }
            asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
            tc::mbar_arrive(&tbar[st]);
        }
    } else if (rank > 0) {
        // ---------------- sums over this CTA's columns: rows warp and warp + 16 of every block
        const int nch = (nblk + C - 2) / (C - 1);            // column blocks of a slice
        const int b0 = (rank - 1) * nch, b1 = min(b0 + nch, nblk);
        const int ngrp = b1 > b0 ? (b1 - b0 + 7) / 8 : 1;    // in groups of 8 column blocks
        // column blocks of the slice in which this lane has a column, and the lane's place in row `warp` of block 0
        const int mine = b1 > b0 ? b1 - b0 - ((int64_t)b1 * kDamasRows > G && (int64_t)(b1 - 1) * kDamasRows + lane >= G)
                                 : 0;
        const double *row0 = Ab + (int64_t)warp * G + (int64_t)b0 * kDamasRows + lane;
        const double *xl = xs + b0 * kDamasRows + lane;
        const int64_t half = 16 * G, block = kDamasRows * G;
        double a0[8], a1[8];
        // the group's elements of rows `warp` and `warp` + 16 of the block whose row `warp` is at `r`, if they exist
        auto fetch = [&](const double *r, bool ok0, bool ok1, int grp) {
            const double *r0 = r + grp * (8 * kDamasRows), *r1 = r0 + half;
            const int n0 = ok0 ? mine - grp * 8 : 0, n1 = ok1 ? mine - grp * 8 : 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                a0[q] = a1[q] = 0.0;
                if (q < n0) a0[q] = __ldg(r0 + q * kDamasRows);
                if (q < n1) a1[q] = __ldg(r1 + q * kDamasRows);
            }
        };
        const bool last0 = (int64_t)(nblk - 1) * kDamasRows + warp < G, last1 = (int64_t)(nblk - 1) * kDamasRows + warp + 16 < G;
        int k = 0;
        const double *rk = row0;   // row `warp` of block k
        if (steps > 0) fetch(rk, true, true, 0);
        for (int64_t t = 0; t < steps; ++t) {
            const int kn = k + 1 == nblk ? 0 : k + 1;
            const double *rn = kn ? rk + block : row0;
            if (t >= 3) {
                if (!__all_sync(0xffffffffu, tc::cluster_wait(&xbar[(t - 3) % kGsRing],
                                                              (uint32_t)((t - 3) / kGsRing) & 1, stop, limit_ns))) {
                    tc::cluster_stop(stop, C);
                    break;
                }
                if (threadIdx.x == 0 && t + 1 < steps)
                    tc::mbar_arrive_expect_tx(&xbar[(t - 3) % kGsRing], kDamasRows * 8);   // for step t + 1
            }
            // places in the slice of block k and of the blocks solved at steps t - 1 and t - 2 (the solver's)
            const int ek = k - b0, e1 = t >= 1 ? (k == 0 ? nblk - 1 : k - 1) - b0 : -1;
            const int e2 = t >= 2 ? (k <= 1 ? nblk - 2 + k : k - 2) - b0 : -1;
            double s0 = 0.0, s1 = 0.0;
            for (int grp = 0; grp < ngrp; ++grp) {
                double c0[8], c1[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    c0[q] = a0[q];
                    c1[q] = a1[q];
                }
                // the next group, or the next block's first, lands while this one is summed and waited for
                if (grp + 1 < ngrp) fetch(rk, k + 1 < nblk || last0, k + 1 < nblk || last1, grp + 1);
                else if (t + 1 < steps) fetch(rn, kn + 1 < nblk || last0, kn + 1 < nblk || last1, 0);
                double p0 = 0.0, p1 = 0.0;
                const int left = b1 - b0 - grp * 8, gk = ek - grp * 8, g1 = e1 - grp * 8, g2 = e2 - grp * 8;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    if (q >= left || q == g1 || q == g2) continue;   // uniform
                    const double xv = xl[(grp * 8 + q) * kDamasRows];
                    double &t0 = q & 1 ? p0 : s0, &t1 = q & 1 ? p1 : s1;
                    // within the block only the columns right of the row; the others are left out and not multiplied
                    // by zero, as an old value (the dirty map's to begin with) may be infinite or NaN
                    if (q == gk) {
                        if (lane > warp) t0 = fma(c0[q], xv, t0);
                        if (lane > warp + 16) t1 = fma(c1[q], xv, t1);
                    } else {
                        t0 = fma(c0[q], xv, t0);
                        t1 = fma(c1[q], xv, t1);
                    }
                }
                s0 += p0;
                s1 += p1;
            }
            // lanes 0..15 end up with row warp's sum, the others with row warp + 16's
            const double give = lane < 16 ? s1 : s0;
            double s = (lane < 16 ? s0 : s1) + __shfl_xor_sync(0xffffffffu, give, 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            const int slot = (int)(t % kGsRing);
            if ((lane & 15) == 0)
                tc::cluster_send(0, part + (slot * kDamasMaxCta + rank) * kDamasRows + warp + (lane ? 16 : 0), s, &pbar[slot]);
            k = kn;
            rk = rn;
        }
    }
    const bool stopped = tc::cluster_end(cluster, stop);
    if (rank == 0)   // a wait ran out, in whichever CTA: no result
        for (int64_t i = threadIdx.x; i < G; i += kDamasThreads)
            xg[i] = stopped ? __longlong_as_double(0x7ff8000000000000ll) : xs[i];
}

}  // namespace acb

using namespace acb;

extern "C" {

int acb_psf_f64(const acb_map_params *p, int num_sources, const int64_t *sources, double wavenumber, const double *r0,
                const double *rm, int round_f32, double *out_psf, void *stream)
{
    if (!p || !sources || !r0 || !rm || !out_psf) return ACB_ERR_ARG;
    if (p->steer_type < 1 || p->steer_type > 4) return ACB_ERR_ARG;
    if (p->num_mics < 1 || p->num_grid <= 0 || num_sources <= 0) return ACB_ERR_SHAPE;
    if (p->glibc_faithful && (!p->sincos_table || p->sincos_table_slots <= 0 ||
                              (p->sincos_table_slots & (p->sincos_table_slots - 1))))
        return ACB_ERR_ARG;
    const int M = p->num_mics;
    const int64_t G = p->num_grid;
    if ((num_sources + 7) / 8 > 65535) return ACB_ERR_SHAPE;
    const int64_t tiles = (G + kPsfTile - 1) / kPsfTile;
    const bool mirror = num_sources == G && tiles * (tiles + 1) / 2 >= kNumSMs;
    const int per = mirror ? 4 : psf_per(G, num_sources), ns = kPsfWarps * per;
    const dim3 grid((unsigned)tiles, (unsigned)((num_sources + ns - 1) / ns));
    const uint64_t mask = p->glibc_faithful ? (uint64_t)p->sincos_table_slots - 1 : 0;
    cudaStream_t s = as_stream(stream);
    auto launch = [&](auto kern) {
        if (const int st = allow_smem(kern, kPsfSmem, kPsfSmem)) return st;
        kern<<<grid, 32 * kPsfWarps, kPsfSmem, s>>>(M, G, num_sources, sources, r0, rm, wavenumber, p->sincos_table, mask,
                                                    p->glibc_faithful, round_f32, out_psf);
        return check_launch();
    };
#define ACB_PSF(ST)                                                                             \
    return mirror     ? launch(psf_kernel<ST, 4, true>)                                         \
           : per == 4 ? launch(psf_kernel<ST, 4, false>)                                        \
           : per == 2 ? launch(psf_kernel<ST, 2, false>)                                        \
                      : launch(psf_kernel<ST, 1, false>)
    switch (p->steer_type) {
    case 1: ACB_PSF(1);
    case 2: ACB_PSF(2);
    case 3: ACB_PSF(3);
    default: ACB_PSF(4);
    }
#undef ACB_PSF
}

int acb_damas_gauss_seidel_f64(const double *psf, int64_t num_grid, int num_bins, const double *dirty_map,
                               double *solution, int n_iter, double relax, int cta_per_bin, void *stream)
{
    if (!psf || !dirty_map || !solution) return ACB_ERR_ARG;
    if (num_grid <= 0 || num_bins <= 0 || n_iter < 0) return ACB_ERR_SHAPE;
    int dev = 0, sms = 0, smem_max = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return ACB_ERR_CUDA;
    const size_t smem = (size_t)damas_smem_doubles(num_grid) * sizeof(double);
    if (smem > (size_t)smem_max) return ACB_ERR_UNSUPPORTED;   // the solution lives in shared memory
    int C = cta_per_bin;
    if (C == 0) {
        C = kDamasMaxCta;
        while (C > 1 && (int64_t)num_bins * C > sms) C >>= 1;
    }
    if (C != 1 && C != 2 && C != 4 && C != 8) return ACB_ERR_ARG;
    if ((int64_t)num_bins * C > 0x7fffffff) return ACB_ERR_SHAPE;
    // the form two blocks ahead: at least six blocks, four CTAs, and its tiles beside the solution
    const int64_t smem_ahead = gs_smem_bytes(num_grid);
    const bool ahead = num_grid > 5 * kDamasRows && C >= 4 && smem_ahead <= smem_max - 1024;
    const size_t smem_used = ahead ? (size_t)smem_ahead : smem;
    if (const int st = ahead ? allow_smem(damas_ahead_kernel, smem_used, smem_max - 1024)
                             : allow_smem(damas_kernel, smem_used, smem_max))
        return st;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(num_bins * C));
    cfg.blockDim = dim3(kDamasThreads);
    cfg.dynamicSmemBytes = smem_used;
    cfg.stream = as_stream(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t err =
        ahead ? cudaLaunchKernelEx(&cfg, damas_ahead_kernel, psf, num_grid, dirty_map, solution, n_iter, relax,
                                   tc_wait_limit_ns())
              : cudaLaunchKernelEx(&cfg, damas_kernel, psf, num_grid, dirty_map, solution, n_iter, relax);
    if (err != cudaSuccess) return ACB_ERR_CUDA;
    return check_launch();
}

}  // extern "C"
