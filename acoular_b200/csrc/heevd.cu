// Batched Hermitian eigendecomposition of CSMs (PowerSpectra._get__evd, acoular/spectra.py:351-364: numpy's
// eigh per bin, eigenvalues ascending, eigenvectors in the columns), hand-written for the device.
//
// Three kernels, one matrix per CTA (or per column slab), every bin of a request in one launch each:
//   heevd_tridiag_kernel : Householder reduction to a real symmetric tridiagonal matrix, A = Q T Q^H.
//                          Step i reflects column i below the diagonal, x -> beta e1 with H = I - tau v v^H
//                          (beta real, tau complex, v_0 = 1), then updates the trailing matrix
//                          A22 <- H^H A22 H = A22 - v w^H - w v^H, p = tau A22 v, w = p - (tau/2)(p^H v) v,
//                          on A22's lower triangle only (half the memory traffic of the full update).
//                          heevd_tridiag_cluster_kernel does it in the shared memory of a cluster where it fits.
//   heevd_tql_kernel     : eigenvalues and eigenvectors of T by implicit QL sweeps with Wilkinson shifts
//                          (the EISPACK tql2 scheme), eigenvectors accumulated in Z.  One warp forms a
//                          sweep's plane rotations from d and e; the others apply those of the sweep before
//                          to their rows of Z.  Then the ascending order of the eigenvalues.
//   heevd_back_kernel    : eigenvectors of A, V = Q Z = H_0 H_1 ... H_{M-2} Z, for a slab of columns held in
//                          shared memory, reflectors applied from the last; each warp owns columns of the
//                          slab, so the reflectors need no barrier; columns written in ascending eigenvalue
//                          order.
// All arithmetic is FP64.  The eigenvectors differ from LAPACK's by a phase per column (any unit factor is an
// eigenvector); the eigenvalue beamformers use them only through |v^H h|.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <cooperative_groups.h>

#include "common.cuh"
#include "tc_common.cuh"

namespace cg = cooperative_groups;

namespace acb {

constexpr int kEvThreads = 256;
constexpr int kEvWarps = kEvThreads / 32;
// the QL kernel's CTA: one warp forms the rotations, four apply them; small, so that every matrix of a 513-bin request
// has its CTA resident at once (the sweeps are a serial recurrence, so a matrix takes the same time in any wave)
constexpr int kQlThreads = 160;
constexpr int kEvMaxRows = 4096;
constexpr int kQlMaxIter = 60;   // QL iterations per eigenvalue before giving up (info = 1)

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b)   // conj(a) * b
{
    return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}

// Block sum of a double (all threads receive it); `red` holds kEvWarps doubles.
__device__ __forceinline__ double block_sum(double v, double *red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kEvWarps; ++w) t += red[w];
    return t;
}

// A (B, M, M) complex128 row-major, overwritten; d, e (B, M); tau (B, M) complex; vh (B, M - 1, M): reflector i
// in entries i + 1 .. M - 1 of row i.
__global__ void __launch_bounds__(kEvThreads) heevd_tridiag_kernel(double2 *__restrict__ Aall, int M,
                                                                   double *__restrict__ dall, double *__restrict__ eall,
                                                                   double2 *__restrict__ tauall,
                                                                   double2 *__restrict__ vhall)
{
    extern __shared__ double2 ev_sm[];
    double2 *v = ev_sm;        // [M]
    double2 *p = ev_sm + M;    // [M]
    __shared__ double red[kEvWarps];
    __shared__ double2 s_tau, s_scale;
    __shared__ double s_beta;
    const int b = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double2 *A = Aall + (int64_t)b * M * M;
    double *d = dall + (int64_t)b * M;
    double *e = eall + (int64_t)b * M;
    double2 *tau = tauall + (int64_t)b * M;
    double2 *vh = vhall + (int64_t)b * (M > 1 ? M - 1 : 1) * M;

    for (int i = 0; i < M - 1; ++i) {
        for (int r = i + 1 + tid; r < M; r += kEvThreads) v[r] = A[(int64_t)r * M + i];
        __syncthreads();
        double part = 0.0;
        for (int r = i + 2 + tid; r < M; r += kEvThreads) part += v[r].x * v[r].x + v[r].y * v[r].y;
        const double xn2 = block_sum(part, red);
        if (tid == 0) {
            const double2 al = v[i + 1];
            d[i] = A[(int64_t)i * M + i].x;
            if (xn2 == 0.0 && al.y == 0.0) {   // already real and reduced: H = I
                s_beta = al.x;
                s_tau = make_double2(0.0, 0.0);
                s_scale = make_double2(0.0, 0.0);
            } else {
                const double beta = -copysign(sqrt(al.x * al.x + al.y * al.y + xn2), al.x);
                s_beta = beta;
                s_tau = make_double2((beta - al.x) / beta, -al.y / beta);
                // 1 / (alpha - beta)
                const double2 den = make_double2(al.x - beta, al.y);
                const double dd = den.x * den.x + den.y * den.y;
                s_scale = make_double2(den.x / dd, -den.y / dd);
            }
            e[i] = s_beta;
            tau[i] = s_tau;
        }
        __syncthreads();
        const double2 tu = s_tau;
        if (tu.x == 0.0 && tu.y == 0.0) {
            for (int r = i + 1 + tid; r < M; r += kEvThreads)
                vh[(int64_t)i * M + r] = make_double2(r == i + 1 ? 1.0 : 0.0, 0.0);
            __syncthreads();
            continue;
        }
        const double2 sc = s_scale;
        for (int r = i + 1 + tid; r < M; r += kEvThreads) {
            const double2 vr = r == i + 1 ? make_double2(1.0, 0.0) : cmul(v[r], sc);
            v[r] = vr;
            vh[(int64_t)i * M + r] = vr;
        }
        __syncthreads();
        // p = tau A22 v: a warp per row, lanes along the row.  Only the lower triangle of A22 is kept up to
        // date (A is Hermitian): row r's entries right of the diagonal are conj(A[c][r]), read down column r
        for (int r = i + 1 + warp; r < M; r += kEvWarps) {
            const double2 *row = A + (int64_t)r * M;
            double ar = 0.0, ai = 0.0;
            for (int c = i + 1 + lane; c < M; c += 32) {
                double2 a;
                if (c <= r) {
                    a = row[c];
                } else {
                    a = A[(int64_t)c * M + r];
                    a.y = -a.y;
                }
                const double2 x = v[c];
                ar = fma(a.x, x.x, fma(-a.y, x.y, ar));
                ai = fma(a.x, x.y, fma(a.y, x.x, ai));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                ar += __shfl_xor_sync(0xffffffffu, ar, o);
                ai += __shfl_xor_sync(0xffffffffu, ai, o);
            }
            if (lane == 0) p[r] = cmul(tu, make_double2(ar, ai));
        }
        __syncthreads();
        // alpha2 = -(tau / 2) (p^H v);  w = p + alpha2 v  (into p)
        double pr = 0.0, pi = 0.0;
        for (int r = i + 1 + tid; r < M; r += kEvThreads) {
            const double2 t = cmulc(p[r], v[r]);
            pr += t.x;
            pi += t.y;
        }
        const double sr = block_sum(pr, red);
        const double si = block_sum(pi, red);
        const double2 al2 = cmul(make_double2(-0.5 * tu.x, -0.5 * tu.y), make_double2(sr, si));
        for (int r = i + 1 + tid; r < M; r += kEvThreads) {
            const double2 t = cmul(al2, v[r]);
            p[r] = make_double2(p[r].x + t.x, p[r].y + t.y);
        }
        __syncthreads();
        // A22 -= v w^H + w v^H on the lower triangle (c <= r): a warp per row, lanes along the row
        for (int r = i + 1 + warp; r < M; r += kEvWarps) {
            for (int c = i + 1 + lane; c <= r; c += 32) {
                const double2 vr = v[r], wr = p[r], vc = v[c], wc = p[c];
                const double2 t1 = cmulc(wc, vr);   // v_r conj(w_c)
                const double2 t2 = cmulc(vc, wr);   // w_r conj(v_c)
                double2 a = A[(int64_t)r * M + c];
                a.x -= t1.x + t2.x;
                a.y -= t1.y + t2.y;
                A[(int64_t)r * M + c] = a;
            }
        }
        __syncthreads();
    }
    if (tid == 0) {
        d[M - 1] = A[(int64_t)(M - 1) * M + (M - 1)].x;
        e[M - 1] = 0.0;
        tau[M - 1] = make_double2(0.0, 0.0);
    }
}

// The same reduction with the lower triangle in the shared memory of a cluster of C CTAs (rows r = rank + C l in CTA
// `rank`, packed), for matrices that fit (up to about 150 rows in one CTA, 205 in two, 270 in four, 335 in eight).
// The rank-2 update of step i - 1 and the product A22 v of step i are one pass over the stored elements: every CTA
// first forms its part of column i of the updated matrix alone and sends it to all; each warp of every CTA derives the
// reflector from it for itself; the pass updates each element a = A[r][c] and adds a v_c to row r's product and
// conj(a) v_r to row c's; every CTA sends its partial products to all, sums the C parts and forms w.  The sends are
// asynchronous stores counted on the receiver's mbarriers: a step has two one-way latencies, no cluster barrier.
// Buffers: a CTA sends its products of step i + 1 only after it has every CTA's column i + 1, which a CTA sends after
// its last read of step i's products: one buffer.  A CTA may send column i + 1 while another still reads column i,
// but column i + 2 only after that one's products of step i + 1: two buffers.  The same order keeps each mbarrier's
// phases apart.
// Bound: the latency of a step (two sends, a warp sum, a block sum, a reciprocal square root, a division), not its 16
// FMAs per stored element; the global-memory form above runs one CTA per matrix and moves each trailing matrix through
// L2 three times per step.
// csm (B, M, M) is read only: its lower triangle, as above.
__host__ __device__ constexpr int ev_packed(int rank, int C, int l) { return l * (rank + 1) + C * (l * (l - 1) / 2); }

template <int MINB>
__global__ void __launch_bounds__(kEvThreads, MINB)
    heevd_tridiag_cluster_kernel(const double2 *__restrict__ csm, int M, double *__restrict__ dall,
                                 double *__restrict__ eall, double2 *__restrict__ tauall, double2 *__restrict__ vhall,
                                 uint64_t limit_ns)
{
    extern __shared__ double2 ev_sm[];
    __shared__ uint64_t bars[2];   // column; products
    __shared__ double red[2][kEvWarps];
    __shared__ int stop_s;
    volatile int *stop = &stop_s;
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int b = blockIdx.x / C;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double2 *v = ev_sm, *w = v + M;                 // [M] pending update: A -= v w^H + w v^H
    double2 *x0 = w + M;                            // [2][M] column i
    double2 *part = x0 + 2 * M;                     // [C][M] products, by sender
    double2 *q = part + C * M;                      // [kEvWarps][M] this CTA's column products, by warp
    double2 *rowp = q + kEvWarps * M;               // [ceil(M / C)] its row products
    double2 *rows = rowp + (M + C - 1) / C;         // packed lower rows
    const int nl = (M - rank + C - 1) / C;
    const double2 *A = csm + (int64_t)b * M * M;
    double *d = dall + (int64_t)b * M;
    double *e = eall + (int64_t)b * M;
    double2 *tau = tauall + (int64_t)b * M;
    double2 *vh = vhall + (int64_t)b * (M > 1 ? M - 1 : 1) * M;
    if (tid == 0) {
        tc::mbar_init(&bars[0], 1);
        tc::mbar_init(&bars[1], 1);
        stop_s = 0;
        tc::fence_mbar_init();
    }
    for (int l = warp; l < nl; l += kEvWarps) {
        const int r = rank + C * l;
        for (int c = lane; c <= r; c += 32) rows[ev_packed(rank, C, l) + c] = __ldg(A + (int64_t)r * M + c);
    }
    for (int r = tid; r < M; r += kEvThreads) v[r] = w[r] = make_double2(0.0, 0.0);
    cluster.sync();

    for (int i = 0; i < M; ++i) {
        double2 *x = x0 + (i & 1) * M;
        const int l0 = i < rank ? 0 : (i - rank) / C + 1;   // first own row below i
        // own part of column i of the updated matrix (row i itself included)
        if (tid == 0) tc::mbar_arrive_expect_tx(&bars[0], (uint32_t)((M - i) * sizeof(double2)));
        const int lx = i % C == rank ? i / C : l0;
        const double2 vi = v[i], wi = w[i];
        for (int l = lx + tid; l < nl; l += kEvThreads) {
            const int r = rank + C * l;
            const double2 t1 = cmulc(wi, v[r]), t2 = cmulc(vi, w[r]);   // v_r conj(w_i), w_r conj(v_i)
            const double2 a = rows[ev_packed(rank, C, l) + i];
            for (int k = 0; k < C; ++k)
                tc::cluster_send(k, x + r, make_double2(a.x - (t1.x + t2.x), a.y - (t1.y + t2.y)), &bars[0]);
        }
        bool here = tc::cluster_wait(&bars[0], i & 1, stop, limit_ns);
        if (rank == 0 && tid == 0) d[i] = x[i].x;
        if (i == M - 1) {
            if (!here) tc::cluster_stop(stop, C);
            break;
        }
        if (tid == 0) tc::mbar_arrive_expect_tx(&bars[1], (uint32_t)(C * (M - 1 - i) * sizeof(double2)));
        // the reflector, by every warp: beta = -sign(Re alpha) |(alpha, x)|, tau = (beta - alpha) / beta,
        // v = (1, x / (alpha - beta)); H = I where the column is real and reduced already
        double xn2 = 0.0;
        for (int r = i + 2 + lane; r < M; r += 32) xn2 = fma(x[r].x, x[r].x, fma(x[r].y, x[r].y, xn2));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) xn2 += __shfl_xor_sync(0xffffffffu, xn2, o);
        const double2 al = x[i + 1];
        const double ss = fma(al.x, al.x, fma(al.y, al.y, xn2));
        const bool reduced = (xn2 == 0.0 && al.y == 0.0) || ss == 0.0;
        double beta = al.x;
        double2 tu = make_double2(0.0, 0.0), sc = tu;
        if (!reduced) {
            const double y = rsqrt(ss);   // 1 / |beta|
            beta = -copysign(ss * y, al.x);
            tu = make_double2(fma(fabs(al.x), y, 1.0), al.y * copysign(y, al.x));
            const double2 den = make_double2(al.x - beta, al.y);
            const double dd = 1.0 / fma(den.x, den.x, den.y * den.y);
            sc = make_double2(den.x * dd, -den.y * dd);
        }
        const double2 first = make_double2(reduced ? 0.0 : 1.0, 0.0);   // v[i + 1]; no update if H = I
        // own rows in groups of four from the last one; a warp's first group has its longest rows and starts its
        // column products, the others add to them
        const int ngrp = (nl - l0 + 3) / 4;
        for (int k = warp; k < ngrp; k += kEvWarps) {
            const int lt = nl - 1 - 4 * k;   // the group's last (longest) row
            const int rmax = rank + C * lt;
            double2 vr[4], wr[4], nr[4], *rp[4];
            int rr[4];
            double acc[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int l = max(lt - j, l0);
                const int r = rank + C * l;
                rr[j] = lt - j >= l0 ? r : -1;   // -1: no such row, no element
                vr[j] = v[r];
                wr[j] = w[r];
                nr[j] = r == i + 1 ? first : cmul(x[r], sc);
                rp[j] = rows + ev_packed(rank, C, l);
                acc[2 * j] = acc[2 * j + 1] = 0.0;
            }
            for (int c = i + 1 + lane; c <= rmax; c += 32) {
                double2 u[4];   // every load before the first store: nothing waits for a row's update
#pragma unroll
                for (int j = 0; j < 4; ++j) u[j] = rp[j][min(c, max(rr[j], 0))];
                const double2 vc = v[c], wc = w[c], nc = c == i + 1 ? first : cmul(x[c], sc);
                double2 qc = make_double2(0.0, 0.0);
                if (k != warp) qc = q[warp * M + c];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const double2 t1 = cmulc(wc, vr[j]), t2 = cmulc(vc, wr[j]);
                    u[j].x -= t1.x + t2.x;
                    u[j].y -= t1.y + t2.y;
                    if (c > rr[j]) u[j] = make_double2(0.0, 0.0);
                    acc[2 * j] = fma(u[j].x, nc.x, fma(-u[j].y, nc.y, acc[2 * j]));
                    acc[2 * j + 1] = fma(u[j].x, nc.y, fma(u[j].y, nc.x, acc[2 * j + 1]));
                    const double2 n = c == rr[j] ? make_double2(0.0, 0.0) : nr[j];   // conj(a) v_r left of the diagonal
                    qc.x = fma(u[j].x, n.x, fma(u[j].y, n.y, qc.x));
                    qc.y = fma(u[j].x, n.y, fma(-u[j].y, n.x, qc.y));
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (c <= rr[j]) rp[j][c] = u[j];
                q[warp * M + c] = qc;
            }
            // the eight sums: halve the values a lane carries at each of three steps, then two plain steps; the
            // lane ends up with value lane / 4
#pragma unroll
            for (int h = 4, o = 16; h >= 1; h >>= 1, o >>= 1)
#pragma unroll
                for (int u = 0; u < h; ++u) {
                    const bool up = lane & o;
                    const double send = up ? acc[u] : acc[u + h], keep = up ? acc[u + h] : acc[u];
                    acc[u] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
            const double other = __shfl_xor_sync(0xffffffffu, acc[0], 4);
            const int l = lt - (lane >> 3);
            if ((lane & 7) == 0 && l >= l0) rowp[l] = make_double2(acc[0], other);
        }
        __syncthreads();
        // this CTA's part of tau A22 v to every CTA
        const int nw = min(ngrp, kEvWarps);
        for (int c = i + 1 + tid; c < M; c += kEvThreads) {
            double2 s = make_double2(0.0, 0.0);
            if (c % C == rank) s = rowp[c / C];
            for (int u = 0; u < nw; ++u) {
                if (c > rank + C * (nl - 1 - 4 * u)) break;   // past this warp's longest row, and the next ones'
                s.x += q[u * M + c].x;
                s.y += q[u * M + c].y;
            }
            s = cmul(tu, s);
            for (int k = 0; k < C; ++k) tc::cluster_send(k, part + rank * M + c, s, &bars[1]);
        }
        here = tc::cluster_wait(&bars[1], i & 1, stop, limit_ns) && here;
        // w = p - (tau / 2) (p^H v) v
        double sr = 0.0, si = 0.0;
        for (int r = i + 1 + tid; r < M; r += kEvThreads) {
            double2 p = part[r];
            for (int k = 1; k < C; ++k) {
                p.x += part[k * M + r].x;
                p.y += part[k * M + r].y;
            }
            const double2 vn = r == i + 1 ? first : cmul(x[r], sc);
            const double2 t = cmulc(p, vn);
            sr += t.x;
            si += t.y;
            w[r] = p;
            v[r] = vn;
            if (rank == i % C) vh[(int64_t)i * M + r] = r == i + 1 ? make_double2(1.0, 0.0) : vn;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sr += __shfl_xor_sync(0xffffffffu, sr, o);
            si += __shfl_xor_sync(0xffffffffu, si, o);
        }
        if (lane == 0) {
            red[0][warp] = sr;
            red[1][warp] = si;
        }
        __syncthreads();
        sr = si = 0.0;
#pragma unroll
        for (int u = 0; u < kEvWarps; ++u) {
            sr += red[0][u];
            si += red[1][u];
        }
        const double2 al2 = cmul(make_double2(-0.5 * tu.x, -0.5 * tu.y), make_double2(sr, si));
        for (int r = i + 1 + tid; r < M; r += kEvThreads) {
            const double2 t = cmul(al2, v[r]);
            w[r] = make_double2(w[r].x + t.x, w[r].y + t.y);
        }
        if (rank == i % C && tid == 0) {
            e[i] = beta;
            tau[i] = tu;
        }
        if (__syncthreads_or(!here)) {
            tc::cluster_stop(stop, C);
            break;
        }
    }
    const bool stopped = tc::cluster_end(cluster, stop);
    if (rank == 0) {
        if (tid == 0) {
            e[M - 1] = 0.0;
            tau[M - 1] = make_double2(0.0, 0.0);
        }
        if (stopped)   // a wait ran out, in whichever CTA: no result
            for (int r = tid; r < M; r += kEvThreads) {
                d[r] = __longlong_as_double(0x7ff8000000000000ll);
                e[r] = 0.0;
                tau[r] = make_double2(0.0, 0.0);
            }
    }
}

// d, e (B, M) -> eigenvalues w (B, M) ascending, Z (B, M, M) column-major (column j = eigenvector of the
// unsorted eigenvalue j), perm (B, M): sorted position q holds unsorted index perm[q]; info[b] = 1 if a QL
// iteration did not converge.
// Warp 0 forms the rotations of a sweep while the other warps apply those of the sweep before to Z, one barrier per
// sweep.  Bound: the serial chain of a rotation (two products, the sum of squares, a reciprocal square root and five
// more dependent operations); the library's hypot and a division made it twice as long, and the application
// waited for it (64 matrices of 112 rows 4.2 -> 2.7 ms).  Lane 0 runs the whole chain by itself, as a sweep reads
// entries that it has stored to a little earlier, and the range test runs beside the reciprocal square root:
// 2.7 -> 1.8 ms, 226 clocks per rotation (the loop in all lanes with only the stores in lane 0, and the test ahead of the
// root: about 350; the loop in all lanes with a warp barrier per rotation: 240).  The application hides behind the chain
// (without it the time is the same).
__global__ void __launch_bounds__(kQlThreads) heevd_tql_kernel(const double *__restrict__ dall,
                                                               const double *__restrict__ eall, int M,
                                                               double *__restrict__ wall, double *__restrict__ Zall,
                                                               int *__restrict__ permall, int *__restrict__ info)
{
    extern __shared__ double ql_sm[];
    double *d = ql_sm;           // [M]
    double *e = ql_sm + M;       // [M]
    double *cs2 = ql_sm + 2 * M; // [2][M] cosine of the rotation of (i, i + 1), by sweep parity
    double *sn2 = ql_sm + 4 * M; // [2][M] sine
    __shared__ int s_m[2], s_stop[2], s_fail;   // rotations i = m - 1 .. stop of a sweep; m = 0: no further sweep
    const int b = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31;
    double *Z = Zall + (int64_t)b * M * M;
    int bad = 0;
    for (int k = tid; k < M; k += kQlThreads) {
        d[k] = dall[(int64_t)b * M + k];
        e[k] = eall[(int64_t)b * M + k];
        bad |= d[k] != d[k] || e[k] != e[k];
    }
    // a NaN in T (a NaN matrix, or a tridiagonalisation that gave up): no result, and no sweeps for one
    bad = __syncthreads_or(bad);
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    if (bad)
        for (int k = tid; k < M; k += kQlThreads) d[k] = nan;
    for (int64_t idx = tid; idx < (int64_t)M * M; idx += kQlThreads)
        Z[idx] = bad ? nan : (idx / M == idx % M) ? 1.0 : 0.0;
    if (tid == 0) s_fail = bad;
    __syncthreads();
    const double eps = 2.220446049250313e-16;
    int l = bad ? M : 0, iter = 0;   // warp 0: the eigenvalue being sought and its sweeps so far
    for (int sweep = 0;; ++sweep) {
        const int buf = sweep & 1;
        if (tid < 32) {
            // the next sweep: skip the eigenvalues that have converged (their off-diagonal is negligible)
            int m = 0;
            while (l < M) {
                m = M - 1;
                for (int k0 = l; k0 < M - 1; k0 += 32) {
                    const int k = k0 + lane;
                    const bool small = k < M - 1 && fabs(e[k]) <= eps * (fabs(d[k]) + fabs(d[k + 1]));
                    const unsigned any = __ballot_sync(0xffffffffu, small);
                    if (any) {
                        m = k0 + __ffs(any) - 1;
                        break;
                    }
                }
                if (m != l && iter < kQlMaxIter) break;
                if (m != l && lane == 0) s_fail = 1;
                ++l;
                iter = 0;
            }
            if (l >= M) {
                if (lane == 0) s_m[buf] = 0;
            } else {
                ++iter;
                double *cs = cs2 + buf * M, *sn = sn2 + buf * M;
                __syncwarp();   // the search's reads come before the chain's stores
                if (lane == 0) {
                    double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
                    const double h = fabs(g) < 1e150 ? sqrt(fma(g, g, 1.0)) : fabs(g);
                    double dn = d[m];   // d[i + 1] of the rotation at hand
                    g = dn - d[l] + e[l] / (g + copysign(h, g));
                    double s = 1.0, c = 1.0, p = 0.0;
                    double en = e[m - 1], dp = d[m - 1];   // read one rotation ahead of the stores
                    int i = m - 1;
                    bool restart = false;
                    for (; i >= l; --i) {
                        const double ei = en, di = dp;
                        const int j = max(i - 1, 0);
                        en = e[j];
                        dp = d[j];
                        const double f = s * ei, bb = c * ei;
                        const double x = fma(f, f, g * g);
                        double rinv = rsqrt(x), r = x * rinv;
                        if (!(x > 1e-280 && x < 1e280)) {
                            r = hypot(f, g);
                            if (r == 0.0) {   // split: deflate and restart from the same l
                                e[i + 1] = 0.0;
                                d[i + 1] = dn - p;
                                e[m] = 0.0;
                                restart = true;
                                break;
                            }
                            rinv = 1.0 / r;
                        }
                        e[i + 1] = r;
                        s = f * rinv;
                        c = g * rinv;
                        g = dn - p;
                        r = (di - g) * s + 2.0 * c * bb;
                        p = s * r;
                        d[i + 1] = g + p;
                        cs[i] = c;
                        sn[i] = s;
                        g = c * r - bb;
                        dn = di;
                    }
                    if (!restart) {
                        d[l] = dn - p;
                        e[l] = g;
                        e[m] = 0.0;
                    }
                    s_m[buf] = m;
                    s_stop[buf] = restart ? i + 1 : l;
                }
                __syncwarp();
            }
        } else if (sweep > 0) {
            // apply the rotations of the sweep before in the order they were formed to every row k of Z.  Rotation i
            // reads entry i and writes entry i + 1 of the row, so every entry is read before it is written: the
            // reads of 8 rotations are issued together, ahead of their writes, and their latency is paid once per 8
            const double *cs = cs2 + (buf ^ 1) * M, *sn = sn2 + (buf ^ 1) * M;
            const int m = s_m[buf ^ 1], stop = s_stop[buf ^ 1];
            for (int k = tid - 32; k < M; k += kQlThreads - 32) {
                double *zk = Z + k;   // entry i of row k at zk[i * M]
                double carry = zk[(int64_t)m * M];
                int i = m - 1;
                for (; i - 7 >= stop; i -= 8) {
                    double zv[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) zv[j] = zk[(int64_t)(i - j) * M];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int ii = i - j;
                        zk[(int64_t)(ii + 1) * M] = sn[ii] * zv[j] + cs[ii] * carry;
                        carry = cs[ii] * zv[j] - sn[ii] * carry;
                    }
                }
                for (; i >= stop; --i) {
                    const double zi = zk[(int64_t)i * M];
                    zk[(int64_t)(i + 1) * M] = sn[i] * zi + cs[i] * carry;
                    carry = cs[i] * zi - sn[i] * carry;
                }
                zk[(int64_t)stop * M] = carry;
            }
        }
        __syncthreads();
        if (s_m[buf] == 0) break;
    }
    // ascending order, ties by index (as a stable sort), NaN last: a permutation whatever the values, since the
    // back-transformation reads columns by it
    for (int k = tid; k < M; k += kQlThreads) {
        const double dk = d[k];
        int rank = 0;
        for (int j = 0; j < M; ++j) {
            const double dj = d[j];
            rank += dk != dk ? dj == dj || j < k : dj < dk || (dj == dk && j < k);
        }
        wall[(int64_t)b * M + rank] = dk;
        permall[(int64_t)b * M + rank] = k;
    }
    if (tid == 0 && info) info[b] = s_fail;
}

// V = Q Z for the output columns [c0, c0 + W) of one matrix, reflectors applied from the last.  The slab
// sits in shared memory column by column (stride M + 1), and warp w owns the slab's columns w, w + 8, ..:
// for each reflector a warp forms tau v^H S[:, j] over its own columns (lanes along the rows, a shuffle
// reduction) and updates them, so no barrier separates the reflectors.  The reflector's entries are read
// by all warps from L1.  V (B, M, M) complex128 row-major, columns = eigenvectors in ascending order.
template <int CPW>
__global__ void __launch_bounds__(kEvThreads) heevd_back_kernel(const double2 *__restrict__ vhall,
                                                                const double2 *__restrict__ tauall,
                                                                const double *__restrict__ Zall,
                                                                const int *__restrict__ permall, int M, int W,
                                                                int ldv, double2 *__restrict__ Vall)
{
    extern __shared__ double2 bk_sm[];
    const int Mp = M + 1;
    double2 *S = bk_sm;                    // [W][Mp]: entry r of slab column j at S[j * Mp + r]
    const int b = blockIdx.x;
    const int c0 = blockIdx.y * W;
    const int nw = min(W, M - c0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double2 *vh = vhall + (int64_t)b * (M > 1 ? M - 1 : 1) * M;
    const double2 *tau = tauall + (int64_t)b * M;
    const double *Z = Zall + (int64_t)b * M * M;
    const int *perm = permall + (int64_t)b * M;
    for (int j = warp; j < nw; j += kEvWarps) {
        const double *zc = Z + (int64_t)perm[c0 + j] * M;   // column-major Z: eigenvector of T
        for (int r = lane; r < M; r += 32) S[j * Mp + r] = make_double2(zc[r], 0.0);
    }
    // this warp's columns (j < nw)
    int nq = 0;
    while (nq < CPW && warp + kEvWarps * nq < nw) ++nq;
    for (int i = M - 2; i >= 0 && nq > 0; --i) {
        const double2 t = __ldg(tau + i);
        if (t.x == 0.0 && t.y == 0.0) continue;
        const double2 *v = vh + (int64_t)i * M;
        double ar[CPW], ai[CPW];
#pragma unroll
        for (int q = 0; q < CPW; ++q) ar[q] = ai[q] = 0.0;
        for (int r = i + 1 + lane; r < M; r += 32) {
            const double2 vr = __ldg(v + r);
#pragma unroll
            for (int q = 0; q < CPW; ++q) {
                if (q >= nq) break;
                const double2 x = cmulc(vr, S[(warp + kEvWarps * q) * Mp + r]);
                ar[q] += x.x;
                ai[q] += x.y;
            }
        }
        double2 sc[CPW];
#pragma unroll
        for (int q = 0; q < CPW; ++q) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                ar[q] += __shfl_xor_sync(0xffffffffu, ar[q], o);
                ai[q] += __shfl_xor_sync(0xffffffffu, ai[q], o);
            }
            sc[q] = cmul(t, make_double2(ar[q], ai[q]));
        }
        for (int r = i + 1 + lane; r < M; r += 32) {
            const double2 vr = __ldg(v + r);
#pragma unroll
            for (int q = 0; q < CPW; ++q) {
                if (q >= nq) break;
                double2 *sp = S + (warp + kEvWarps * q) * Mp + r;
                const double2 u = cmul(vr, sc[q]);
                *sp = make_double2(sp->x - u.x, sp->y - u.y);
            }
        }
    }
    __syncthreads();
    double2 *V = Vall + (int64_t)b * M * ldv;   // row stride ldv (M, or the number of selected columns)
    for (int idx = tid; idx < M * W; idx += kEvThreads) {
        const int r = idx / W, j = idx % W;
        if (j < nw) V[(int64_t)r * ldv + c0 + j] = S[j * Mp + r];
    }
}

// The same for one selected column per CTA of one warp, M <= 32 NR: the column stays in registers (row lane + 32 q),
// and the reflectors stream through a ring of 8 rows in shared memory by cp.async, so that a reflector costs its two
// passes of FMAs and one warp sum instead of a round trip to L2 (735 -> 127 us for 16 matrices of 256 rows).
constexpr int kBackRing = 8;

template <int NR>
__global__ void __launch_bounds__(32) heevd_back_select_kernel(const double2 *__restrict__ vhall,
                                                               const double2 *__restrict__ tauall,
                                                               const double *__restrict__ Zall, int M, int E,
                                                               double2 *__restrict__ Vall)
{
    extern __shared__ double2 bk_sm[];   // [kBackRing][M]
    const int b = blockIdx.x, j = blockIdx.y, lane = threadIdx.x;
    const double2 *vh = vhall + (int64_t)b * (M > 1 ? M - 1 : 1) * M;
    const double2 *tau = tauall + (int64_t)b * M;
    const double *zc = Zall + (int64_t)b * M * M + (int64_t)j * M;
    auto fetch = [&](int i) {   // reflector i (entries i + 1 ..) into ring slot i % kBackRing
        if (i >= 0)
            for (int r = i + 1 + lane; r < M; r += 32) {
                const uint32_t dst = tc::smem_u32(bk_sm + (size_t)(i % kBackRing) * M + r);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(vh + (int64_t)i * M + r)
                             : "memory");
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int q = 0; q < kBackRing - 1; ++q) fetch(M - 2 - q);
    double2 x[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        const int r = lane + 32 * q;
        x[q] = make_double2(r < M ? zc[r] : 0.0, 0.0);
    }
    double2 tn = M > 1 ? __ldg(tau + M - 2) : make_double2(0.0, 0.0);
    for (int i = M - 2; i >= 0; --i) {
        const double2 t = tn;
        tn = __ldg(tau + max(i - 1, 0));
        asm volatile("cp.async.wait_group %0;" ::"n"(kBackRing - 2) : "memory");
        __syncwarp();   // every lane's part of reflector i has landed, and reflector i + 1 is read
        fetch(i - (kBackRing - 1));
        const double2 *v = bk_sm + (size_t)(i % kBackRing) * M;
        double2 u[NR];
        double ar = 0.0, ai = 0.0;
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            const int r = lane + 32 * q;
            u[q] = r > i && r < M ? v[r] : make_double2(0.0, 0.0);
            const double2 c = cmulc(u[q], x[q]);
            ar += c.x;
            ai += c.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ar += __shfl_xor_sync(0xffffffffu, ar, o);
            ai += __shfl_xor_sync(0xffffffffu, ai, o);
        }
        const double2 sc = cmul(t, make_double2(ar, ai));
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            const double2 c = cmul(u[q], sc);
            x[q] = make_double2(x[q].x - c.x, x[q].y - c.y);
        }
    }
    double2 *V = Vall + (int64_t)b * M * E + j;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        const int r = lane + 32 * q;
        if (r < M) V[(int64_t)r * E] = x[q];
    }
}

// ------------------------------------------------------------------------------------------------
// Selected eigenpairs (acb_heevd_select_f64): the eigenvalues of chosen ranks and their eigenvectors
// only, for consumers that use a few components (BeamformerEig's default n = -1 takes the largest).
// After the same tridiagonalisation, one warp per selected rank k:
//   - the k-th smallest eigenvalue of T by multisection: each round the 32 lanes evaluate the Sturm
//     count (the number of sign changes of the leading minors of T - x I, i.e. of eigenvalues
//     below x) at 32 points spread over the current interval, which then narrows to the gap between two
//     neighbouring points (about 33x per round, from the Gershgorin interval down to 2 eps |lambda|, or
//     eps ||T|| for eigenvalues near zero, the accuracy of the QL iteration);
//   - its eigenvector by inverse iteration: T - lambda I factored once by Gaussian elimination with
//     partial pivoting (a tridiagonal factor gains one superdiagonal of fill-in), then three solves from
//     a fixed start vector, each rescaled by its largest entry; zero pivots are replaced by eps ||T||;
//   - the back-transformation by the reflectors (heevd_back_kernel on the selected columns).
// The QL sweeps and their accumulation of all M eigenvectors are skipped.
// ------------------------------------------------------------------------------------------------
constexpr int kSelMax = 4;

struct EvSel {
    int n;
    int idx[kSelMax];
};

// Number of eigenvalues of T below x: the sign changes of the leading principal minors of T - x I,
// p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2} (one FMA on the serial path; the pivots' ratios would need a division),
// with T scaled by the power of two `sc` to a norm of about 1 (e2: squares of the scaled off-diagonal) and the pair
// rescaled every 8 steps.  A minor that vanishes is replaced by -1e-30 times the one before (a shift of d_i by 1e-30).
__device__ __forceinline__ int ev_sturm(const double *d, const double *e2, int M, double x, double sc)
{
    double p1 = (d[0] - x) * sc, p0 = 1.0;
    if (p1 == 0.0) p1 = -1e-30;
    int cnt = p1 < 0.0;
    for (int i0 = 1; i0 < M; i0 += 8) {
        double a[8], q[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = min(i0 + u, M - 1);
            a[u] = (d[i] - x) * sc;
            q[u] = e2[i - 1];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (i0 + u >= M) break;
            double p = fma(a[u], p1, -(q[u] * p0));
            if (p == 0.0) p = -1e-30 * p1;
            cnt += (p < 0.0) != (p1 < 0.0);
            p0 = p1;
            p1 = p;
        }
        // exact power of two that brings the larger of the two to [1, 2)
        const int ex = ilogb(fmax(fabs(p0), fabs(p1)));
        p0 = scalbn(p0, -ex);
        p1 = scalbn(p1, -ex);
    }
    return cnt;
}

__host__ __device__ constexpr size_t ev_select_smem(int M, int E)
{
    return ((size_t)3 * M + (size_t)5 * M * E) * sizeof(double) + (size_t)M * E;
}

__global__ void __launch_bounds__(32 * kSelMax) heevd_select_kernel(const double *__restrict__ dall,
                                                                    const double *__restrict__ eall, int M,
                                                                    EvSel sel, double *__restrict__ wsel,
                                                                    double *__restrict__ Zall,
                                                                    int *__restrict__ permall)
{
    extern __shared__ double sl_sm[];
    double *d = sl_sm;           // [M]
    double *e = sl_sm + M;       // [M] off-diagonal (e[M - 1] = 0)
    double *e2 = sl_sm + 2 * M;  // [M] its squares
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    double *u0 = sl_sm + 3 * M + (size_t)w * 5 * M;   // pivots (as reciprocals after the factorisation)
    double *u1 = u0 + M;                              // first superdiagonal of U
    double *u2 = u1 + M;                              // second superdiagonal (fill-in)
    double *mu = u2 + M;                              // multipliers
    double *y = mu + M;                               // iterate
    unsigned char *pv = reinterpret_cast<unsigned char *>(sl_sm + 3 * M + (size_t)sel.n * 5 * M) + (size_t)w * M;
    for (int i = tid; i < M; i += blockDim.x) {
        d[i] = dall[(int64_t)b * M + i];
        const double ei = i < M - 1 ? eall[(int64_t)b * M + i] : 0.0;
        e[i] = ei;
    }
    __syncthreads();
    const double eps = 2.220446049250313e-16;
    // Gershgorin interval, the norm of T and the pivot floor
    double lo = INFINITY, hi = -INFINITY, emax2 = 0.0;
    for (int i = lane; i < M; i += 32) {
        const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + fabs(e[i]);
        lo = fmin(lo, d[i] - r);
        hi = fmax(hi, d[i] + r);
        emax2 = fmax(emax2, e[i] * e[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        emax2 = fmax(emax2, __shfl_xor_sync(0xffffffffu, emax2, o));
    }
    double *zc = Zall + (int64_t)b * M * M + (int64_t)w * M;   // column w of Z
    if (lane == 0) permall[(int64_t)b * M + w] = w;
    const double pivmin = 2.2250738585072014e-308 * fmax(1.0, emax2);
    const double tnorm = fmax(fabs(lo), fabs(hi));
    const double fudge = 2.0 * eps * tnorm + 2.0 * pivmin;
    lo -= fudge;
    hi += fudge;
    const int k = sel.idx[w];
    // the scaled squares, by all ranks' warps together (each has formed the same norm from T)
    const double tsc = tnorm > 0.0 ? scalbn(1.0, -ilogb(tnorm)) : 1.0;
    for (int i = tid; i < M; i += blockDim.x) e2[i] = (e[i] * tsc) * (e[i] * tsc);
    __syncthreads();
    for (int it = 0; it < 64; ++it) {
        const double width = hi - lo;
        if (width <= fmax(2.0 * eps * fmax(fabs(lo), fabs(hi)), eps * tnorm) || width <= 4.0 * pivmin) break;
        const double x = lo + width * (double)(lane + 1) / 33.0;
        const int c = ev_sturm(d, e2, M, x, tsc);
        const unsigned bal = __ballot_sync(0xffffffffu, c > k);   // points above the k-th eigenvalue
        const double x31 = __shfl_sync(0xffffffffu, x, 31);
        if (bal == 0) {
            lo = x31;
        } else {
            const int j0 = __ffs(bal) - 1;
            const double xh = __shfl_sync(0xffffffffu, x, j0);
            const double xl = __shfl_sync(0xffffffffu, x, j0 > 0 ? j0 - 1 : 0);
            if (j0 > 0) lo = xl;
            hi = xh;
        }
    }
    // a NaN in T, which fmin, fmax and the counts pass over: no result.  lam is NaN then, and through the solves its
    // vector (looked for ahead of the counts, with or without an early return, it made the kernel 7 % slower)
    bool bad = false;
    for (int i = lane; i < M; i += 32) bad |= d[i] != d[i] || e[i] != e[i];
    const double lam = __any_sync(0xffffffffu, bad) ? __longlong_as_double(0x7ff8000000000000ll) : 0.5 * (lo + hi);
    if (lane == 0) {
        wsel[(int64_t)b * sel.n + w] = lam;
        const double tiny = tnorm > 0.0 ? eps * tnorm : 2.2250738585072014e-308;
        // T - lam I = P L U
        double a = d[0] - lam, bs = M > 1 ? e[0] : 0.0;
        for (int i = 0; i < M - 1; ++i) {
            const double l = e[i], m = d[i + 1] - lam, n = i + 2 < M ? e[i + 1] : 0.0;
            if (fabs(a) >= fabs(l)) {
                if (fabs(a) < tiny) a = a < 0.0 ? -tiny : tiny;
                const double f = l / a;
                pv[i] = 0;
                u0[i] = a;
                u1[i] = bs;
                u2[i] = 0.0;
                mu[i] = f;
                a = m - f * bs;
                bs = n;
            } else {
                const double f = a / l;
                pv[i] = 1;
                u0[i] = l;
                u1[i] = m;
                u2[i] = n;
                mu[i] = f;
                a = bs - f * m;
                bs = -f * n;
            }
        }
        if (fabs(a) < tiny) a = a < 0.0 ? -tiny : tiny;
        u0[M - 1] = a;
    }
    __syncwarp();
    for (int i = lane; i < M; i += 32) {
        u0[i] = 1.0 / u0[i];
        y[i] = 1.0 + 0.25 * (double)((i * 2654435761u) % 1009u) / 1009.0;
    }
    for (int it = 0; it < 3; ++it) {
        __syncwarp();
        if (lane == 0) {
            // the two recurrences, each step's operands read before the step before stores
            double cur = y[0], nx = M > 1 ? y[1] : 0.0, f = mu[0];
            bool sw = M > 1 && pv[0];
            for (int i = 0; i < M - 1; ++i) {
                const int j = min(i + 2, M - 1), k1 = min(i + 1, M - 2);
                const double nx2 = y[j], f2 = mu[k1];
                const bool sw2 = pv[k1];
                y[i] = sw ? nx : cur;
                cur = sw ? fma(-f, nx, cur) : fma(-f, cur, nx);
                nx = nx2;
                f = f2;
                sw = sw2;
            }
            double y1 = cur * u0[M - 1], y2 = 0.0;   // y[i + 1], y[i + 2]
            y[M - 1] = y1;
            int i = M - 2;
            double r = y[max(i, 0)], b1 = u1[max(i, 0)], b2 = M > 2 ? u2[max(i, 0)] : 0.0, b0 = u0[max(i, 0)];
            for (; i >= 0; --i) {
                const int j = max(i - 1, 0);
                const double rn = y[j], b1n = u1[j], b2n = u2[j], b0n = u0[j];
                const double yi = fma(-b1, y1, fma(-b2, y2, r)) * b0;
                y[i] = yi;
                y2 = y1;
                y1 = yi;
                r = rn;
                b1 = b1n;
                b2 = b2n;
                b0 = b0n;
            }
        }
        __syncwarp();
        double mx = 0.0;
        for (int i = lane; i < M; i += 32) mx = fmax(mx, fabs(y[i]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const double sc = mx > 0.0 ? 1.0 / mx : 1.0;
        for (int i = lane; i < M; i += 32) y[i] *= sc;
    }
    __syncwarp();
    double ss = 0.0;
    for (int i = lane; i < M; i += 32) ss += y[i] * y[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const double inv = ss > 0.0 ? 1.0 / sqrt(ss) : 0.0;
    for (int i = lane; i < M; i += 32) zc[i] = y[i] * inv;
}

struct EvWorkspace {
    size_t A, d, e, tau, vh, Z, perm, total;
};

static EvWorkspace ev_layout(int M, int B)
{
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    EvWorkspace w;
    size_t off = 0;
    w.A = off;
    off += up((size_t)B * M * M * sizeof(double2));
    w.d = off;
    off += up((size_t)B * M * sizeof(double));
    w.e = off;
    off += up((size_t)B * M * sizeof(double));
    w.tau = off;
    off += up((size_t)B * M * sizeof(double2));
    w.vh = off;
    off += up((size_t)B * (M > 1 ? M - 1 : 1) * M * sizeof(double2));
    w.Z = off;
    off += up((size_t)B * M * M * sizeof(double));
    w.perm = off;
    off += up((size_t)B * M * sizeof(int));
    w.total = off;
    return w;
}

// CTAs per matrix of the cluster form, 0 if the matrix does not fit eight: the fewest that hold it.
static size_t ev_cluster_smem(int M, int C)
{
    const int nl = (M + C - 1) / C;   // vectors, then rank C - 1's rows, the longest
    return ((size_t)M * (4 + C + kEvWarps) + nl + ev_packed(C - 1, C, nl)) * sizeof(double2);
}

static int ev_cluster_ctas(int M)
{
    for (int C = 1; C <= 8; C *= 2)
        if (ev_cluster_smem(M, C) <= 225 * 1024) return C;
    return 0;
}

// Tridiagonalisation of B matrices: the cluster form where it fits, else a working copy and the global-memory form.
static int tridiag_launch(const void *csm, int B, int M, double2 *A, double *d, double *e, double2 *tau, double2 *vh,
                          cudaStream_t s)
{
    // many small matrices: the CTAs of the global-memory form are resident together and hide each other's latency
    // (select of 500 matrices of 32 rows 0.27 against 0.33 ms; 20 of them 0.22 against 0.19; 513 of 64 rows equal)
    const int C = M < 48 && B > 2 * kNumSMs ? 0 : ev_cluster_ctas(M);
    if (C > 0) {
        const size_t smem = ev_cluster_smem(M, C);
        // two CTAs per SM where their memory fits: then with 128 registers (some spilled), else with all it needs
        auto kern = smem <= 110 * 1024 ? heevd_tridiag_cluster_kernel<2> : heevd_tridiag_cluster_kernel<1>;
        if (const int st = allow_smem(kern, smem, (smem <= 110 * 1024 ? 110 : 225) * 1024)) return st;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(B * C));
        cfg.blockDim = dim3(kEvThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)C;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaLaunchKernelEx(&cfg, kern, static_cast<const double2 *>(csm), M, d, e, tau, vh, tc_wait_limit_ns()) !=
            cudaSuccess)
            return ACB_ERR_CUDA;
        return check_launch();
    }
    const cudaError_t err = cudaMemcpyAsync(A, csm, (size_t)B * M * M * sizeof(double2), cudaMemcpyDeviceToDevice, s);
    if (err != cudaSuccess) {
        set_cuda_error(err);
        return ACB_ERR_CUDA;
    }
    const size_t smem = 2 * (size_t)M * sizeof(double2);
    if (const int st = allow_smem(heevd_tridiag_kernel, smem, 2 * kEvMaxRows * sizeof(double2))) return st;
    heevd_tridiag_kernel<<<B, kEvThreads, smem, s>>>(A, M, d, e, tau, vh);
    return check_launch();
}

// Columns per back-transformation slab: as many as fit beside the reflector in the shared memory (<= 32).
static int ev_slab(int M)
{
    int W = 32;
    while (W > 1 && (size_t)(M + 1) * W * sizeof(double2) > 200 * 1024) W >>= 1;
    return W;
}

}  // namespace acb

using namespace acb;

extern "C" {

size_t acb_heevd_workspace_bytes(int num_mics, int num_bins)
{
    if (num_mics < 1 || num_bins < 1) return 0;
    return ev_layout(num_mics, num_bins).total;
}

int acb_heevd_f64(const void *csm, int num_bins, int num_mics, double *eigval, void *eigvec, int *info,
                  void *workspace, size_t workspace_bytes, void *stream)
{
    if (!csm || !eigval || !eigvec || !workspace) return ACB_ERR_ARG;
    const int M = num_mics, B = num_bins;
    if (M < 1 || B < 1 || M > kEvMaxRows || B > 65535) return ACB_ERR_SHAPE;
    const EvWorkspace lay = ev_layout(M, B);
    if (workspace_bytes < lay.total) return ACB_ERR_WORKSPACE;
    const int W = ev_slab(M);
    if ((size_t)(M + 1) * W * sizeof(double2) > 200 * 1024) return ACB_ERR_UNSUPPORTED;
    cudaStream_t s = as_stream(stream);
    char *ws = static_cast<char *>(workspace);
    double2 *A = reinterpret_cast<double2 *>(ws + lay.A);
    double *d = reinterpret_cast<double *>(ws + lay.d);
    double *e = reinterpret_cast<double *>(ws + lay.e);
    double2 *tau = reinterpret_cast<double2 *>(ws + lay.tau);
    double2 *vh = reinterpret_cast<double2 *>(ws + lay.vh);
    double *Z = reinterpret_cast<double *>(ws + lay.Z);
    int *perm = reinterpret_cast<int *>(ws + lay.perm);
    const size_t sm2 = 6 * (size_t)M * sizeof(double);
    int st = allow_smem(heevd_tql_kernel, sm2, 6 * kEvMaxRows * sizeof(double));
    if (st) return st;
    st = tridiag_launch(csm, B, M, A, d, e, tau, vh, s);
    if (st) return st;
    heevd_tql_kernel<<<B, kQlThreads, sm2, s>>>(d, e, M, eigval, Z, perm, info);
    st = check_launch();
    if (st) return st;
    const size_t smem = (size_t)(M + 1) * W * sizeof(double2);
    // columns per warp: the slab's W columns over the 8 warps
    auto back = W >= 32 ? heevd_back_kernel<4> : (W >= 16 ? heevd_back_kernel<2> : heevd_back_kernel<1>);
    st = allow_smem(back, smem, 200 * 1024);
    if (st) return st;
    back<<<dim3(B, (M + W - 1) / W), kEvThreads, smem, s>>>(vh, tau, Z, perm, M, W, M,
                                                           static_cast<double2 *>(eigvec));
    return check_launch();
}

int acb_heevd_select_f64(const void *csm, int num_bins, int num_mics, int num_sel, const int *sel, double *eigval,
                         void *eigvec, void *workspace, size_t workspace_bytes, void *stream)
{
    if (!csm || !sel || !eigval || !eigvec || !workspace) return ACB_ERR_ARG;
    const int M = num_mics, B = num_bins, E = num_sel;
    if (M < 1 || B < 1 || M > kEvMaxRows || B > 65535 || E < 1 || E > kSelMax || E > M) return ACB_ERR_SHAPE;
    EvSel es;
    es.n = E;
    for (int j = 0; j < kSelMax; ++j) es.idx[j] = 0;
    for (int j = 0; j < E; ++j) {
        if (sel[j] < 0 || sel[j] >= M) return ACB_ERR_ARG;
        es.idx[j] = sel[j];
    }
    const size_t sm3 = ev_select_smem(M, E);
    if (sm3 > 200 * 1024) return ACB_ERR_UNSUPPORTED;
    const EvWorkspace lay = ev_layout(M, B);
    if (workspace_bytes < lay.total) return ACB_ERR_WORKSPACE;
    cudaStream_t s = as_stream(stream);
    char *ws = static_cast<char *>(workspace);
    double2 *A = reinterpret_cast<double2 *>(ws + lay.A);
    double *d = reinterpret_cast<double *>(ws + lay.d);
    double *e = reinterpret_cast<double *>(ws + lay.e);
    double2 *tau = reinterpret_cast<double2 *>(ws + lay.tau);
    double2 *vh = reinterpret_cast<double2 *>(ws + lay.vh);
    double *Z = reinterpret_cast<double *>(ws + lay.Z);
    int *perm = reinterpret_cast<int *>(ws + lay.perm);
    int st = allow_smem(heevd_select_kernel, sm3, 200 * 1024);
    if (st) return st;
    st = tridiag_launch(csm, B, M, A, d, e, tau, vh, s);
    if (st) return st;
    heevd_select_kernel<<<B, 32 * E, sm3, s>>>(d, e, M, es, eigval, Z, perm);
    st = check_launch();
    if (st) return st;
    if (M <= 512) {   // registers for the column, 8 reflectors in shared memory
        const size_t ring = (size_t)kBackRing * M * sizeof(double2);
        auto back = M <= 64 ? heevd_back_select_kernel<2>
                            : (M <= 128 ? heevd_back_select_kernel<4>
                                        : (M <= 256 ? heevd_back_select_kernel<8> : heevd_back_select_kernel<16>));
        st = allow_smem(back, ring, kBackRing * 512 * sizeof(double2));
        if (st) return st;
        back<<<dim3(B, E), 32, ring, s>>>(vh, tau, Z, M, E, static_cast<double2 *>(eigvec));
        return check_launch();
    }
    // the E eigenvectors of T sit in columns 0 .. E-1 of each matrix's Z, perm[j] = j: one slab of E columns
    const size_t smem = (size_t)(M + 1) * E * sizeof(double2);
    st = allow_smem(heevd_back_kernel<1>, smem, 200 * 1024);
    if (st) return st;
    heevd_back_kernel<1><<<dim3(B, 1), kEvThreads, smem, s>>>(vh, tau, Z, perm, M, E, E,
                                                              static_cast<double2 *>(eigvec));
    return check_launch();
}

}  // extern "C"
