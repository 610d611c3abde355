// Shared helpers for the acoular_b200 CUDA kernels (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/acoular_b200.h"

namespace acb {

// Record the last CUDA error text for acb_last_cuda_error().
void set_cuda_error(cudaError_t e);

// Limit of one bounded device-side wait of the tensor-core kernels and of the exchanges inside a cluster
// (acb_tc_set_wait_limit_ns).
uint64_t tc_wait_limit_ns();

inline int check_launch()
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_cuda_error(e);
        return ACB_ERR_CUDA;
    }
    return ACB_OK;
}

constexpr int kSmemMost = 227 * 1024;   // of a CTA on sm_100a, static and dynamic

// Let `kern` be launched with `bytes` of dynamic shared memory; `most` is the largest that any call asks for.  The limit
// belongs to the function, not to the call, so every call sets the same one: with each call's own size another thread's
// call could lower it between this call's setting and its launch, which then fails.
template <class... Args>
inline int allow_smem(void (*kern)(Args...), size_t bytes, size_t most)
{
    cudaError_t e = bytes > most ? cudaErrorInvalidValue
                                 : cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e == cudaSuccess) return ACB_OK;
    cudaGetLastError();   // reported here, not by the next launch
    set_cuda_error(e);
    return ACB_ERR_CUDA;
}

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

constexpr int kNumSMs = 148;

// Distance |g - m| with the contraction order the reference's fastmath dist_mat compiles to:
// sqrt(fma(d2, d2, fma(d1, d1, d0 * d0))) (acoular/environments.py:65-103).
__device__ __forceinline__ double dist3(double g0, double g1, double g2, double m0, double m1, double m2)
{
    const double d0 = __dsub_rn(g0, m0);
    const double d1 = __dsub_rn(g1, m1);
    const double d2 = __dsub_rn(g2, m2);
    return __dsqrt_rn(__fma_rn(d2, d2, __fma_rn(d1, d1, __dmul_rn(d0, d0))));
}

// D (16 x 8) += A (16 x 8) B (8 x 8), FP64.  Lane (g = lane / 4, t = lane % 4) holds A rows g, g + 8 at columns
// t, t + 4 (a0: g,t  a1: g+8,t  a2: g,t+4  a3: g+8,t+4), B rows t, t + 4 of column g, and D rows g, g + 8 at
// columns 2t, 2t + 1.  The products of one element are added as a chain of FMAs.
__device__ __forceinline__ void mma_f64(double (&d)[4], double a0, double a1, double a2, double a3, double b0,
                                        double b1)
{
    asm(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64.rn {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// Exception table of the host C library's float32 cosf/sinf (built by acb_sincos_table_build_host): open
// addressing, linear probing.  Entry layout: bits 63..32 = float bits of x, bits 31..16 = tags of the slot (below),
// bits 15..8 = int8 ulp delta of cos, bits 7..0 = int8 ulp delta of sin; an all-ones word marks an empty slot.
// Two things keep the lookups (random 32-byte sectors of a 64 MB table) few and short:
//   tol   An exception can only occur where the FP64 value lies within tol units (of 2^-29 float32 ulp) of the
//         midpoint of two float32 values: the table holds, under kSincosMetaKey, the largest distance of any of its
//         entries (0.0607 ulp for glibc 2.39), so three arguments in four are never looked up.  tol < 0: no table.
//   tags  Bit 16 + tag of a slot's word is set for every key with this home slot (whoever occupies it), tag = 4
//         other bits of the key's hash: unless the bit is set, one load answers the lookup, with no walk.
// A table without the meta entry has no tags: tol is then half an ulp and every occupied home slot is walked.
// Bound: issue slots.  Instructions per value, the caller's own work included: 108 in psf_kernel, 152 in
// map_eig_small_kernel (23 and 33 of them FP64).  Measured (B200; before: a lookup and its walk for every value and the
// library's sincos, 194 instructions): map of one eigen-component, 16 bins x 160,801 points x 256 mics, 7.9 -> 5.1 ms;
// point-spread function 1681 x 1681 x 64 mics 1.72 -> 1.03 ms (3.7 and 0.48 with what those kernels changed since).
struct SincosTable {
    const uint64_t *table;
    uint64_t mask;
    int tol;
    uint32_t untagged;   // all tag bits if the table has none
};

constexpr uint32_t kSincosMetaKey = 0xfffffffeu;   // sign bit set: never the magnitude of an argument
__host__ __device__ constexpr uint64_t sincos_hash(uint32_t key)
{
    return static_cast<uint64_t>(key) * 0x9E3779B97F4A7C15ull;   // home slot: bits 20 and up; tag: bits 60..63
}

__device__ __forceinline__ SincosTable sincos_table(const uint64_t *table, uint64_t mask, bool faithful)
{
    SincosTable t{table, mask, -1, 0u};
    if (faithful) {
        const uint64_t e = __ldg(table + ((sincos_hash(kSincosMetaKey) >> 20) & mask));
        const bool meta = static_cast<uint32_t>(e >> 32) == kSincosMetaKey;
        t.tol = meta ? static_cast<int>((static_cast<uint32_t>(e) & 0xffffu) << 13) : 0x10000000;
        t.untagged = meta ? 0u : 0xffff0000u;
    }
    return t;
}

// Walk the table for float32 argument magnitude `x`.
__device__ __forceinline__ void sincos_exception(const SincosTable &t, float x, int &dcos, int &dsin)
{
    const uint32_t key = __float_as_uint(x);
    uint64_t slot = sincos_hash(key) >> 20;
    dcos = 0;
    dsin = 0;
    for (int probe = 0; probe < 64; ++probe) {  // bounded: the table is built at < 50 % load
        const uint64_t e = __ldg(t.table + (slot & t.mask));
        if (e == ~0ull) return;
        if (static_cast<uint32_t>(e >> 32) == key) {
            dcos = static_cast<int8_t>((e >> 8) & 0xff);
            dsin = static_cast<int8_t>(e & 0xff);
            return;
        }
        ++slot;
    }
}

static __device__ const double2 kSincosPoints[64] = {
#include "sincos_points.inc"
};

// The general FP64 sincos, out of line: only arguments beyond the table-driven range come here.
static __device__ __noinline__ void sincos_any(double x, double *s, double *c) { sincos(x, s, c); }

// FP64 cos/sin of a float32 argument, table driven (the scheme of P. T. P. Tang, Table-lookup algorithms for
// elementary functions, 1991): x = n pi/32 + r with |r| <= pi/64, pi/32 split in a part of 38 bits (n times it is
// exact for n < 2^15) and its remainder; cos/sin of n pi/32 from the table, those of r from their Taylor series
// (next terms 2e-20 and 4e-18), combined as C + (C (cos r - 1) - S sin r).  About one FP64 ulp; results near zero
// (C = 0 exactly) keep the relative accuracy of r.  17 FP64 operations, no branch but the range check.
__device__ __forceinline__ void sincos_small(float x, double &c, double &s)   // |x| < 3000
{
    const double xd = static_cast<double>(x);
    const double magic = 6755399441055744.0;   // 1.5 2^52: the addition rounds to an integer
    const double t = fma(xd, 0x1.45f306dc9c883p+3, magic);
    const double nd = t - magic;
    const double2 p = __ldg(kSincosPoints + (__double2loint(t) & 63));
    double r = fma(-nd, 0x1.921fb54440000p-4, xd);
    r = fma(-nd, 0x1.68c234c4c6629p-43, r);
    const double r2 = r * r;
    const double cm = r2 * fma(r2, fma(r2, fma(r2, 1.0 / 40320.0, -1.0 / 720.0), 1.0 / 24.0), -0.5);
    const double sr = fma(r * r2, fma(r2, fma(r2, -1.0 / 5040.0, 1.0 / 120.0), -1.0 / 6.0), r);
    c = fma(p.x, cm, fma(-p.y, sr, p.x));
    s = fma(p.y, cm, fma(p.x, sr, p.y));
}

// Float32 cos/sin of float32 arguments: correctly rounded value through FP64 evaluation,
// optionally corrected to the host C library's cosf/sinf by the exception table.  The table holds
// non-negative arguments; a negative one is looked up by its magnitude (the C library's cosf is even
// and its sinf odd, bit for bit, and a delta on the bits of a float changes its magnitude).
// K arguments at a time, in two halves, so that their loads are in flight together: begin evaluates and loads the home
// slots' words, finish corrects (about one lane in 150 walks the table).  Issue slots bound the callers: the range
// test and the test for a walk are one branch for all K, and the lookups are predicated loads, no branches.
// Measured (B200; before: a branch per argument for each): FP64 map of 256 mics x 160,801 points x 12 bins 20.9 -> 20.4
// ms, DAMAS of 64 mics 9.74 -> 9.63 ms.
template <int K>
struct SincosPending {
    float x[K], c[K], s[K];
    uint64_t word[K];   // the home slot's word, all ones where no lookup is needed
};

// Load of a word where `p` holds, all ones elsewhere.
__device__ __forceinline__ uint64_t sincos_word(const uint64_t *at, bool p)
{
    uint64_t w;
    asm("{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %2, 0;\n\t"
        "mov.b64 %0, -1;\n\t"
        "@q ld.global.nc.b64 %0, [%1];\n\t}"
        : "=&l"(w)
        : "l"(at), "r"((int)p));
    return w;
}

template <int K>
__device__ __forceinline__ void sincos_begin(SincosPending<K> &v, const SincosTable &t)
{
    double sd[K], cd[K];
    uint32_t big = 0;
#pragma unroll
    for (int q = 0; q < K; ++q) big = max(big, __float_as_uint(fabsf(v.x[q])));
    if (big < 0x453b8000u) {   // 3000.0f; infinities and NaN compare above
#pragma unroll
        for (int q = 0; q < K; ++q) sincos_small(v.x[q], cd[q], sd[q]);
    } else {
#pragma unroll
        for (int q = 0; q < K; ++q) {
            if (fabsf(v.x[q]) < 3000.0f) sincos_small(v.x[q], cd[q], sd[q]);
            else sincos_any(static_cast<double>(v.x[q]), &sd[q], &cd[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < K; ++q) {
        v.c[q] = __double2float_rn(cd[q]);
        v.s[q] = __double2float_rn(sd[q]);
        // distance of the FP64 values from a float32 rounding midpoint, from their 29 low mantissa bits
        const int mc = abs((__double2loint(cd[q]) & 0x1fffffff) - 0x10000000);
        const int ms = abs((__double2loint(sd[q]) & 0x1fffffff) - 0x10000000);
        v.word[q] = sincos_word(t.table + ((sincos_hash(__float_as_uint(fabsf(v.x[q]))) >> 20) & t.mask),
                                min(mc, ms) <= t.tol);
    }
}

template <int K>
__device__ __forceinline__ void sincos_finish(SincosPending<K> &v, const SincosTable &t)
{
    bool walk[K], any = false;
#pragma unroll
    for (int q = 0; q < K; ++q) {
        const uint32_t tag = 16u + static_cast<uint32_t>(sincos_hash(__float_as_uint(fabsf(v.x[q]))) >> 60);
        walk[q] = v.word[q] != ~0ull && (((static_cast<uint32_t>(v.word[q]) | t.untagged) >> tag) & 1u);
        any |= walk[q];
    }
    if (!any) return;
#pragma unroll
    for (int q = 0; q < K; ++q) {
        if (!walk[q]) continue;
        int dc, ds;
        sincos_exception(t, fabsf(v.x[q]), dc, ds);
        if (dc) v.c[q] = __int_as_float(__float_as_int(v.c[q]) + dc);
        if (ds) v.s[q] = __int_as_float(__float_as_int(v.s[q]) + ds);
    }
}

__device__ __forceinline__ void sincos_f32_arg(float x, const SincosTable &t, float &c, float &s)
{
    SincosPending<1> v;
    v.x[0] = x;
    sincos_begin(v, t);
    sincos_finish(v, t);
    c = v.c[0];
    s = v.s[0];
}

}  // namespace acb
