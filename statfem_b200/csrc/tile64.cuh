// FP64 building blocks of the dense and block eliminations: the matrix
// instruction, the reciprocal and the inverse of a 32 x 32 block.
#pragma once

namespace sfc {
namespace {

// D (8 x 8) += A (8 x 4) B (4 x 8): lane l holds A[l / 4][l % 4], B[l % 4][l / 4], D[l / 4][2 (l % 4) + 0, 1]
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// The range of recip: d positive and below 2^1022, d and 1 / d normal numbers,
// by the exponent (as FP64 comparisons a block elimination took 4 % longer)
__device__ __forceinline__ bool recip_takes(double d)
{
    return (unsigned)__double2hiint(d) - 0x00100000u < 0x7fc00000u;
}

// 1 / d by Newton's iteration on the hardware's approximation (about 20 bits;
// two steps reach rounding), which flushes subnormal numbers, its own result
// among them, to zero: outside its range the result is no reciprocal.  No
// branch, so that other work fits into its latency.
__device__ __forceinline__ double recip(double d)
{
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
    x = fma(x, fma(-d, x, 1.0), x);
    return fma(x, fma(-d, x, 1.0), x);
}

// The sweep that inverts a symmetric block of up to 32 columns, by the first
// four warps of the CTA: warp w holds rows 8 w .. 8 w + 7 in v, lane j column
// j, identity past the block; `steps` pivots, a multiple of eight.  The result
// is the negative inverse.  The symmetric form makes the pivot column equal to
// the pivot row, so a step exchanges one row through buf (2 x 32); the next
// row is updated and published before the rest of a step, which runs inside
// the next pivot's latency.  pivot(k, d, inv): false drops pivot k (its row
// and column become zero), else inv = 1 / d.  32 columns 2.9 us; 7.0 with 256
// threads, a division and a full barrier per step, 6.9 with one warp (its 31
// updates per step bound it).
template <class F>
__device__ __forceinline__ void sweep_inverse(double (&v)[8], int steps, double *buf, F &&pivot)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) buf[lane] = v[0];
    asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll 1
    for (int b = 0; 8 * b < steps; ++b) {
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const int k = 8 * b + t, t1 = (t + 1) & 7;
            const bool own = warp == b, next = warp == (t == 7 ? b + 1 : b);
            const double *sh = buf + 32 * (t & 1);
            double *nx = buf + 32 * (t1 & 1);
            double row[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) row[i] = sh[8 * warp + i];
            const double mine = sh[lane];
            double inv = 0.0;
            const bool drop = !pivot(k, sh[k], inv), me = lane == k;
            const double f = me ? inv : drop ? 0.0 : -mine * inv;
            if (next) {
                v[t1] = drop ? (me ? 0.0 : v[t1]) : fma(row[t1], f, me ? 0.0 : v[t1]);
                nx[lane] = v[t1];
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (next && i == t1) continue;
                if (own && i == t) v[i] = me ? -inv : -f;
                else v[i] = drop ? (me ? 0.0 : v[i]) : fma(row[i], f, me ? 0.0 : v[i]);
            }
        }
    }
}

}  // namespace
}  // namespace sfc
