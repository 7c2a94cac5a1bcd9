// FP64 PCG for one right-hand side as one persistent cooperative kernel, and
// the diagonal (DIA) copy of the operator that its product reads.
//
// The iteration of the plain method (point Jacobi) and of the two-level
// preconditioner (coarse.cu) on S x = b, with the scalars of every iteration
// in their own slots, as separate launches cost five launches and 26 us an
// iteration on small meshes, whatever their work.  Here the phases of an
// iteration (product with p.q; x, r update with the dots and the coarse
// restriction; coarse product; p update) follow one another behind grid
// barriers of a cooperative launch (co-resident blocks by construction; every
// wait has a limit, after which the kernel reports a timeout).
//
// On meshes numbered along a lattice every row couples to the same offsets,
// so the values are also kept by diagonals, [offset][row] ([offset][3 x 3]
// [node] on 3-dof meshes): a warp reads 32 consecutive rows of a diagonal in
// one piece and no column indices.  Only the diagonals above and on the main
// one are kept (the operator is symmetric, which is checked): the entry below
// is read from the row above it, and the copy is a third of the CSR's bytes,
// so that it stays in L2 between iterations up to about a million rows (80^3
// Poisson: 60 MB against 172; all 27 diagonals, 115 MB, took 27 us a product,
// the CSR 79).

#include <algorithm>
#include <cmath>
#include <vector>

#include "pcg.cuh"

namespace sfc {
namespace {

// Nonzeros up to which one cluster of 16 blocks runs the solve.  An iteration
// takes it 10.3 us at 29 thousand (64 x 64 square; the grid 11.7) and 19.5 at
// 230 thousand (181 x 181; the grid 13).
constexpr double kClusterWork = 1e5;
// The same for rows of indices (renumbered squares, us: 57 thousand 14.9, the
// grid 8.8; 26 thousand 9.6), and from where those of 16 lanes go as launches,
// shorter ones from twice as many (renumbered cubes: 0.77 million 16.4, as
// launches 18; 2.5 million 32.5 and 28.5; 13.8 million 148 and 111; squares of
// 2.5 million 31 and 38)
constexpr double kClusterRows = 4e4, kLaunchRows = 2e6;

enum { PQ, RZ, RR, CE, SUMS };  // p.q, r.z (the smoother's share), r.r, c.e

// Adds the M values of the warp's lanes to c[M agg ..]: lanes of consecutive
// nodes of one aggregate (a run of the lattice's line) are summed first.
template <int M>
__device__ void restrict_add(double *c, int agg, double (&v)[M])
{
    const int lane = threadIdx.x & 31;
    const int left = __shfl_up_sync(0xffffffffu, agg, 1);
    const bool head = lane == 0 || left != agg;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const unsigned after = lane == 31 ? 0u : heads >> (lane + 1);
    const int run = after ? __ffs(after) : 32 - lane;  // lanes to the end of the run
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const double w = __shfl_down_sync(0xffffffffu, v[m], o);
            if (o < run) v[m] += w;
        }
    if (head && agg >= 0)
#pragma unroll
        for (int m = 0; m < M; ++m) atomicAdd(c + (int64_t)M * agg + m, v[m]);
}

// The restriction by the aggregates' own lists, as many warps to one as the grid
// has: where the nodes of an aggregate are scattered over the numbering, an
// atomic per node and mode queues up on its addresses (6,859 nodes, 27 aggregates
// of six modes: an iteration 35.1 us, 27.1 with the lists and their barrier)
template <int PRE>
__device__ void restrict_lists(const PcgArgs &g, double *c)
{
    constexpr int M = PRE == 1 ? 1 : 6;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5), per = max((int64_t)1, min((int64_t)16, warps / g.nagg));
    for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < per * g.nagg; w += warps) {
        const int64_t a = w / per;
        const int32_t end = g.agg_ptr[a + 1];
        double v[M];
#pragma unroll
        for (int m = 0; m < M; ++m) v[m] = 0.0;
        for (int32_t t = g.agg_ptr[a] + (int32_t)(w % per) * 32 + lane; t < end; t += (int32_t)per * 32) {
            const int64_t n = g.agg_nodes[t];
            if constexpr (PRE == 1) {
                if (g.agg[n] >= 0) v[0] += g.r[n];
            } else {
                const float4 m = g.mode[n];
                const int bits = (int)m.w;
                const double r0 = bits & 1 ? 0.0 : g.r[3 * n], r1 = bits & 2 ? 0.0 : g.r[3 * n + 1],
                             r2 = bits & 4 ? 0.0 : g.r[3 * n + 2];
                v[0] += r0;
                v[1] += r1;
                v[2] += r2;
                v[3] += (double)m.y * r2 - (double)m.z * r1;
                v[4] += (double)m.z * r0 - (double)m.x * r2;
                v[5] += (double)m.x * r1 - (double)m.y * r0;
            }
        }
#pragma unroll
        for (int m = 0; m < M; ++m) {
            v[m] = warp_total(v[m]);
            if (lane == 0) atomicAdd(c + M * a + m, v[m]);
        }
    }
}

__device__ __forceinline__ void block_jacobi(const float *D, const double (&r)[3], double (&z)[3])
{
#pragma unroll
    for (int i = 0; i < 3; ++i)
        z[i] = (double)D[3 * i] * r[0] + (double)D[3 * i + 1] * r[1] + (double)D[3 * i + 2] * r[2];
}

// PRE: 0 point Jacobi, 1 two-level with one constant per aggregate, 2
// two-level with nodal blocks and six rigid-body modes.  r -= alpha q (INIT:
// r = b) with r.z (the Jacobi share) and r.r, and the restriction of r into c.
// x += alpha p waits for the p update, which reads p anyway.
template <int PRE, bool INIT, bool LIST>
__device__ void update(const PcgArgs &g, double alpha, double *c, double &rz, double &rr)
{
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    rz = rr = 0.0;
    if constexpr (PRE == 0) {
        for (int64_t i = t0; i < g.N; i += nt) {
            const double ri = INIT ? g.b[i] : g.r[i] - alpha * g.q[i];
            g.r[i] = ri;
            rz += ri * (g.dinv[i] * ri);
            rr += ri * ri;
        }
    } else if constexpr (PRE == 1) {
        // whole warps take every trip: the restriction shuffles
        for (int64_t base = t0 - (threadIdx.x & 31); base < g.N; base += nt) {
            const int64_t i = base + (threadIdx.x & 31);
            double v[1] = {0.0};
            int a = -1;
            if (i < g.N) {
                const double ri = INIT ? g.b[i] : g.r[i] - alpha * g.q[i];
                g.r[i] = ri;
                rz += ri * (g.dinv[i] * ri);
                rr += ri * ri;
                a = g.agg[i];
                v[0] = a >= 0 ? ri : 0.0;
            }
            if (!LIST) restrict_add<1>(c, a, v);
        }
    } else {
        for (int64_t base = t0 - (threadIdx.x & 31); base < g.nodes; base += nt) {
            const int64_t n = base + (threadIdx.x & 31);
            double v[6] = {0, 0, 0, 0, 0, 0};
            int a = -1;
            if (n < g.nodes) {
                double rv[3], zv[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const int64_t k = 3 * n + i;
                    rv[i] = INIT ? g.b[k] : g.r[k] - alpha * g.q[k];
                    g.r[k] = rv[i];
                }
                block_jacobi(g.bdinv + 9 * n, rv, zv);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    rz += rv[i] * zv[i];
                    rr += rv[i] * rv[i];
                }
                const float4 m = g.mode[n];
                const int bits = (int)m.w;
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    if ((bits >> i) & 1) rv[i] = 0.0;
                a = g.agg[n];
                v[0] = rv[0];
                v[1] = rv[1];
                v[2] = rv[2];
                v[3] = (double)m.y * rv[2] - (double)m.z * rv[1];
                v[4] = (double)m.z * rv[0] - (double)m.x * rv[2];
                v[5] = (double)m.x * rv[1] - (double)m.y * rv[0];
            }
            if (!LIST) restrict_add<6>(c, a, v);
        }
    }
}

// e = Ac c, one, two or four warps per row, as many as the grid's warps allow
// in one pass; returns this thread's part of c.e
__device__ double coarse_product(const PcgArgs &g, const double *c, double *shr)
{
    const int nw = blockDim.x >> 5;
    const int64_t warps = (int64_t)gridDim.x * nw;
    const int W = 4 * g.nc <= warps ? 4 : 2 * g.nc <= warps ? 2 : 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = warp % W, per = nw / W;
    double dot = 0.0;
    for (int64_t row0 = (int64_t)blockIdx.x * per; row0 < g.nc; row0 += (int64_t)gridDim.x * per) {
        const int64_t row = row0 + warp / W;
        const bool in = row < g.nc && warp / W < per;
        double s[4] = {0, 0, 0, 0};
        if (in) {
            const double *A = g.ac + row * g.nc;
            int64_t k = sub * 32 + lane;
            for (; k + 7 * 32 * W < g.nc; k += 8 * 32 * W)
#pragma unroll
                for (int u = 0; u < 8; ++u) s[u & 3] += A[k + 32 * W * u] * c[k + 32 * W * u];
            for (; k + 3 * 32 * W < g.nc; k += 4 * 32 * W)
#pragma unroll
                for (int u = 0; u < 4; ++u) s[u] += A[k + 32 * W * u] * c[k + 32 * W * u];
            for (; k < g.nc; k += 32 * W) s[0] += A[k] * c[k];
        }
        double t = warp_total((s[0] + s[1]) + (s[2] + s[3]));
        if (W > 1) {
            if (lane == 0) shr[warp] = t;
            __syncthreads();
            t = 0.0;
            if (sub == 0)
                for (int w = 0; w < W; ++w) t += shr[min(warp + w, 31)];
            __syncthreads();
        }
        if (in && sub == 0 && lane == 0) {
            g.e[row] = t;
            dot += t * c[row];
        }
    }
    return dot;
}

// x += alpha p, p = z + beta p (INIT: x = 0, p = z)
template <int PRE, bool INIT>
__device__ void direction(const PcgArgs &g, double alpha, double beta)
{
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    if constexpr (PRE == 2) {
        for (int64_t n = t0; n < g.nodes; n += nt) {
            double rv[3], zv[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) rv[i] = g.r[3 * n + i];
            block_jacobi(g.bdinv + 9 * n, rv, zv);
            const float4 m = g.mode[n];
            const int bits = (int)m.w;
            const double *ea = g.e + 6 * (int64_t)g.agg[n];
            const double dx = m.x, dy = m.y, dz = m.z;
            const double cc[3] = {ea[0] + ea[4] * dz - ea[5] * dy, ea[1] + ea[5] * dx - ea[3] * dz,
                                  ea[2] + ea[3] * dy - ea[4] * dx};
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double z = zv[i] + (((bits >> i) & 1) ? 0.0 : cc[i]);
                const int64_t k = 3 * n + i;
                const double p = INIT ? 0.0 : g.p[k];
                g.x[k] = INIT ? 0.0 : g.x[k] + alpha * p;
                g.p[k] = INIT ? z : z + beta * p;
            }
        }
    } else {
        for (int64_t i = t0; i < g.N; i += nt) {
            double z = g.dinv[i] * g.r[i];
            if constexpr (PRE == 1) {
                const int a = g.agg[i];
                if (a >= 0) z += g.e[a];
            }
            const double p = INIT ? 0.0 : g.p[i];
            g.x[i] = INIT ? 0.0 : g.x[i] + alpha * p;
            g.p[i] = INIT ? z : z + beta * p;
        }
    }
}

// LIST: the restriction by the aggregates' lists, a phase of its own
template <int F, int PRE, bool CL, bool LIST = false>
__global__ void __launch_bounds__(CL ? 512 : 1024, 1) k_pcg64(const __grid_constant__ PcgArgs g)
{
    __shared__ CommShared sh;
    Comm<CL> comm{g, sh};
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    double rz, rr, none = 0.0;
    update<PRE, true, LIST>(g, 0.0, g.c, rz, rr);
    if (!comm.template sum<2>(rz, rr, sum_slot(RZ, 0), sum_slot(RR, 0))) return;
    if (rr == 0.0) {
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.N; i += (int64_t)gridDim.x * blockDim.x) g.x[i] = 0.0;
        if (first) g.out[1] = 1;
    } else {
        if constexpr (PRE > 0) {
            if constexpr (LIST) {
                restrict_lists<PRE>(g, g.c);
                if (!comm.barrier()) return;
            }
            double ce = coarse_product(g, g.c, sh.rows);
            if (!comm.template sum<1>(ce, none, sum_slot(CE, 0), 0)) return;
            rz += ce;
        }
        direction<PRE, true>(g, 0.0, 0.0);
        if (!comm.barrier()) return;
        const double thr = g.tol * g.tol * rr;
        // `at` is it mod kSumRing, counted: with the slots by it & 3 the same loop
        // took 15.3 us instead of 13.0 on 33,124 rows
        int it = 0, at = 0;
        for (; it < g.max_iter; ++it) {
            const int nx = at == kSumRing - 1 ? 0 : at + 1;
            double pq = product<F>(g, g.p, g.q);
            if (!comm.template sum<1>(pq, none, ring_slot(PQ, at), 0)) return;
            if (!CL && first) clear_slots<SUMS>(g.sums, at);
            if (!(pq > 0.0)) {
                if (first) g.out[2] = 1;
                break;
            }
            // c of this iteration; the other one is cleared for the next
            double *c = g.c + ((it + 1) & 1) * g.nc;
            const double alpha = rz / pq;
            double rzn;
            update<PRE, false, LIST>(g, alpha, c, rzn, rr);
            if (!comm.template sum<2>(rzn, rr, ring_slot(RZ, nx), ring_slot(RR, nx))) return;
            if (rr <= thr) {
                for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.N; i += (int64_t)gridDim.x * blockDim.x)
                    g.x[i] += alpha * g.p[i];
                if (first) {
                    g.out[0] = it + 1;
                    g.out[1] = 1;
                }
                break;
            }
            if constexpr (PRE > 0) {
                if constexpr (LIST) {
                    restrict_lists<PRE>(g, c);
                    if (!comm.barrier()) return;
                }
                double ce = coarse_product(g, c, sh.rows);
                double *other = g.c + (it & 1) * g.nc;
                for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < g.nc; k += (int64_t)gridDim.x * blockDim.x)
                    other[k] = 0.0;
                if (!comm.template sum<1>(ce, none, ring_slot(CE, nx), 0)) return;
                rzn += ce;
            }
            direction<PRE, false>(g, alpha, rzn / rz);
            rz = rzn;
            at = nx;
            if (!comm.barrier()) return;
        }
        if (first && it == g.max_iter) g.out[0] = it;
    }
    if constexpr (CL) cg::this_cluster().sync();  // shared memory stays until the others have read it
}

// ---- the same as launches ---------------------------------------------------
// For large matrices of rows of indices, whose product wants all the warps that
// an SM can hold, in blocks that finish at their own pace: of an iteration's 82
// us on 274,625 renumbered nodes of a cube the persistent kernel's product took
// 70 and the wait for its last block 9; as a kernel of its own it takes 51.  The
// sums' slots and what they hold are those of k_pcg64; kernel boundaries are its
// barriers.  out[1] is set in iteration out[0] and stops every later one.
__device__ void add_sums(double a, double b, double *sa, double *sb)
{
    __shared__ double sh[2][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    a = warp_total(a);
    b = warp_total(b);
    if (lane == 0) {
        sh[0][warp] = a;
        sh[1][warp] = b;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[threadIdx.x][w];
        double *to = threadIdx.x ? sb : sa;
        if (to) atomicAdd(to, t);
    }
}

template <int PRE, bool INIT, bool LIST>
__global__ void __launch_bounds__(256) k_step_update(const __grid_constant__ PcgArgs g, int it)
{
    if (g.out[1] | g.out[2]) return;
    double alpha = 0.0, rz, rr;
    if (!INIT) {
        const double pq = g.sums[sum_slot(PQ, it)];
        if (!(pq > 0.0)) {
            if (blockIdx.x == 0 && threadIdx.x == 0) g.out[2] = 1;
            return;
        }
        alpha = (g.sums[sum_slot(RZ, it)] + g.sums[sum_slot(CE, it)]) / pq;
    }
    const int to = INIT ? 0 : it + 1;
    update<PRE, INIT, LIST>(g, alpha, g.c + (to & 1) * g.nc, rz, rr);
    add_sums(rz, rr, g.sums + sum_slot(RZ, to), g.sums + sum_slot(RR, to));
}

// the coarse correction of slot `to`; clears the other restriction
__global__ void __launch_bounds__(256) k_step_coarse(const __grid_constant__ PcgArgs g, int to)
{
    if (g.out[1] | g.out[2]) return;
    __shared__ double rows[32];
    const double ce = coarse_product(g, g.c + (to & 1) * g.nc, rows);
    double *other = g.c + ((to + 1) & 1) * g.nc;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < g.nc; k += (int64_t)gridDim.x * blockDim.x) other[k] = 0.0;
    add_sums(ce, 0.0, g.sums + sum_slot(CE, to), nullptr);
}

__global__ void __launch_bounds__(256) k_step_restrict(const __grid_constant__ PcgArgs g, int to)
{
    if (g.out[1] | g.out[2]) return;
    restrict_lists<1>(g, g.c + (to & 1) * g.nc);
}

template <int PRE, bool INIT>
__global__ void __launch_bounds__(256) k_step_direction(const __grid_constant__ PcgArgs g, int it, double thr)
{
    if (g.out[2] || (!INIT && g.out[1] && g.out[0] != it + 1)) return;
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    if (INIT) {
        direction<PRE, true>(g, 0.0, 0.0);
        return;
    }
    const double rz = g.sums[sum_slot(RZ, it)] + g.sums[sum_slot(CE, it)], alpha = rz / g.sums[sum_slot(PQ, it)];
    if (g.sums[sum_slot(RR, it + 1)] <= thr) {
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.N; i += (int64_t)gridDim.x * blockDim.x)
            g.x[i] += alpha * g.p[i];
        if (first) {
            g.out[0] = it + 1;
            g.out[1] = 1;
        }
        return;
    }
    direction<PRE, false>(g, alpha, (g.sums[sum_slot(RZ, it + 1)] + g.sums[sum_slot(CE, it + 1)]) / rz);
    if (first) clear_slots<SUMS>(g.sums, it);
}

// y = S x by diagonals; dot += x.y; skipped when *done
template <bool BLOCK>
__global__ void __launch_bounds__(256) k_dia_spmv64(const __grid_constant__ PcgArgs g, const double *x, double *y,
                                                    double *dot, const int *done)
{
    __shared__ double sh[8];
    if (done && *done) return;
    double d = 0.0;
    const int64_t rows = BLOCK ? g.nodes : g.N;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rows; i += (int64_t)gridDim.x * blockDim.x) {
        if constexpr (BLOCK) {
            double s[3];
            bdia_node(g.a, g.off, g.nd, g.nodes, i, x, s);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                y[3 * i + k] = s[k];
                d += x[3 * i + k] * s[k];
            }
        } else {
            const double s = dia_row(g.a, g.off, g.nd, g.N, i, x);
            y[i] = s;
            d += x[i] * s;
        }
    }
    if (dot) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = d;
        __syncthreads();
        if (threadIdx.x == 0) {
            double v = 0.0;
            for (int w = 0; w < 8; ++w) v += sh[w];
            atomicAdd(dot, v);
        }
    }
}

// the longest row (length << 32 | row)
__global__ void k_longest_row(const int32_t *__restrict__ rp, int64_t rows, unsigned long long *best)
{
    unsigned long long b = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rows; i += (int64_t)gridDim.x * blockDim.x)
        b = max(b, ((unsigned long long)(rp[i + 1] - rp[i]) << 32) | (unsigned long long)i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    if ((threadIdx.x & 31) == 0) atomicMax(best, b);
}

struct Offsets {
    int nd;
    int off[kDiaMax];  // ascending, symmetric about the main diagonal at nd / 2
};

// Every entry lies on one of the diagonals (else *bad)
__global__ void k_dia_check(const __grid_constant__ Offsets o, const int32_t *__restrict__ rp,
                            const int32_t *__restrict__ col, int64_t rows, int *bad)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rows; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t k = rp[i];
        const int32_t e = rp[i + 1];
        for (int d = 0; d < o.nd && k < e; ++d) k += col[k] - (int)i == o.off[d];
        if (k < e) atomicExch(bad, 1);  // the columns are sorted
    }
}

// BELOW = false: the diagonals on and above the main one (W values per
// entry).  BELOW = true: compares the entries below, stored or not, with them,
// *bad where they differ by more than rounding of the main diagonal.
template <int W, bool BELOW>
__global__ void k_dia_fill(const __grid_constant__ Offsets o, const int32_t *__restrict__ rp,
                           const int32_t *__restrict__ col, const double *__restrict__ a, int64_t rows,
                           double *__restrict__ dia, int *bad)
{
    const int h = o.nd / 2;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rows; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t k = rp[i];
        const int32_t e = rp[i + 1];
        for (int d = 0; d < (BELOW ? h : o.nd); ++d) {
            const bool hit = k < e && col[k] - (int)i == o.off[d];
            const int64_t at = i + o.off[d];
            if (BELOW && at >= 0) {  // an entry that is not stored is zero
                const double tol = 1e-12 * (fabs(dia[i]) + fabs(dia[at]));
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    const int t = W == 9 ? (w % 3) * 3 + w / 3 : 0;  // transposed block
                    const double up = dia[((int64_t)(h - d) * W + t) * rows + at];
                    if (!(fabs((hit ? a[(int64_t)k * W + w] : 0.0) - up) <= tol)) atomicExch(bad, 1);
                }
            }
            if (!BELOW && d >= h)
#pragma unroll
                for (int w = 0; w < W; ++w)
                    dia[((int64_t)(d - h) * W + w) * rows + i] = hit ? a[(int64_t)k * W + w] : 0.0;
            k += hit;
        }
    }
}

// The pattern's diagonals (scalar rows or node rows): those of its longest
// row, if every entry lies on one and the padding stays below a quarter.
void dia_pattern(sfc_system *s)
{
    sfc_ctx *ctx = s->ctx;
    s->dia_tried = true;
    s->dia_nd = 0;
    const bool block = s->has_bsr;
    const int32_t *rp = block ? s->bptr.p : s->row_ptr.p, *col = block ? s->bcol.p : s->col.p;
    const int64_t rows = block ? s->nodes : s->N, entries = block ? s->nblocks : s->nnz;
    unsigned long long *best = reinterpret_cast<unsigned long long *>(ctx->dsmall.p + 8);
    SFC_CK(cudaMemsetAsync(best, 0, sizeof(*best), ctx->stream));
    k_longest_row<<<grid_for(rows, 256), 256, 0, ctx->stream>>>(rp, rows, best);
    count_launch(ctx);
    unsigned long long h = 0;
    download(ctx, &h, best, 1);
    const int len = (int)(h >> 32);
    const int64_t row = (int64_t)(h & 0xffffffffu);
    if (len < 1 || len > kDiaMax || (double)len * rows > 1.25 * entries + 1024.0 * len) return;
    int32_t start = 0;
    download(ctx, &start, rp + row, 1);
    int32_t c[kDiaMax];
    download(ctx, c, col + start, len);
    Offsets o{};
    o.nd = len;
    for (int d = 0; d < len; ++d) o.off[d] = c[d] - (int)row;
    DevInt bad = status_word(ctx, 4);
    SFC_CK(cudaMemsetAsync(bad.p, 0, sizeof(int), ctx->stream));
    if (len % 2 == 0 || o.off[len / 2] != 0) return;
    for (int d = 0; d < len; ++d)
        if (o.off[d] != -o.off[len - 1 - d]) return;
    k_dia_check<<<grid_for(rows, 256), 256, 0, ctx->stream>>>(o, rp, col, rows, bad.p);
    count_launch(ctx);
    int hb = 1;
    download(ctx, &hb, bad.p, 1);
    if (hb) return;
    s->dia_nd = len;
    for (int d = 0; d < len; ++d) s->dia_off[d] = o.off[d];
}

// the diagonal copy of the current operator; false where there is none
bool dia_prepare(sfc_system *s)
{
    sfc_ctx *ctx = s->ctx;
    if (!s->dia_tried) dia_pattern(s);
    if (!s->dia_nd) return false;
    if (s->dia_serial == s->op_serial) return s->dia_ok;
    const bool block = s->has_bsr;
    const int64_t rows = block ? s->nodes : s->N;
    const int kept = s->dia_nd / 2 + 1;
    if (!reserve_spare(spare(s->dia, (size_t)kept * rows * (block ? 9 : 1)))) {  // no room for a second copy
        s->dia_nd = 0;
        return false;
    }
    Offsets o{};
    o.nd = s->dia_nd;
    std::copy(s->dia_off, s->dia_off + o.nd, o.off);
    const unsigned grid = grid_for(rows, 256);
    DevInt bad = status_word(ctx, 4);
    SFC_CK(cudaMemsetAsync(bad.p, 0, sizeof(int), ctx->stream));
    if (block) {
        k_dia_fill<9, false><<<grid, 256, 0, ctx->stream>>>(o, s->bptr.p, s->bcol.p, s->bval64.p, rows, s->dia.p, bad.p);
        k_dia_fill<9, true><<<grid, 256, 0, ctx->stream>>>(o, s->bptr.p, s->bcol.p, s->bval64.p, rows, s->dia.p, bad.p);
    } else {
        k_dia_fill<1, false><<<grid, 256, 0, ctx->stream>>>(o, s->row_ptr.p, s->col.p, s->a_op.p, rows, s->dia.p, bad.p);
        k_dia_fill<1, true><<<grid, 256, 0, ctx->stream>>>(o, s->row_ptr.p, s->col.p, s->a_op.p, rows, s->dia.p, bad.p);
    }
    count_launch(ctx, 2);
    int hb = 1;
    download(ctx, &hb, bad.p, 1);
    s->dia_serial = s->op_serial;
    s->dia_ok = hb == 0;
    return s->dia_ok;
}

PcgArgs operator_args(sfc_system *s, bool dia)
{
    PcgArgs g{};
    g.N = s->N;
    g.nodes = s->nodes;
    if (dia) {
        g.a = s->dia.p;
        const int h = s->dia_nd / 2;
        g.nd = h + 1;
        std::copy(s->dia_off + h, s->dia_off + s->dia_nd, g.off);
    }
    return g;
}

using PcgKernel = void (*)(PcgArgs);

template <int PRE, bool LIST>
PcgStats pcg64_launches(sfc_system *s, const PcgArgs &g)
{
    sfc_ctx *ctx = s->ctx;
    constexpr int kCheck = 16;
    const unsigned grid = grid_for(g.N, 256, ctx->sm_count * 8), rows = grid_for(g.nc * 32, 256, ctx->sm_count * 8);
    cudaStream_t st = ctx->stream;
    auto coarse = [&](int to) {
        if constexpr (PRE > 0) {
            if (LIST) k_step_restrict<<<grid, 256, 0, st>>>(g, to);
            k_step_coarse<<<rows, 256, 0, st>>>(g, to);
            count_launch(ctx, LIST ? 2 : 1);
        }
    };
    k_step_update<PRE, true, LIST><<<grid, 256, 0, st>>>(g, 0);
    coarse(0);
    k_step_direction<PRE, true><<<grid, 256, 0, st>>>(g, 0, 0.0);
    count_launch(ctx, 2);
    double rr = 0.0;
    download(ctx, &rr, g.sums + sum_slot(RR, 0), 1);
    if (rr == 0.0) return {0, true};
    const double thr = g.tol * g.tol * rr;
    for (int it = 0; it < g.max_iter; ++it) {
        spmv_op64_dot(s, g.p, g.q, g.sums + sum_slot(PQ, it), g.out + 1);
        k_step_update<PRE, false, LIST><<<grid, 256, 0, st>>>(g, it);
        coarse(it + 1);
        k_step_direction<PRE, false><<<grid, 256, 0, st>>>(g, it, thr);
        count_launch(ctx, 2);
        if ((it + 1) % kCheck && it + 1 < g.max_iter) continue;
        int h[3];
        download(ctx, h, g.out, 3);
        if (h[2]) fail(SFC_ERR_NOT_SPD, "PCG breakdown: p^T A p <= 0");
        if (h[1]) return {h[0], true};
    }
    return {g.max_iter, false};
}

}  // namespace

bool dia_spmv64(sfc_system *s, const double *x, double *y, double *dot, const int *done)
{
    // only the copy that a solve has made: a single product does not pay for it
    if (!s->dia_nd || s->dia_serial != s->op_serial || !s->dia_ok) return false;
    const PcgArgs g = operator_args(s, true);
    const unsigned grid = grid_for(s->has_bsr ? s->nodes : s->N, 256, s->ctx->sm_count * 8);
    if (s->has_bsr) k_dia_spmv64<true><<<grid, 256, 0, s->ctx->stream>>>(g, x, y, dot, done);
    else k_dia_spmv64<false><<<grid, 256, 0, s->ctx->stream>>>(g, x, y, dot, done);
    return true;
}

void dia_ensure(sfc_system *s) { dia_prepare(s); }

bool dia_offsets(sfc_system *s)
{
    if (!s->dia_tried) dia_pattern(s);
    return s->dia_nd > 0;
}

Format grid_operator(sfc_system *s, PcgArgs &g, bool blocks)
{
    const bool dia = dia_prepare(s);
    g = operator_args(s, dia);
    if (dia) return s->has_bsr ? BDIA : DIA;
    // node blocks where there are no diagonals, unless the tuner chose rows
    if (s->has_bsr && (blocks || s->spmv_lanes == 0)) {
        g.rp = s->bptr.p;
        g.col = s->bcol.p;
        g.a = s->bval64.p;
        return BSR;
    }
    g.rp = s->row_ptr.p;
    g.col = s->col.p;
    g.a = s->a_op.p;
    const double avg = (double)s->nnz / (double)std::max<int64_t>(s->N, 1);
    g.lanes = s->spmv_lanes > 0 ? s->spmv_lanes : avg > 24 ? 32 : avg > 12 ? 16 : avg > 6 ? 8 : 4;
    return CSR;
}

PcgStats pcg64(sfc_system *s, const double *b, double *x, double tol, int max_iter, bool two)
{
    sfc_ctx *ctx = s->ctx;
    const int64_t N = s->N;
    const CoarseSpace &cs = s->coarse;
    const int pre = !two ? 0 : cs.dof == 1 ? 1 : 2;
    PcgArgs g{};
    Format f = grid_operator(s, g, pre == 2);
    s->w64.reserve(3 * N);
    g.b = b;
    g.x = x;
    g.r = s->w64.p;
    g.p = g.r + N;
    g.q = g.p + N;
    g.dinv = s->dinv.p;
    g.bdinv = s->bdinv32.p;
    if (pre) {
        s->coarse.c64.reserve(2 * cs.nc);
        s->coarse.e64.reserve(cs.nc);
        g.agg = pre == 1 ? cs.agg_free.p : cs.node_agg.p;
        g.mode = cs.mode.p;
        g.ac = cs.a64.p;
        g.nc = cs.nc;
        g.agg_ptr = cs.agg_ptr.p;
        g.agg_nodes = cs.agg_nodes.p;
        g.nagg = cs.nagg;
        g.c = s->coarse.c64.p;
        g.e = s->coarse.e64.p;
        SFC_CK(cudaMemsetAsync(g.c, 0, 2 * cs.nc * sizeof(double), ctx->stream));
    }
    s->flags.reserve(4);
    g.out = s->flags.p;
    g.bar = reinterpret_cast<unsigned *>(s->flags.p + 3);
    g.tol = tol;
    g.max_iter = max_iter;
    SFC_CK(cudaMemsetAsync(s->flags.p, 0, 4 * sizeof(int), ctx->stream));
    if (f == CSR && (double)s->nnz > (g.lanes >= 16 ? 1 : 2) * kLaunchRows) {
        constexpr size_t slots = SUMS * kSumRing;
        s->scal.reserve(slots);
        g.sums = s->scal.p;
        SFC_CK(cudaMemsetAsync(g.sums, 0, slots * sizeof(double), ctx->stream));
        ProfScope ps(ctx, "pcg64", 0.0);
        return !pre ? pcg64_launches<0, false>(s, g) : cs.scattered ? pcg64_launches<1, true>(s, g) : pcg64_launches<1, false>(s, g);
    }
    // One cluster of up to 16 blocks while a thread has few rows: a barrier
    // takes it 1.0 us and a sum 1.5, the grid 1.6 and 2.5.
    static const PcgKernel table[2][5][5] = {
        {{k_pcg64<CSR, 0, false>, k_pcg64<CSR, 1, false>, nullptr, k_pcg64<CSR, 1, false, true>, nullptr},
         {k_pcg64<DIA, 0, false>, k_pcg64<DIA, 1, false>, nullptr, nullptr, nullptr},
         {k_pcg64<BSR, 0, false>, nullptr, k_pcg64<BSR, 2, false>, nullptr, k_pcg64<BSR, 2, false, true>},
         {k_pcg64<BDIA, 0, false>, nullptr, k_pcg64<BDIA, 2, false>, nullptr, nullptr},
         {k_pcg64<BDIA8, 0, false>, nullptr, k_pcg64<BDIA8, 2, false>, nullptr, nullptr}},
        {{k_pcg64<CSR, 0, true>, k_pcg64<CSR, 1, true>, nullptr, k_pcg64<CSR, 1, true, true>, nullptr},
         {k_pcg64<DIA, 0, true>, k_pcg64<DIA, 1, true>, nullptr, nullptr, nullptr},
         {k_pcg64<BSR, 0, true>, nullptr, k_pcg64<BSR, 2, true>, nullptr, k_pcg64<BSR, 2, true, true>},
         {k_pcg64<BDIA, 0, true>, nullptr, k_pcg64<BDIA, 2, true>, nullptr, nullptr},
         {k_pcg64<BDIA8, 0, true>, nullptr, k_pcg64<BDIA8, 2, true>, nullptr, nullptr}}};
    // Eight lanes per node while that leaves every warp with one piece of work: a
    // thread per node uses a tenth of the SMs at a few thousand nodes (an iteration
    // on 1,331, 6,859 and 17,576 nodes: 22.9, 23.3, 23.7 us; 8.5, 10.2, 13.2 so).
    if (f == BDIA && s->nodes * 8 <= 1024 * (int64_t)ctx->sm_count) f = BDIA8;
    // the aggregates' lists where their nodes are scattered (and so no diagonals)
    const int form = pre && cs.scattered && (f == CSR || f == BSR) ? pre + 2 : pre;
    SFC_REQUIRE(table[0][f][form], "no PCG kernel for this operator and preconditioner");
    const int64_t threads = f == BSR ? s->nodes * 32 : f == BDIA8 ? s->nodes * 8 : f == BDIA ? s->nodes : f == CSR ? N * g.lanes : N;
    const double work = f == BSR || f == BDIA || f == BDIA8 ? (double)s->nblocks * 9 : (double)s->nnz;
    ProfScope ps(ctx, "pcg64", 0.0);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    cfg.stream = ctx->stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    bool cluster = work <= (f == CSR ? kClusterRows : kClusterWork);
    if (cluster) {
        unsigned blocks = 1;
        while (blocks < 16 && (int64_t)blocks * 512 < threads) blocks *= 2;
        const PcgKernel kernel = table[1][f][form];
        SFC_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = blocks;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(512);
        int fit = 0;
        cluster = cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) == cudaSuccess && fit > 0;
        if (cluster) SFC_CK(cudaLaunchKernelEx(&cfg, kernel, g));
        else cudaGetLastError();
    }
    if (!cluster) {
        const PcgKernel kernel = table[0][f][form];
        int occ = 0;
        SFC_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 1024, 0));
        attr.id = cudaLaunchAttributeCooperative;
        attr.val.cooperative = 1;
        // blocks of 512 while they fit one to an SM, then one per SM of the
        // size that spreads the rows over all of them
        const int64_t sm = ctx->sm_count;
        const unsigned block = f == BDIA8 ? (unsigned)std::max<int64_t>(128, std::min<int64_t>(1024, ((threads + sm - 1) / sm + 127) / 128 * 128))
                               : threads <= 512 * sm ? 512 : (unsigned)std::min<int64_t>(1024, ((threads + sm - 1) / sm + 127) / 128 * 128);
        cfg.blockDim = dim3(block);
        cfg.gridDim = dim3(grid_for(threads, block, (int)sm * std::max(occ, 1)));
        constexpr size_t slots = SUMS * kSumRing;
        s->scal.reserve(slots);
        g.sums = s->scal.p;
        SFC_CK(cudaMemsetAsync(g.sums, 0, slots * sizeof(double), ctx->stream));
        SFC_CK(cudaLaunchKernelEx(&cfg, kernel, g));
    }
    count_launch(ctx);
    int h[3];
    download(ctx, h, g.out, 3);
    if (h[2] == 2) fail(SFC_ERR_TIMEOUT, "a grid barrier of the PCG kernel gave up");
    if (h[2]) fail(SFC_ERR_NOT_SPD, "PCG breakdown: p^T A p <= 0");
    return {h[0], h[1] != 0};
}

}  // namespace sfc
