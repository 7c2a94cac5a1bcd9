// The operator of the persistent FP64 solvers (pcg.cu; the learned CG of
// mpnn.cu), its product with a vector by the grid, and sums and barriers over
// the grid.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace sfc {

namespace cg = cooperative_groups;

constexpr int kDiaMax = 32;    // diagonals of the pattern
// BDIA8: block diagonals, eight lanes to a node
enum Format { CSR = 0, DIA = 1, BSR = 2, BDIA = 3, BDIA8 = 4 };

struct PcgArgs {
    int64_t N, nodes;          // dofs; nodes of a 3-dof mesh
    const int32_t *rp, *col;   // CSR rows, or node-block rows
    const double *a;           // CSR values, diagonals or node blocks
    int lanes;                 // lanes per CSR row
    int nd;                    // diagonals kept: the main one, then those above it
    int off[kDiaMax / 2 + 1];
    const double *b, *dinv;
    const float *bdinv;        // nodal block inverses
    double *x, *r, *p, *q;
    // coarse space
    const int32_t *agg;        // aggregate of a node; scalar meshes: -1 where constrained
    const float4 *mode;
    const double *ac;          // nc x nc inverse
    int64_t nc;
    double *c, *e;             // [2][nc], [nc]
    // nodes by aggregate, where the numbering scatters those of an aggregate
    const int32_t *agg_ptr, *agg_nodes;
    int64_t nagg;
    double *sums;              // [sum][kSumRing]: slots of the sums, zero at the start
    unsigned *bar;
    double tol;
    int max_iter;
    int *out;                  // iterations, converged, error
};

// Slots of a sum over the grid, by iteration: the one in use, those whose last
// readers and first writers lie a barrier apart from its own, and the one that
// an iteration clears for the third one after it.
constexpr int kSumRing = 4;

namespace {

// slot of sum k in iteration it, and the clearing: by one thread of the grid,
// behind the first barrier of iteration it (every block has then read what
// iteration it - 1 and those before it added up)
__host__ __device__ __forceinline__ int ring_slot(int k, int at) { return k * kSumRing + at; }
__host__ __device__ __forceinline__ int sum_slot(int k, int it) { return ring_slot(k, it & (kSumRing - 1)); }
template <int SUMS>
__device__ __forceinline__ void clear_slots(double *sums, int it)
{
#pragma unroll
    for (int k = 0; k < SUMS; ++k) sums[sum_slot(k, it + 3)] = 0.0;
}

__device__ __forceinline__ double warp_total(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct CommShared {
    double warps[2][32], rows[32];
    double part[2][2];
    int ok;
};

// Sums over all blocks, each of them also a barrier.  CL: the blocks are one
// cluster (hardware barrier, shares read through distributed shared memory).
// Else a cooperative grid: an atomic per block into the sum's own slot and a
// counter (2.3 us a sum; reading every block's share instead took 2.9, and
// polling the shares themselves, without a counter, 4.3: the polls queue up
// behind one another on a few lines of L2).  The counter's wait is bounded
// (2^22 polls, seconds): a block that gives up reports it, and so does every
// other in its turn.
template <bool CL>
struct Comm {
    const PcgArgs &g;
    CommShared &sh;
    unsigned target = 0;
    int turn = 0;

    __device__ bool barrier()
    {
        if constexpr (CL) {
            cg::this_cluster().sync();  // releases and acquires global memory too
            return true;
        } else {
            __syncthreads();
            if (threadIdx.x == 0) {
                target += gridDim.x;
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(g.bar) : "memory");
                unsigned v = 0;
                int n = 0;
                do {
                    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(g.bar) : "memory");
                } while ((int)(v - target) < 0 && ++n < (1 << 22));
                sh.ok = (int)(v - target) >= 0;
                if (!sh.ok) atomicExch(g.out + 2, 2);
                __threadfence();
            }
            __syncthreads();
            return sh.ok != 0;
        }
    }

    // a (and b, M = 2) <- the sum over all threads
    template <int M>
    __device__ bool sum(double &a, double &b, int slot0, int slot1)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
        a = warp_total(a);
        if (M == 2) b = warp_total(b);
        if (lane == 0) {
            sh.warps[0][warp] = a;
            if (M == 2) sh.warps[1][warp] = b;
        }
        __syncthreads();
        if (warp < M) {
            const double t = warp_total(lane < nw ? sh.warps[warp][lane] : 0.0);
            if (lane == 0) {
                if (CL) sh.part[turn][warp] = t;
                else atomicAdd(g.sums + (warp ? slot1 : slot0), t);
            }
        }
        if (!barrier()) return false;
        if constexpr (CL) {
            cg::cluster_group cl = cg::this_cluster();
            const bool in = lane < (int)cl.num_blocks();
            const double *part = cl.map_shared_rank(&sh.part[turn][0], in ? lane : 0);
            a = warp_total(in ? part[0] : 0.0);
            if (M == 2) b = warp_total(in ? part[1] : 0.0);
            turn ^= 1;
        } else {
            a = g.sums[slot0];
            if (M == 2) b = g.sums[slot1];
        }
        return true;
    }
};

// row i of S x
__device__ __forceinline__ double dia_row(const double *a, const int *off, int nd, int64_t N, int64_t i, const double *x)
{
    double s = a[i] * x[i];
    constexpr int U = 4;
    for (int d0 = 1; d0 < nd; d0 += U) {
        double v[2 * U], xv[2 * U];
#pragma unroll
        for (int d = 0; d < U; ++d) {
            const bool in = d0 + d < nd;
            const int64_t o = in ? off[d0 + d] : 0, up = i + o, dn = i - o;
            const double *ad = a + (int64_t)(in ? d0 + d : 0) * N;
            const bool u = in && up < N, l = in && dn >= 0;
            v[2 * d] = u ? ad[i] : 0.0;
            xv[2 * d] = u ? x[up] : 0.0;
            v[2 * d + 1] = l ? ad[dn] : 0.0;
            xv[2 * d + 1] = l ? x[dn] : 0.0;
        }
#pragma unroll
        for (int d = 0; d < 2 * U; ++d) s += v[d] * xv[d];
    }
    return s;
}

// s += block d of node at (below: its transpose) times x of node j
__device__ __forceinline__ void bdia_block(const double *a, int64_t nodes, int d, int64_t at, int64_t j, bool below,
                                           const double *x, double (&s)[3])
{
    double v[9], xv[3];
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = a[((int64_t)d * 9 + k) * nodes + at];
#pragma unroll
    for (int k = 0; k < 3; ++k) xv[k] = x[3 * j + k];
#pragma unroll
    for (int r = 0; r < 3; ++r)
        s[r] += below ? v[r] * xv[0] + v[3 + r] * xv[1] + v[6 + r] * xv[2]
                      : v[3 * r] * xv[0] + v[3 * r + 1] * xv[1] + v[3 * r + 2] * xv[2];
}

// share `sub` of eight of the three rows of node i
__device__ __forceinline__ void bdia_share(const double *a, const int *off, int nd, int64_t nodes, int64_t i, int sub,
                                           const double *x, double (&s)[3])
{
    if (sub == 0) bdia_block(a, nodes, 0, i, i, false, x, s);
#pragma unroll 1
    for (int b = sub + 1; b < 2 * nd; b += 8) {  // 1, 2: above and below on the first diagonal, and so on
        if (b == 2 * nd - 1) break;
        const int d = (b + 1) >> 1;
        const int64_t j = b & 1 ? i + off[d] : i - off[d];
        if (j >= 0 && j < nodes) bdia_block(a, nodes, d, b & 1 ? i : j, j, !(b & 1), x, s);
    }
}

// the three rows of node i, a thread per node: the operand's three values
// serve three rows (a thread per row read them three times and was bound by
// its L1 wavefronts: 63 us for 48^3 elasticity)
__device__ __forceinline__ void bdia_node(const double *a, const int *off, int nd, int64_t nodes, int64_t i,
                                          const double *x, double (&s)[3])
{
    s[0] = s[1] = s[2] = 0.0;
    bdia_block(a, nodes, 0, i, i, false, x, s);
#pragma unroll 1
    for (int d = 1; d < nd; ++d) {
        const int64_t up = i + off[d], dn = i - off[d];
        if (up < nodes) bdia_block(a, nodes, d, i, up, false, x, s);
        if (dn >= 0) bdia_block(a, nodes, d, dn, dn, true, x, s);
    }
}

// q = S p over the grid's share of the rows; returns this thread's part of p.q
template <int F>
__device__ double product(const PcgArgs &g, const double *p, double *q)
{
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    double dot = 0.0;
    if constexpr (F == DIA) {
        for (int64_t i = t0; i < g.N; i += nt) {
            const double s = dia_row(g.a, g.off, g.nd, g.N, i, p);
            q[i] = s;
            dot += p[i] * s;
        }
    } else if constexpr (F == BDIA8) {  // four nodes to a warp
        for (int64_t base = (t0 >> 5) * 4; base < g.nodes; base += (nt >> 5) * 4) {
            const int64_t i = base + (lane & 3);
            double s[3] = {0.0, 0.0, 0.0};
            if (i < g.nodes) bdia_share(g.a, g.off, g.nd, g.nodes, i, lane >> 2, p, s);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
                if (lane < 4 && i < g.nodes) {
                    q[3 * i + k] = s[k];
                    dot += p[3 * i + k] * s[k];
                }
            }
        }
    } else if constexpr (F == BDIA) {
        for (int64_t i = t0; i < g.nodes; i += nt) {
            double s[3];
            bdia_node(g.a, g.off, g.nd, g.nodes, i, p, s);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                q[3 * i + k] = s[k];
                dot += p[3 * i + k] * s[k];
            }
        }
    } else if constexpr (F == BSR) {
        for (int64_t i = t0 >> 5; i < g.nodes; i += nt >> 5) {
            double s0 = 0.0, s1 = 0.0, s2 = 0.0;
            for (int32_t b = g.rp[i] + lane; b < g.rp[i + 1]; b += 32) {
                const int64_t j = g.col[b];
                const double *v = g.a + 9 * (int64_t)b;
                const double x0 = p[3 * j], x1 = p[3 * j + 1], x2 = p[3 * j + 2];
                s0 += v[0] * x0 + v[1] * x1 + v[2] * x2;
                s1 += v[3] * x0 + v[4] * x1 + v[5] * x2;
                s2 += v[6] * x0 + v[7] * x1 + v[8] * x2;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                s1 += __shfl_xor_sync(0xffffffffu, s1, o);
                s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            }
            if (lane < 3) {
                const double s = lane == 0 ? s0 : lane == 1 ? s1 : s2;
                q[3 * i + lane] = s;
                dot += p[3 * i + lane] * s;
            }
        }
    } else {
        // two groups of rows at a time (row bounds, columns and operands of one are
        // a chain of loads), the matrix past L1, which the operand may keep
        constexpr int U = 2;
        const int G = g.lanes, per = 32 / G;
        const int64_t step = (nt >> 5) * per;
        for (int64_t base = (t0 >> 5) * per; base < g.N; base += U * step) {
            const int64_t i0 = base + lane / G;
            int32_t k[U], e[U];
            double s[U];
            bool more = false;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int64_t i = i0 + u * step;
                k[u] = i < g.N ? g.rp[i] + lane % G : 0;
                e[u] = i < g.N ? g.rp[i + 1] : 0;
                s[u] = 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) more |= k[u] < e[u];
            while (more) {
                int32_t c[U];
                double a[U];
                more = false;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    c[u] = k[u] < e[u] ? __ldcs(g.col + k[u]) : -1;
                    a[u] = k[u] < e[u] ? __ldcs(g.a + k[u]) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (c[u] >= 0) s[u] += a[u] * p[c[u]];
                    k[u] += G;
                    more |= k[u] < e[u];
                }
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < U; ++u) {
                for (int o = G / 2; o > 0; o >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o, G);
                const int64_t i = i0 + u * step;
                if (i < g.N && lane % G == 0) {
                    q[i] = s[u];
                    dot += p[i] * s[u];
                }
            }
        }
    }
    return dot;
}

}  // namespace

// pcg.cu: the operator's best form for such a kernel (the diagonal copy where
// there is one; node blocks if `blocks` or the tuner left the choice open),
// into g
Format grid_operator(sfc_system *s, PcgArgs &g, bool blocks);

}  // namespace sfc
