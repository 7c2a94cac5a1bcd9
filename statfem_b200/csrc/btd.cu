// Direct FP64 solve of symmetric positive definite block-tridiagonal systems
// (the lines of a 2-D grid, the dofs of a bar): the replacement of the
// reference's Eigen::SparseLU (corlib/SystemSolveEigenSparse.hpp:273-404)
// where the matrix has that form.
//
// With A_ii the line blocks and B_i the sparse coupling of line i to the line
// before it, elimination runs from both ends towards the middle line k:
//   D_0 = A_00,  X_i = D_i^-1,  D_i = A_ii - B_i X_{i-1} B_i^T      (and mirrored)
//   z_i = b_i - B_i X_{i-1} z_{i-1},  x_k = X_k z_k,
//   x_i = X_i (z_i - B_{i+1}^T x_{i+1})
// so the only dense work is one m x m inverse per line (m^3 multiply-adds;
// the coupling has at most four entries per row) and two products of the
// inverse blocks with the right-hand sides.
//
// One thread-block cluster takes one instance: the first half of its CTAs
// runs the chain from the first line, the second half the chain from the
// last, in step (the chain is what bounds the time, so halving its length
// halves the time and costs no extra work).  Measured: one 151 x 151 grid
// with 32 columns 4.4 ms on 16 CTAs (factor 40 us a line, of which the
// sequential pivot inverses 14 and the updates 7; solve 9 us a line), 33 of
// them at once 7.8 ms; Jacobi-PCG took 264 ms for 40 grids of sides 32 to 150
// where this takes 6.5 ms.  A chain's CTAs share
// the block's rows in groups of eight, dealt round-robin, in shared memory;
// block Gauss-Jordan with 32-wide panels: every CTA reads the panel's rows,
// inverts the pivot block itself (all of them the same way, so no second
// exchange is needed) and updates its rows with FP64 tensor-core products
// (m8n8k4).  The only
// waits are cluster barriers.

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "btd.cuh"
#include "tile64.cuh"

namespace cg = cooperative_groups;

namespace sfc {
namespace {

constexpr int TT = 256;          // threads per CTA
constexpr int NW = TT / 32;      // warps per CTA
constexpr int PW = 32;           // panel width
constexpr int ZLD = 36;          // row stride of the z block in shared memory
constexpr int kLineMax = 320;    // longest line
constexpr int kLaneCols = kLineMax / 32;

__host__ __device__ inline int btd_ld(int mp) { return ((mp + 15) & ~15) + 8; }  // = 8 mod 16 doubles
__host__ __device__ inline int btd_rows(int m, int C) { return 8 * (((m + 7) / 8 + C - 1) / C); }

__host__ __device__ inline size_t btd_smem(int m, int C)
{
    const int mp = (m + 7) & ~7, ld = btd_ld(mp), rows = btd_rows(m, C);
    const size_t panel = (size_t)PW * ld > (size_t)mp * ZLD ? (size_t)PW * ld : (size_t)mp * ZLD;
    return 8 * ((size_t)rows * ld + panel + 4 * PW + (size_t)rows * (kBtdSide + kBtdSide + kBtdMid)) +
           4 * (size_t)rows * (kBtdSide + kBtdSide + kBtdMid) + 64;
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}

struct Sm {
    double *A;      // own rows [rows][ld]
    double *P;      // raw panel [PW][ld], or z [mp][ZLD]
    double *buf;    // pivot row / column exchange [2][2][PW]
    double *ev;     // entries of the own rows: previous line | next line | own line
    int *ec;
    int *word;
};

struct Inst {
    int64_t r0;
    int n, m, mp, ld, nb, mid, steps;
};

__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cl_barrier()
{
    __threadfence();
    cl_arrive();
    cl_wait();
}

// line of a chain at a step (the last step is the middle line, chain 0 only); -1: none
__device__ __forceinline__ int line_at(const Inst &q, int chain, int st)
{
    if (st == q.steps - 1) return chain == 0 ? q.mid : -1;
    if (chain == 0) return st < q.mid ? st : -1;
    const int l = q.nb - 1 - st;
    return l > q.mid ? l : -1;
}

// In-place inverse of the kw x kw symmetric positive definite block at P (row
// stride ld) by the first four warps (sweep_inverse).  Returns whether every
// pivot was positive and in the reciprocal's range: the pivots of an elimination
// in any symmetric order are positive if and only if the matrix is positive
// definite.
__device__ bool pivot_inverse(double *P, int ld, int kw, double *buf)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = 8 * warp + i;
        v[i] = r < kw && lane < kw ? P[(size_t)r * ld + lane] : (r == lane ? 1.0 : 0.0);
    }
    bool ok = true;
    sweep_inverse(v, kw, buf, [&](int, double d, double &inv) {
        ok = ok && recip_takes(d);
        inv = recip(d);
        return true;
    });
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = 8 * warp + i;
        if (r < kw && lane < kw) P[(size_t)r * ld + lane] = -v[i];
    }
    return ok;
}

// the entries of this chain's own rows of `line` into shared memory
__device__ void stage_entries(const BtdArgs &a, const Inst &q, const Sm &s, int line, int c, int C, int nloc)
{
    constexpr int E = 2 * kBtdSide + kBtdMid;
    for (int t = threadIdx.x; t < nloc * 8 * E; t += TT) {
        const int lr = t / E, e = t % E;
        const int r = ((lr >> 3) * C + c) * 8 + (lr & 7);
        const int64_t d = (int64_t)line * q.m + r;
        double v = 0.0;
        int k = 0;
        if (line >= 0 && r < q.m && d < q.n) {
            const int64_t i = q.r0 + d;
            if (e < kBtdSide) {
                v = a.lv[i * kBtdSide + e];
                k = a.lc[i * kBtdSide + e];
            } else if (e < 2 * kBtdSide) {
                v = a.uv[i * kBtdSide + e - kBtdSide];
                k = a.uc[i * kBtdSide + e - kBtdSide];
            } else {
                v = a.mv[i * kBtdMid + e - 2 * kBtdSide];
                k = a.mc[i * kBtdMid + e - 2 * kBtdSide];
            }
        }
        s.ev[t] = v;
        s.ec[t] = k;
    }
}

// D rows of `line` in A: own-line entries minus the eliminated neighbours'
// share, Y = X B^T of the chain's previous line (and of the other chain's
// last line for the middle)
__device__ void build_block(const Inst &q, const Sm &s, int line, int c, int C, int nloc, const double *Yl,
                            const double *Yu, double *G)
{
    constexpr int E = 2 * kBtdSide + kBtdMid;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int lr = warp; lr < nloc * 8; lr += NW) {
        const int r = ((lr >> 3) * C + c) * 8 + (lr & 7);
        double *row = s.A + (size_t)lr * q.ld;
        const bool valid = r < q.m && (int64_t)line * q.m + r < q.n;
        const double *ev = s.ev + lr * E;
        const int *ec = s.ec + lr * E;
        double v[kLaneCols];
#pragma unroll
        for (int u = 0; u < kLaneCols; ++u) v[u] = !valid && lane + 32 * u == r ? 1.0 : 0.0;
#pragma unroll
        for (int e = 0; e < 2 * kBtdSide; ++e) {
            const double *Y = e < kBtdSide ? Yl : Yu;
            const double w = ev[e];
            if (!Y || w == 0.0) continue;
            const double *y = Y + (size_t)ec[e] * q.mp + lane;
#pragma unroll
            for (int u = 0; u < kLaneCols; ++u)
                if (lane + 32 * u < q.mp) v[u] -= w * y[32 * u];
        }
#pragma unroll
        for (int u = 0; u < kLaneCols; ++u)
            if (lane + 32 * u < q.mp) row[lane + 32 * u] = v[u];
        __syncwarp();
        if (lane < kBtdMid && valid && ev[2 * kBtdSide + lane] != 0.0)
            row[ec[2 * kBtdSide + lane]] += ev[2 * kBtdSide + lane];
        __syncwarp();
        if (r < PW)  // a row of the first panel
            for (int j = lane; j < q.mp; j += 32) G[(size_t)r * q.mp + j] = row[j];
    }
}

// Gauss-Jordan inverse of the chain's block, rows distributed over its CTAs.
// A panel's rows reach the other CTAs through a double buffer G in global
// memory (L2), written as the step before finishes them: 0.8 us a panel
// against 3.3 us through distributed shared memory at 182 columns on eight
// CTAs, whose owners serve every reader in turn, and one cluster barrier
// instead of two (factor of the 182 x 182 grid 6.5 -> 5.1 ms).
__device__ void invert_block(const Inst &q, const Sm &s, bool have, int c, int C, int nloc, double *G, int *bad)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lr4 = lane >> 2, lk4 = lane & 3;
    const int np = (q.mp + PW - 1) / PW, ld = q.ld;
    for (int p = 0; p < np; ++p) {
        const int c0 = p * PW, kw = min(PW, q.mp - c0);
        cl_barrier();  // the panel's rows are published
        if (!have) continue;
        const double *Gp = G + (size_t)(p & 1) * PW * q.mp;
        double *Gn = G + (size_t)((p + 1) & 1) * PW * q.mp;
        for (int r = warp; r < kw; r += NW)
            for (int j = lane; 2 * j < q.mp; j += 32)
                cp_async16(s.P + (size_t)r * ld + 2 * j, Gp + (size_t)r * q.mp + 2 * j);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        // every CTA of the chain takes the same pivots: the first one reports
        if (warp < PW / 8 && !pivot_inverse(s.P + c0, ld, kw, s.buf) && c == 0 && threadIdx.x == 0) *bad = 1;
        __syncthreads();
        const int g0 = c0 >> 3, g1 = g0 + (kw >> 3), nk = kw >> 2, nt = kw >> 3;
        // panel columns: -A V for the other rows, V for the pivot rows; two
        // row groups x four column tiles per round, all read before any is written
        for (int l0 = 0; l0 < nloc; l0 += 2) {
            const int lg = l0 + (warp >> 2), ct = warp & 3;
            const int g = lg * C + c;
            const bool act = lg < nloc && ct < nt, piv = g >= g0 && g < g1;
            double *row = s.A + (size_t)(lg * 8 + lr4) * ld + c0;
            double acc[2] = {0.0, 0.0};
            if (act) {
                if (piv) {
                    const double *v = s.P + (size_t)((g - g0) * 8 + lr4) * ld + c0 + ct * 8 + 2 * lk4;
                    acc[0] = -v[0];
                    acc[1] = -v[1];
                } else {
#pragma unroll
                    for (int k = 0; k < PW / 4; ++k)
                        if (k < nk)
                            dmma(acc, row[4 * k + lk4], s.P[(size_t)(4 * k + lk4) * ld + c0 + ct * 8 + lr4]);
                }
            }
            __syncthreads();
            if (act) {
                const int rn = 8 * g + lr4 - (c0 + PW);  // row of the next panel
                const double2 v = make_double2(-acc[0], -acc[1]);
                *reinterpret_cast<double2 *>(row + ct * 8 + 2 * lk4) = v;
                if (rn >= 0 && rn < PW)
                    *reinterpret_cast<double2 *>(Gn + (size_t)rn * q.mp + c0 + ct * 8 + 2 * lk4) = v;
            }
        }
        __syncthreads();
        // the other columns, two tiles of eight per warp: the rows' panel
        // columns (now -A V, or V) times the raw panel
        const int tiles = (q.mp >> 3) - nt;
        for (int t0 = 2 * warp; t0 < tiles; t0 += 2 * NW) {
            const int ta = t0 < g0 ? t0 : t0 + nt, t1 = t0 + 1;
            const bool two = t1 < tiles;
            const int tb = !two ? ta : t1 < g0 ? t1 : t1 + nt;
            double ba[PW / 4], bb[PW / 4];
#pragma unroll
            for (int k = 0; k < PW / 4; ++k) {
                ba[k] = k < nk ? s.P[(size_t)(4 * k + lk4) * ld + ta * 8 + lr4] : 0.0;
                bb[k] = k < nk ? s.P[(size_t)(4 * k + lk4) * ld + tb * 8 + lr4] : 0.0;
            }
            for (int lg = 0; lg < nloc; ++lg) {
                const int g = lg * C + c;
                const bool piv = g >= g0 && g < g1;
                double *row = s.A + (size_t)(lg * 8 + lr4) * ld;
                double2 *pa = reinterpret_cast<double2 *>(row + ta * 8 + 2 * lk4);
                double2 *pb = reinterpret_cast<double2 *>(row + tb * 8 + 2 * lk4);
                double ca[2] = {0.0, 0.0}, cb[2] = {0.0, 0.0};
                if (!piv) {
                    const double2 x = *pa, y = *pb;
                    ca[0] = x.x;
                    ca[1] = x.y;
                    cb[0] = y.x;
                    cb[1] = y.y;
                }
#pragma unroll
                for (int k = 0; k < PW / 4; ++k)
                    if (k < nk) {
                        const double av = row[c0 + 4 * k + lk4];
                        dmma(ca, av, ba[k]);
                        dmma(cb, av, bb[k]);
                    }
                *pa = make_double2(ca[0], ca[1]);
                if (two) *pb = make_double2(cb[0], cb[1]);
                if (g >= g1 && g < g1 + PW / 8) {  // the next panel's rows
                    double *o = Gn + (size_t)((g - g1) * 8 + lr4) * q.mp + 2 * lk4;
                    *reinterpret_cast<double2 *>(o + ta * 8) = make_double2(ca[0], ca[1]);
                    if (two) *reinterpret_cast<double2 *>(o + tb * 8) = make_double2(cb[0], cb[1]);
                }
            }
        }
    }
    __syncthreads();
}

// the entries of two rows of the chain's next line towards this line (rows
// threadIdx.x and threadIdx.x + TT), loaded before the inverse that they meet
struct Couple {
    double v[2][kBtdSide];
    int k[2][kBtdSide];
};

__device__ void load_couple(const BtdArgs &a, const Inst &q, int line, int chain, Couple &p)
{
    const double *val = chain == 0 ? a.lv : a.uv;
    const int16_t *col = chain == 0 ? a.lc : a.uc;
    const int next = chain == 0 ? line + 1 : line - 1;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int j = threadIdx.x + TT * u;
        const int64_t d = (int64_t)next * q.m + j;
        double2 v0 = make_double2(0.0, 0.0), v1 = v0;
        short4 k = make_short4(0, 0, 0, 0);
        if (j < q.m && d < q.n) {
            v0 = reinterpret_cast<const double2 *>(val + (q.r0 + d) * kBtdSide)[0];
            v1 = reinterpret_cast<const double2 *>(val + (q.r0 + d) * kBtdSide)[1];
            k = *reinterpret_cast<const short4 *>(col + (q.r0 + d) * kBtdSide);
        }
        p.v[u][0] = v0.x;
        p.v[u][1] = v0.y;
        p.v[u][2] = v1.x;
        p.v[u][3] = v1.y;
        p.k[u][0] = k.x;
        p.k[u][1] = k.y;
        p.k[u][2] = k.z;
        p.k[u][3] = k.w;
    }
}

// X rows to the workspace, and Y = X B^T towards the chain's next line
__device__ void store_block(const Inst &q, const Sm &s, int line, int c, int C, int nloc, double *X, double *Y,
                            const Couple &p, bool coupling)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int lr = warp; lr < nloc * 8; lr += NW) {
        const int r = ((lr >> 3) * C + c) * 8 + (lr & 7);
        if (r >= q.m) continue;
        double *dst = X + ((size_t)line * q.m + r) * q.mp;
        const double *row = s.A + (size_t)lr * q.ld;
        for (int j = lane; j < q.mp; j += 32) dst[j] = row[j];
    }
    if (!coupling) return;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int j = threadIdx.x + TT * u;
        if (j >= q.mp) break;
        for (int lr = 0; lr < nloc * 8; ++lr) {
            const int r = ((lr >> 3) * C + c) * 8 + (lr & 7);
            if (r >= q.m) break;
            const double *row = s.A + (size_t)lr * q.ld;
            double y = 0.0;
#pragma unroll
            for (int e = 0; e < kBtdSide; ++e)
                if (p.v[u][e] != 0.0) y += p.v[u][e] * row[p.k[u][e]];
            Y[(size_t)r * q.mp + j] = y;
        }
    }
}

__device__ Inst load_inst(const BtdArgs &a, int inst)
{
    Inst q;
    q.r0 = a.row0[inst];
    q.n = (int)(a.row0[inst + 1] - q.r0);
    q.m = a.line[inst];
    q.mp = (q.m + 7) & ~7;
    q.ld = btd_ld(q.mp);
    q.nb = (q.n + q.m - 1) / q.m;
    q.mid = q.nb / 2;
    q.steps = max(q.mid, q.nb - 1 - q.mid) + 1;
    return q;
}

__device__ Sm carve(unsigned char *raw, int lmax, int C)
{
    const int mp = (lmax + 7) & ~7, ld = btd_ld(mp), rows = btd_rows(lmax, C);
    const size_t panel = (size_t)PW * ld > (size_t)mp * ZLD ? (size_t)PW * ld : (size_t)mp * ZLD;
    Sm s;
    s.A = reinterpret_cast<double *>(raw);
    s.P = s.A + (size_t)rows * ld;
    s.buf = s.P + panel;
    s.ev = s.buf + 4 * PW;
    s.ec = reinterpret_cast<int *>(s.ev + (size_t)rows * (2 * kBtdSide + kBtdMid));
    s.word = s.ec + (size_t)rows * (2 * kBtdSide + kBtdMid);
    return s;
}

__device__ __forceinline__ int local_groups(const Inst &q, int c, int C)
{
    const int G = q.mp >> 3;
    return c < G ? (G - c + C - 1) / C : 0;
}

__device__ void factor(const BtdArgs &a, const Inst &q, const Sm &s, int chain, int c, int C,
                       double *X, double *Y, int *bad)
{
    const int nloc = local_groups(q, c, C);
    const size_t ysz = (size_t)q.m * q.mp;
    double *G = Y + 2 * ysz + (size_t)chain * 2 * PW * q.mp;
    stage_entries(a, q, s, line_at(q, chain, 0), c, C, nloc);
    for (int st = 0; st < q.steps; ++st) {
        const int line = line_at(q, chain, st);
        const bool have = line >= 0, last = st == q.steps - 1;
        cl_barrier();  // Y of the previous step is written
        if (have) {
            __syncthreads();
            const double *Yl = nullptr, *Yu = nullptr;
            if (last) {
                Yl = line > 0 ? Y : nullptr;
                Yu = line + 1 < q.nb ? Y + ysz : nullptr;
            } else if (st > 0) {
                (chain == 0 ? Yl : Yu) = Y + chain * ysz;
            }
            build_block(q, s, line, c, C, nloc, Yl, Yu, G);
        }
        Couple cp;
        if (have && !last) load_couple(a, q, line, chain, cp);
        __syncthreads();
        invert_block(q, s, have, c, C, nloc, G, bad);
        if (have) store_block(q, s, line, c, C, nloc, X, Y + chain * ysz, cp, !last);
        if (!last) stage_entries(a, q, s, line_at(q, chain, st + 1), c, C, nloc);
    }
    cl_barrier();
}

// own rows of X of `line` into shared memory, asynchronously
__device__ void prefetch_block(const Inst &q, const Sm &s, int line, int c, int C, int nloc, const double *X)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (line < 0) return;
    for (int lr = warp; lr < nloc * 8; lr += NW) {
        const int r = ((lr >> 3) * C + c) * 8 + (lr & 7);
        if (r >= q.m) continue;
        const double *src = X + ((size_t)line * q.m + r) * q.mp;
        double *dst = s.A + (size_t)lr * q.ld;
        for (int j = lane; 2 * j < q.mp; j += 32) cp_async16(dst + 2 * j, src + 2 * j);
    }
}

// own rows of z (32 columns): b (use_b) minus the coupling with the solution
// rows of the neighbouring lines; the entries were staged before
__device__ void line_rhs(const BtdArgs &a, const Inst &q, const Sm &s, int line, int col0, int c, int C, int nloc,
                         bool use_b, bool lower, bool upper)
{
    constexpr int E = 2 * kBtdSide + kBtdMid, UR = 3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool ok = col0 + lane < a.ncols;
    const int64_t base = q.r0 + (int64_t)line * q.m;
    for (int l0 = warp; l0 < nloc * 8; l0 += NW * UR) {
        double v[UR];
#pragma unroll
        for (int u = 0; u < UR; ++u) {
            const int lr = l0 + u * NW, r = ((lr >> 3) * C + c) * 8 + (lr & 7);
            v[u] = 0.0;
            if (lr >= nloc * 8 || r >= q.m || (int64_t)line * q.m + r >= q.n || !ok) continue;
            if (use_b) v[u] = a.B[(base + r) * a.ld + col0 + lane];
            const double *ev = s.ev + lr * E;
            const int *ec = s.ec + lr * E;
            if (lower)
#pragma unroll
                for (int e = 0; e < kBtdSide; ++e)
                    if (ev[e] != 0.0) v[u] -= ev[e] * a.U[(base - q.m + ec[e]) * a.ld + col0 + lane];
            if (upper)
#pragma unroll
                for (int e = kBtdSide; e < 2 * kBtdSide; ++e)
                    if (ev[e] != 0.0) v[u] -= ev[e] * a.U[(base + q.m + ec[e]) * a.ld + col0 + lane];
        }
#pragma unroll
        for (int u = 0; u < UR; ++u) {
            const int lr = l0 + u * NW, r = ((lr >> 3) * C + c) * 8 + (lr & 7);
            if (lr < nloc * 8) s.P[(size_t)r * ZLD + lane] = v[u];
        }
    }
}

// the other CTAs' rows of z
__device__ void gather_z(cg::cluster_group &cl, const Inst &q, const Sm &s, int chain, int c, int C)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int UR = 8;
    for (int r0 = warp; r0 < q.mp; r0 += NW * UR) {
        double v[UR];
#pragma unroll
        for (int u = 0; u < UR; ++u) {
            const int r = r0 + u * NW, o = (r >> 3) % C;
            if (r < q.mp && o != c) v[u] = cl.map_shared_rank(s.P, chain * C + o)[(size_t)r * ZLD + lane];
        }
#pragma unroll
        for (int u = 0; u < UR; ++u) {
            const int r = r0 + u * NW, o = (r >> 3) % C;
            if (r < q.mp && o != c) s.P[(size_t)r * ZLD + lane] = v[u];
        }
    }
}

// own rows of X z: into U (add = false) or onto it
__device__ void line_product(const BtdArgs &a, const Inst &q, const Sm &s, int line, int col0, int c, int C, int nloc,
                             bool add)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lr4 = lane >> 2, lk4 = lane & 3;
    for (int u = warp; u < nloc * 4; u += NW) {
        const int lg = u >> 2, ct = u & 3;
        const int r = (lg * C + c) * 8 + lr4, cc = col0 + ct * 8 + 2 * lk4;
        const bool row_ok = r < q.m && (int64_t)line * q.m + r < q.n;
        double *o = a.U + (q.r0 + (int64_t)line * q.m + r) * a.ld + cc;
        double old0 = 0.0, old1 = 0.0;
        if (add && row_ok) {
            if (cc < a.ncols) old0 = o[0];
            if (cc + 1 < a.ncols) old1 = o[1];
        }
        const double *x = s.A + (size_t)(lg * 8 + lr4) * q.ld + lk4;
        const double *z = s.P + (size_t)lk4 * ZLD + ct * 8 + lr4;
        double acc[2] = {0.0, 0.0}, acc2[2] = {0.0, 0.0};
#pragma unroll 4
        for (int k = 0; k < q.mp; k += 8) {
            dmma(acc, x[k], z[(size_t)k * ZLD]);
            dmma(acc2, x[k + 4], z[(size_t)(k + 4) * ZLD]);
        }
        if (row_ok) {
            if (cc < a.ncols) o[0] = old0 + (acc[0] + acc2[0]);
            if (cc + 1 < a.ncols) o[1] = old1 + (acc[1] + acc2[1]);
        }
    }
}

__device__ void solve_tile(cg::cluster_group &cl, const BtdArgs &a, const Inst &q, const Sm &s, int col0, int chain,
                           int c, int C, const double *X)
{
    const int nloc = local_groups(q, c, C);
    // steps 0 .. steps - 1 towards the middle, then back to step 0
    const int total = 2 * q.steps - 1;
    auto at = [&](int t) { return line_at(q, chain, t < q.steps ? t : total - 1 - t); };
    stage_entries(a, q, s, at(0), c, C, nloc);
    prefetch_block(q, s, at(0), c, C, nloc, X);
    __syncthreads();
    for (int t = 0; t < total; ++t) {
        const int line = at(t);
        const bool fwd = t < q.steps, last = t == q.steps - 1;
        if (line >= 0) {
            const bool lower = !fwd ? chain == 1 : last ? line > 0 : chain == 0 && t > 0;
            const bool upper = !fwd ? chain == 0 : last ? line + 1 < q.nb : chain == 1 && t > 0;
            line_rhs(a, q, s, line, col0, c, C, nloc, fwd, lower, upper);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        cl_arrive();
        cl_wait();  // the rows of z (and this CTA's block) are in place
        if (line >= 0) {
            gather_z(cl, q, s, chain, c, C);
            __syncthreads();
            line_product(a, q, s, line, col0, c, C, nloc, !fwd);
        }
        __syncthreads();
        if (t + 1 < total) {
            stage_entries(a, q, s, at(t + 1), c, C, nloc);
            prefetch_block(q, s, at(t + 1), c, C, nloc, X);
        }
        cl_barrier();  // the solution rows are written
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

__global__ void __launch_bounds__(TT, 2) k_btd_batch(BtdArgs a)
{
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char raw[];
    const int C = a.chain, rank = (int)cl.block_rank(), chain = rank / C, c = rank % C;
    Sm s = carve(raw, a.lmax, C);
    const int slot = blockIdx.x / (2 * C);
    double *X = a.X + slot * a.xstride, *Y = a.Y + slot * a.ystride;
    for (;;) {
        if (rank == 0 && threadIdx.x == 0) *s.word = atomicAdd(a.queue, 1);
        cl.sync();
        const int qi = *cl.map_shared_rank(s.word, 0);
        cl.sync();
        if (qi >= a.n_inst) break;
        const int inst = a.order[qi];
        const Inst q = load_inst(a, inst);
        factor(a, q, s, chain, c, C, X, Y, a.bad + inst);
        for (int c0 = 0; c0 < a.ncols; c0 += kBtdCols) solve_tile(cl, a, q, s, c0, chain, c, C, X);
    }
}

__global__ void __launch_bounds__(TT) k_btd_factor(BtdArgs a)
{
    extern __shared__ __align__(16) unsigned char raw[];
    const int C = a.chain, rank = (int)cg::this_cluster().block_rank();
    Sm s = carve(raw, a.lmax, C);
    const Inst q = load_inst(a, 0);
    factor(a, q, s, rank / C, rank % C, C, a.X, a.Y, a.bad);
}

// one cluster per tile of 32 columns
__global__ void __launch_bounds__(TT) k_btd_solve(BtdArgs a)
{
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char raw[];
    const int C = a.chain, rank = (int)cl.block_rank();
    Sm s = carve(raw, a.lmax, C);
    const Inst q = load_inst(a, 0);
    solve_tile(cl, a, q, s, (int)(blockIdx.x / (2 * C)) * kBtdCols, rank / C, rank % C, C, a.X);
}

// row i's entries by line: padded with zero values
template <bool FILL>
__global__ void k_btd_entries(BtdArgs a, int *bad)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.N; i += (int64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = a.n_inst;
        while (hi - lo > 1) {
            const int md = (lo + hi) >> 1;
            if (a.row0[md] <= i) lo = md;
            else hi = md;
        }
        const int64_t r0 = a.row0[lo], r1 = a.row0[lo + 1];
        const int m = a.line[lo];
        const int64_t line = (i - r0) / m;
        int nl = 0, nu = 0, nm = 0;
        for (int32_t k = a.rp[i]; k < a.rp[i + 1]; ++k) {
            const int64_t j = a.col[k];
            const int64_t lj = j >= r0 && j < r1 ? (j - r0) / m : line + 9;
            const int cj = (int)(j - r0 - lj * m);
            if (lj == line) {
                if (nm == kBtdMid) {
                    nm = 1 << 20;
                    break;
                }
                if (FILL) {
                    a.mc[i * kBtdMid + nm] = (int16_t)cj;
                    a.mv[i * kBtdMid + nm] = a.a[k];
                }
                ++nm;
            } else if (lj == line - 1 && nl < kBtdSide) {
                if (FILL) {
                    a.lc[i * kBtdSide + nl] = (int16_t)cj;
                    a.lv[i * kBtdSide + nl] = a.a[k];
                }
                ++nl;
            } else if (lj == line + 1 && nu < kBtdSide) {
                if (FILL) {
                    a.uc[i * kBtdSide + nu] = (int16_t)cj;
                    a.uv[i * kBtdSide + nu] = a.a[k];
                }
                ++nu;
            } else {
                nm = 1 << 20;
                break;
            }
        }
        if (FILL) {
            for (; nm < kBtdMid; ++nm) {
                a.mc[i * kBtdMid + nm] = 0;
                a.mv[i * kBtdMid + nm] = 0.0;
            }
            for (; nl < kBtdSide; ++nl) {
                a.lc[i * kBtdSide + nl] = 0;
                a.lv[i * kBtdSide + nl] = 0.0;
            }
            for (; nu < kBtdSide; ++nu) {
                a.uc[i * kBtdSide + nu] = 0;
                a.uv[i * kBtdSide + nu] = 0.0;
            }
        } else if (nm > kBtdMid) {
            atomicExch(bad, 1);
        }
    }
}

// largest distance of an entry from the diagonal
__global__ void k_bandwidth(const int32_t *__restrict__ rp, const int32_t *__restrict__ col, int64_t N, int *bw)
{
    int w = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
        for (int32_t k = rp[i]; k < rp[i + 1]; ++k) w = max(w, abs(col[k] - (int)i));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w = max(w, __shfl_xor_sync(0xffffffffu, w, o));
    if ((threadIdx.x & 31) == 0) atomicMax(bw, w);
}

// per column: |b - S x|^2, |b|^2, |x|^2 (out[3][ncols]) and the largest
// absolute row sum of S (out[3 ncols], the bits of a non-negative double);
// behind it whether the factor is *bad.  With R, b - S x goes there too
// ([row][ncols]).  A block takes 32 columns (a lane each) and a share of the rows.
__global__ void __launch_bounds__(256) k_btd_check(const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                                                   const double *__restrict__ a, const double *__restrict__ B,
                                                   const double *__restrict__ X, int64_t N, int ld, int ncols,
                                                   const int *bad, double *out, double *__restrict__ R)
{
    __shared__ double sh[3][8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.y * 32 + lane;
    const bool ok = c < ncols;
    double rr = 0.0, bb = 0.0, xx = 0.0, big = 0.0;
    for (int64_t i = blockIdx.x * 8 + warp; i < N; i += (int64_t)gridDim.x * 8) {
        const double b = ok ? B[i * ld + c] : 0.0, x = ok ? X[i * ld + c] : 0.0;
        double r = b, sum = 0.0;
        for (int32_t k = rp[i]; k < rp[i + 1]; ++k) {
            const double v = a[k];
            sum += fabs(v);
            if (ok) r -= v * X[(int64_t)col[k] * ld + c];
        }
        if (R && ok) R[i * ncols + c] = r;
        rr += r * r;
        bb += b * b;
        xx += x * x;
        big = fmax(big, sum);
    }
    sh[0][warp][lane] = rr;
    sh[1][warp][lane] = bb;
    sh[2][warp][lane] = xx;
    __syncthreads();
    if (warp < 3 && ok) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += sh[warp][w][lane];
        atomicAdd(out + (int64_t)warp * ncols + c, t);
    }
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) out[3 * (int64_t)ncols + 1] = *bad;
    if (blockIdx.y == 0 && lane == 0)
        atomicMax(reinterpret_cast<unsigned long long *>(out + 3 * (int64_t)ncols),
                  (unsigned long long)__double_as_longlong(big));
}

// X += D (D: [row][ncols])
__global__ void k_btd_correct(double *__restrict__ X, const double *__restrict__ D, int64_t N, int ld, int ncols)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < N * ncols; t += (int64_t)gridDim.x * blockDim.x)
        X[t / ncols * ld + t % ncols] += D[t];
}

template <class K>
cudaLaunchConfig_t btd_config(K kernel, const BtdPlan &p, int clusters, cudaStream_t st, cudaLaunchAttribute *attr)
{
    allow_shared(kernel);
    SFC_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = 2 * p.chain;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(clusters * 2 * p.chain), 1, 1);
    cfg.blockDim = dim3(TT, 1, 1);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

bool btd_plan(sfc_ctx *ctx, BtdPlan &p, const int32_t *rp, const int32_t *col, int64_t N, int n_inst,
              const int64_t *row0, const int32_t *line, const int32_t *order, bool keep_blocks)
{
    p.usable = false;
    p.factored = 0;
    p.n = n_inst;
    p.N = N;
    p.lmax = 0;
    int64_t xmax = 0, nmax = 0;
    for (int i = 0; i < n_inst; ++i) {
        const int64_t n = row0[i + 1] - row0[i], m = line[i], mp = (m + 7) & ~7;
        if (m < 1 || m > kLineMax || n < 1 || n > (1 << 30)) return false;
        p.lmax = std::max(p.lmax, (int)m);
        xmax = std::max(xmax, (n + m - 1) / m * m * mp);
        nmax = std::max(nmax, n);
    }
    // CTAs per chain: the fewest that leave room for two CTAs on an SM (two
    // instances then hide each other's pivot inverses), more while the
    // clusters do not fill the device and each CTA keeps two row groups
    const size_t lim = kMaxShared;
    int C = 1;
    while (C < 8 && btd_smem(p.lmax, C) > 112 * 1024) C *= 2;
    while (C < 8 && 2 * C * n_inst < ctx->sm_count && (p.lmax + 7) / 8 >= 4 * C) C *= 2;
    if (btd_smem(p.lmax, C) > lim) return false;
    upload(ctx, p.row0, row0, n_inst + 1);
    upload(ctx, p.line, line, n_inst);
    upload(ctx, p.order, order, n_inst);
    p.word.reserve(2);
    p.bad.reserve(n_inst);
    BtdArgs a{};
    a.rp = rp;
    a.col = col;
    a.n_inst = n_inst;
    a.row0 = p.row0.p;
    a.line = p.line.p;
    a.N = N;
    SFC_CK(cudaMemsetAsync(p.word.p, 0, 2 * sizeof(int), ctx->stream));
    k_btd_entries<false><<<grid_for(N, 256), 256, 0, ctx->stream>>>(a, p.word.p + 1);
    count_launch(ctx);
    int bad = 1;
    download(ctx, &bad, p.word.p + 1, 1);
    if (bad) return false;
    int clusters = 0;
    for (; C <= 8; C *= 2) {
        p.chain = C;
        p.smem = btd_smem(p.lmax, C);
        if (p.smem > lim) continue;
        cudaLaunchAttribute attr;
        cudaLaunchConfig_t cfg = btd_config(k_btd_batch, p, 1, ctx->stream, &attr);
        if (cudaOccupancyMaxActiveClusters(&clusters, k_btd_batch, &cfg) == cudaSuccess && clusters > 0) break;
        cudaGetLastError();
        clusters = 0;
    }
    if (clusters == 0) return false;
    p.slots = keep_blocks ? 1 : std::min(clusters, n_inst);
    const int mp = (p.lmax + 7) & ~7;
    const size_t entries = N * (2 * kBtdSide + kBtdMid);
    if (!reserve_spare(spare(p.cols, entries), spare(p.vals, entries), spare(p.X, (size_t)p.slots * xmax),
                       spare(p.Y, (size_t)p.slots * 2 * (p.lmax + 2 * PW) * mp))) {  // the iterative solver needs less
        p.cols.release();
        p.vals.release();
        p.X.release();
        p.Y.release();
        return false;
    }
    p.usable = true;
    return true;
}

BtdArgs btd_args(BtdPlan &p, const int32_t *rp, const int32_t *col, const double *val)
{
    BtdArgs a{};
    a.rp = rp;
    a.col = col;
    a.a = val;
    a.n_inst = p.n;
    a.row0 = p.row0.p;
    a.line = p.line.p;
    a.order = p.order.p;
    a.N = p.N;
    a.lc = p.cols.p;
    a.uc = a.lc + p.N * kBtdSide;
    a.mc = a.uc + p.N * kBtdSide;
    a.lv = p.vals.p;
    a.uv = a.lv + p.N * kBtdSide;
    a.mv = a.uv + p.N * kBtdSide;
    a.X = p.X.p;
    a.Y = p.Y.p;
    a.xstride = (int64_t)(p.X.n / p.slots);
    a.ystride = (int64_t)(p.Y.n / p.slots);
    a.queue = p.word.p;
    a.bad = p.bad.p;
    a.chain = p.chain;
    a.lmax = p.lmax;
    return a;
}

void btd_launch_batch(sfc_ctx *ctx, const BtdPlan &p, const BtdArgs &a, cudaStream_t st)
{
    k_btd_entries<true><<<grid_for(a.N, 256), 256, 0, st>>>(a, nullptr);
    SFC_CK(cudaGetLastError());
    SFC_CK(cudaMemsetAsync(a.queue, 0, sizeof(int), st));
    SFC_CK(cudaMemsetAsync(a.bad, 0, a.n_inst * sizeof(int), st));
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = btd_config(k_btd_batch, p, p.slots, st, &attr);
    SFC_CK(cudaLaunchKernelEx(&cfg, k_btd_batch, a));
}

void btd_launch_factor(sfc_ctx *ctx, const BtdPlan &p, const BtdArgs &a)
{
    k_btd_entries<true><<<grid_for(a.N, 256), 256, 0, ctx->stream>>>(a, nullptr);
    SFC_CK(cudaMemsetAsync(a.bad, 0, sizeof(int), ctx->stream));
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = btd_config(k_btd_factor, p, 1, ctx->stream, &attr);
    SFC_CK(cudaLaunchKernelEx(&cfg, k_btd_factor, a));
    count_launch(ctx, 2);
}

void btd_launch_solve(sfc_ctx *ctx, const BtdPlan &p, const BtdArgs &a)
{
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = btd_config(k_btd_solve, p, (a.ncols + kBtdCols - 1) / kBtdCols, ctx->stream, &attr);
    SFC_CK(cudaLaunchKernelEx(&cfg, k_btd_solve, a));
    count_launch(ctx);
}

namespace {

// The lines of a small-bandwidth system: 32 dofs where the bandwidth allows
// it (one panel per line; the whole system as one line up to 64 dofs), else
// the grid line of a triangulated grid (bandwidth - 1: the last node of a
// line has no neighbour two lines on), else the bandwidth.
void plan_system(sfc_system *s)
{
    BtdPlan &p = s->btd;
    sfc_ctx *ctx = s->ctx;
    p.tried = true;
    p.usable = false;
    if (s->N > (1 << 20) || s->has_bsr) return;
    p.word.reserve(2);
    SFC_CK(cudaMemsetAsync(p.word.p, 0, 2 * sizeof(int), ctx->stream));
    k_bandwidth<<<grid_for(s->N, 256), 256, 0, ctx->stream>>>(s->row_ptr.p, s->col.p, s->N, p.word.p);
    count_launch(ctx);
    int bw = 0;
    download(ctx, &bw, p.word.p, 1);
    p.width = std::max(bw - 1, 1);
    const int64_t row0[2] = {0, s->N};
    const int32_t order = 0;
    for (const int m : {s->N <= 64 ? (int)s->N : 32, bw - 1, bw}) {
        if (m < 1 || m > kLineMax || (int64_t)m > s->N || m < bw - 1) continue;
        const int32_t line = m;
        if (btd_plan(ctx, p, s->row_ptr.p, s->col.p, s->N, 1, row0, &line, &order, true)) return;
    }
}

}  // namespace

bool btd_applies(sfc_system *s)
{
    if (!s->btd.tried) plan_system(s);
    return s->btd.usable;
}

// A chain's step takes a factor of 6 + 0.1 m + 0.0009 m^2 us and, there and back,
// a solve of 7 + 0.07 m (m dofs to a line; fitted to the times at direct_pays,
// within 15 %), 1.3 times that in chains of a few CTAs with three row groups and
// more each; the clusters of a wave beside one another, 32 columns to a cluster.
double btd_estimate(const sfc_system *s, int nrhs)
{
    const BtdPlan &p = s->btd;
    const double m = p.lmax, steps = std::ceil((double)p.N / m) / 2 + 1;
    const int tiles = (nrhs + kBtdCols - 1) / kBtdCols, wave = std::max(1, s->ctx->sm_count / (2 * p.chain));
    const double factor = p.factored == s->op_serial ? 0.0 : 6 + 0.1 * m + 0.0009 * m * m;
    const double full = p.chain < 8 && btd_rows(p.lmax, p.chain) >= 24 ? 1.3 : 1.0;
    return 60 + full * steps * (factor + (7 + 0.07 * m) * ((tiles + wave - 1) / wave));
}

bool btd_solve_system(sfc_system *s, const double *B, double *X, int nrhs, int ld, double tol, bool recurrence,
                      double *max_rel)
{
    sfc_ctx *ctx = s->ctx;
    BtdPlan &p = s->btd;
    if (!btd_applies(s)) return false;
    BtdArgs a = btd_args(p, s->row_ptr.p, s->col.p, s->a_op.p);
    a.B = B;
    a.U = X;
    a.ld = ld;
    a.ncols = nrhs;
    if (p.factored != s->op_serial) {
        btd_launch_factor(ctx, p, a);
        p.factored = s->op_serial;
    }
    btd_launch_solve(ctx, p, a);
    const size_t nn = 3 * (size_t)nrhs + 2;
    p.norms.reserve(nn);
    std::vector<double> h(nn);
    const dim3 grid((unsigned)std::min<int64_t>((s->N + 31) / 32, 2 * ctx->sm_count), (unsigned)((nrhs + 31) / 32));
    auto check = [&](double *R) {
        SFC_CK(cudaMemsetAsync(p.norms.p, 0, nn * sizeof(double), ctx->stream));
        k_btd_check<<<grid, 256, 0, ctx->stream>>>(s->row_ptr.p, s->col.p, s->a_op.p, B, X, s->N, ld, nrhs, a.bad,
                                                  p.norms.p, R);
        count_launch(ctx);
        if (!R) download(ctx, h.data(), p.norms.p, nn);
    };
    // every column within tol; with `floor` one whose residual is at the
    // rounding of its own terms, on a system that rounding does not swamp,
    // will do (a nearly singular one has solutions so large that any residual
    // is at theirs)
    auto within = [&](bool floor) {
        double worst = 0.0;
        for (int c = 0; c < nrhs; ++c) {
            const double r = std::sqrt(h[c]), b = std::sqrt(h[nrhs + c]), x = std::sqrt(h[2 * (size_t)nrhs + c]);
            const double terms = 8.0 * 2.2e-16 * (h[3 * (size_t)nrhs] * x + b);
            if (!(r <= tol * b || (floor && r <= terms && terms <= 1e-8 * b))) return false;
            if (b > 0) worst = std::max(worst, r / b);
        }
        *max_rel = worst;
        return true;
    };
    check(nullptr);
    if (h[nn - 1] != 0.0) return false;  // not positive definite: for the iteration to report
    if (within(recurrence)) return true;
    // a residual above tol: once more on it with the same factor, twice at most
    const size_t n = (size_t)s->N * nrhs;
    DBuf<double> R, D;
    if (!reserve_spare(spare(R, n), spare(D, n))) return false;
    BtdArgs e = a;
    e.B = R.p;
    e.U = D.p;
    e.ld = nrhs;
    for (int step = 0; step < 2; ++step) {
        check(R.p);
        btd_launch_solve(ctx, p, e);
        k_btd_correct<<<grid_for((int64_t)n, 256), 256, 0, ctx->stream>>>(X, D.p, s->N, ld, nrhs);
        count_launch(ctx);
        check(nullptr);
        if (within(recurrence)) return true;
    }
    return false;
}

}  // namespace sfc
