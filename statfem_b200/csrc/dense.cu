// Dense FP64 inverse of a symmetric positive (semi)definite matrix by block
// Gauss-Jordan elimination without pivoting, on the GPU: the in-place form
//     A[k,k] <- D^-1,  A[k,j] <- D^-1 A[k,j],  A[i,k] <- -A[i,k] D^-1,
//     A[i,j] <- A[i,j] - A[i,k] D^-1 A[k,j]
// for 32-wide panels k (D the panel's diagonal block), one launch per panel: a
// tile's own values are read and written by one CTA, and the panel's rows and
// columns, which the others read, were copied by the launch before.  Used for
// the coarse matrix of the two-level preconditioner (with dependent pivots
// dropped: a generalised inverse on the independent modes) and for the
// sensor-space matrices of the KOH likelihood and posterior
// (LikelihoodKOH.ipp:75-120, 311-361), where a non-positive pivot is the
// reference's failed LLT.  The Schur-complement pivots are the squared
// diagonal of the Cholesky factor, so their logarithms sum to log det A.

#include <algorithm>

#include "common.cuh"
#include "tile64.cuh"

namespace sfc {

namespace {

constexpr int kGJ = 32;     // panel width
constexpr int kGjTile = 64; // tile of A per CTA

// The sweep of gj_block_inverse, with 1 / d by recip or by division; returns
// whether every pivot taken was in recip's range (the same in all threads)
template <int LD, bool DIVIDE>
__device__ __forceinline__ bool gj_sweep(const double *D, int kb, const double *thr, double *buf, double (&v)[8],
                                         int &ndrop, double *pivots)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = 8 * warp + i;
        v[i] = r < kb && lane < kb ? D[r * LD + lane] : (r == lane ? 1.0 : 0.0);
    }
    bool ok = true;
    ndrop = 0;
    sweep_inverse(v, kGJ, buf, [&](int k, double d, double &inv) {
        const bool drop = k < kb && !(d > thr[k]);
        if (threadIdx.x == 0 && k < kb) {
            if (pivots) pivots[k] = d;
            ndrop += drop;
        }
        ok = ok && (drop || recip_takes(d));
        if (!drop) inv = DIVIDE ? 1.0 / d : recip(d);
        return !drop;
    });
    return ok;
}

// Inverse of the kb x kb symmetric block in D (row stride LD) by the first
// four warps (sweep_inverse), written to out (32 x 32, zero outside).  A pivot
// not above rel x the dof's original diagonal (thr) is dropped: its row and
// column are zeroed.  A block with a pivot outside recip's range is swept again,
// with divisions (with the choice at each pivot a step of 1,000 x 1,000 took
// 17.2 us, 16.3 so).  buf: 2 x 32.
template <int LD>
__device__ void gj_block_inverse(const double *D, int kb, const double *thr, double *buf, double *out, int *dropped,
                                 double *pivots)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[8];
    int ndrop;
    if (!gj_sweep<LD, false>(D, kb, thr, buf, v, ndrop, pivots)) gj_sweep<LD, true>(D, kb, thr, buf, v, ndrop, pivots);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = 8 * warp + i;
        out[r * kGJ + lane] = r < kb && lane < kb ? -v[i] : 0.0;
    }
    if (threadIdx.x == 0 && ndrop) atomicAdd(dropped, ndrop);
}

// The original diagonal (x rel: the thresholds of the pivots) and the inverse
// of the first diagonal block; the other CTAs copy the first panel's rows
// (rowp[m][j]) and columns (colp[i][m]), kGjTile of either
__global__ void __launch_bounds__(256) k_gj_first(const double *__restrict__ A, int64_t n, double rel,
                                                  double *__restrict__ thr, double *__restrict__ dinv,
                                                  double *__restrict__ rowp, double *__restrict__ colp, int *dropped,
                                                  double *pivots)
{
    __shared__ double D[kGJ * (kGJ + 1)], buf[2 * kGJ], st[kGJ];
    const int kb = (int)min((int64_t)kGJ, n);
    if (blockIdx.x > 0) {
        const int64_t j0 = (int64_t)(blockIdx.x - 1) * kGjTile;
#pragma unroll
        for (int u = 0; u < kGjTile * kGJ / 256; ++u) {
            const int t = threadIdx.x + 256 * u, l = t / kGjTile, j = t % kGjTile, i = t / kGJ, m = t % kGJ;
            if (l < kb && j0 + j < n) rowp[l * n + j0 + j] = A[l * n + j0 + j];
            if (m < kb && j0 + i < n) colp[(j0 + i) * kGJ + m] = A[(j0 + i) * n + m];
        }
        return;
    }
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) thr[i] = rel * A[i * n + i];
    for (int t = threadIdx.x; t < kGJ * kGJ; t += blockDim.x) {
        const int r = t / kGJ, c = t % kGJ;
        D[r * (kGJ + 1) + c] = r < kb && c < kb ? A[r * n + c] : 0.0;
    }
    if (threadIdx.x < kGJ) st[threadIdx.x] = threadIdx.x < kb ? rel * A[threadIdx.x * (n + 1)] : 0.0;
    __syncthreads();
    if (threadIdx.x < 128) gj_block_inverse<kGJ + 1>(D, kb, st, buf, dinv, dropped, pivots);
}

// One panel, a 64 x 64 tile of A per CTA, in place, with D^-1 of the panel's
// diagonal block in dinv and its rows and columns as they were in rowp, colp:
//   rows of the panel:     A[i][j] = r[i - k0][j],  r = D^-1 rowp[:, j] (D^-1 itself inside the block)
//   columns of the panel:  A[i][j] = -colp[i] r[:, j]
//   elsewhere:             A[i][j] -= colp[i] r[:, j]
// on FP64 matrix instructions, every CTA forming the r of its columns itself
// and copying what it has of the next panel's rows and columns.  The first CTA
// takes the tile with the next panel's diagonal block and inverts that too,
// while the others are at their products: the chain from panel to panel is a
// launch, a tile and an inverse of 3 us.  1,000 x
// 1,000: 468 us; 1,202 as two launches per panel, the inverse (with a barrier
// of the whole CTA and a division per pivot) before the panel's products.
__global__ void __launch_bounds__(256) k_gj_step(double *__restrict__ A, int64_t n, int64_t k0, int kb,
                                                 const double *__restrict__ thr, const double *__restrict__ rowp,
                                                 const double *__restrict__ colp, double *__restrict__ rown,
                                                 double *__restrict__ coln, const double *__restrict__ dinv,
                                                 double *__restrict__ dnext, int *dropped, double *pivots)
{
    constexpr int T = kGjTile, LC = kGJ + 4, LR = T + 4;  // odd multiples of four: no bank conflicts
    __shared__ double sD[kGJ * LC], sC[T * LC], sR[kGJ * LR];
    __shared__ double buf[2 * kGJ], st[kGJ];
    const int gt = (int)((n + T - 1) / T);
    const int64_t kn = k0 + kGJ;  // the next panel
    const int crit = (int)(min(kn, n - 1) / T);
    int b = blockIdx.x;
    b = b == 0 ? crit * gt + crit : b == crit * gt + crit ? 0 : b;
    const int64_t i0 = (int64_t)(b / gt) * T, j0 = (int64_t)(b % gt) * T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, q = lane & 3;
    const int wi = 16 * (warp & 3), wj = 32 * (warp >> 2);  // the warp's 16 x 32 of the tile
    double own[2][4][2];
    {  // every load of a thread in flight before the stores
        double vd[4], vc[8], vr[8];
#pragma unroll
        for (int u = 0; u < 4; ++u) vd[u] = dinv[threadIdx.x + 256 * u];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int t = threadIdx.x + 256 * u;
            const int i = t / kGJ, m = t % kGJ, l = t / T, j = t % T;
            vc[u] = (i0 + i < n && m < kb) ? colp[(i0 + i) * kGJ + m] : 0.0;
            vr[u] = (l < kb && j0 + j < n) ? rowp[l * n + j0 + j] : 0.0;
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const int64_t i = i0 + wi + 8 * x + r, j = j0 + wj + 8 * y + 2 * q + v;
                    own[x][y][v] = i < n && j < n ? A[i * n + j] : 0.0;
                }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int t = threadIdx.x + 256 * u;
            sD[(t / kGJ) * LC + t % kGJ] = vd[u];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int t = threadIdx.x + 256 * u;
            sC[(t / kGJ) * LC + t % kGJ] = vc[u];
            sR[(t / T) * LR + t % T] = vr[u];
        }
        if (threadIdx.x < kGJ) st[threadIdx.x] = kn + threadIdx.x < n ? thr[kn + threadIdx.x] : 0.0;
    }
    __syncthreads();
    {  // r: rows 8 (warp % 4) .., columns wj .. of it
        double p[4][2];
#pragma unroll
        for (int y = 0; y < 4; ++y) p[y][0] = p[y][1] = 0.0;
        const int m0 = 8 * (warp & 3);
#pragma unroll
        for (int k = 0; k < kGJ; k += 4) {
            const double a = sD[(m0 + r) * LC + k + q];
#pragma unroll
            for (int y = 0; y < 4; ++y) dmma(p[y], a, sR[(k + q) * LR + wj + 8 * y + r]);
        }
        __syncthreads();
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int m = m0 + r, j = wj + 8 * y + 2 * q + v;
                const int64_t in = j0 + j - k0;  // column of the block
                sR[m * LR + j] = in >= 0 && in < kb ? sD[m * LC + in] : p[y][v];
            }
    }
    __syncthreads();
    double s[2][4][2];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) s[x][y][0] = s[x][y][1] = 0.0;
#pragma unroll
    for (int k = 0; k < kGJ; k += 4) {
        const double a0 = sC[(wi + r) * LC + k + q], a1 = sC[(wi + 8 + r) * LC + k + q];
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const double bv = sR[(k + q) * LR + wj + 8 * y + r];
            dmma(s[0][y], a0, bv);
            dmma(s[1][y], a1, bv);
        }
    }
    __syncthreads();  // sD is free for the next block
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int ti = wi + 8 * x + r, tj = wj + 8 * y + 2 * q + v;
                const int64_t i = i0 + ti, j = j0 + tj;
                const bool in_r = i >= k0 && i < k0 + kb, in_c = j >= k0 && j < k0 + kb;
                const double w = in_r ? sR[(i - k0) * LR + tj] : in_c ? -s[x][y][v] : own[x][y][v] - s[x][y][v];
                if (i >= n || j >= n) continue;
                const bool nr = i >= kn && i < kn + kGJ, nc = j >= kn && j < kn + kGJ;
                A[i * n + j] = w;
                if (nr) rown[(i - kn) * n + j] = w;
                if (nc) coln[i * kGJ + j - kn] = w;
                if (blockIdx.x == 0 && nr && nc) sD[(i - kn) * LC + j - kn] = w;
            }
    if (blockIdx.x != 0 || kn >= n) return;
    __syncthreads();
    if (threadIdx.x < 128)
        gj_block_inverse<LC>(sD, (int)min((int64_t)kGJ, n - kn), st, buf, dnext, dropped, pivots ? pivots + kn : nullptr);
}

}  // namespace

void GjScratch::drop_graphs()
{
    for (auto &g : graphs)
        if (g.exec) cudaGraphExecDestroy(g.exec);
    graphs.clear();
}

GjScratch::~GjScratch() { drop_graphs(); }

void GjScratch::reserve(int64_t n)
{
    if ((size_t)n > diag.n || (size_t)(2 * kGJ * n) > std::min(rowp.n, colp.n) || !word.p) drop_graphs();  // buffers move
    diag.reserve(n);
    rowp.reserve(2 * kGJ * n);
    colp.reserve(2 * kGJ * n);
    dinv.reserve(2 * kGJ * kGJ);
    word.reserve(1);
}

namespace {
void gj_enqueue(cudaStream_t st, double *A, int64_t n, double rel, GjScratch &w, double *pivots)
{
    cudaMemsetAsync(w.word.p, 0, sizeof(int), st);
    const unsigned gt = (unsigned)((n + kGjTile - 1) / kGjTile);
    double *D[2] = {w.dinv.p, w.dinv.p + kGJ * kGJ}, *R[2] = {w.rowp.p, w.rowp.p + kGJ * n},
           *C[2] = {w.colp.p, w.colp.p + kGJ * n};
    k_gj_first<<<1 + gt, 256, 0, st>>>(A, n, rel, w.diag.p, D[0], R[0], C[0], w.word.p, pivots);
    int p = 0;
    for (int64_t k0 = 0; k0 < n; k0 += kGJ, p ^= 1) {
        const int kb = (int)std::min<int64_t>(kGJ, n - k0);
        k_gj_step<<<gt * gt, 256, 0, st>>>(A, n, k0, kb, w.diag.p, R[p], C[p], R[p ^ 1], C[p ^ 1], D[p], D[p ^ 1],
                                           w.word.p, pivots);
    }
}
}  // namespace

// The launch sequence of one inverse depends only on (A, n, rel, pivots) and
// the scratch buffers, so it is captured once into a CUDA graph and replayed
// (n / 32 + 1 short launches would otherwise be host-bound).
void spd_inverse_gj(sfc_ctx *ctx, double *A, int64_t n, double rel, GjScratch &w, double *pivots, int *dropped)
{
    w.reserve(n);
    const int nlaunch = 1 + (int)((n + kGJ - 1) / kGJ);
    GjScratch::Graph *g = nullptr;
    for (auto &e : w.graphs)
        if (e.A == A && e.n == n && e.rel == rel && e.pivots == pivots) g = &e;
    if (!g) {
        if (w.graphs.size() >= 8) w.drop_graphs();
        cudaStream_t st;
        SFC_CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        cudaGraph_t graph = nullptr;
        cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            gj_enqueue(st, A, n, rel, w, pivots);
            e = cudaStreamEndCapture(st, &graph);
        }
        cudaStreamDestroy(st);
        SFC_CK(e);
        cudaGraphExec_t exec = nullptr;
        e = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        SFC_CK(e);
        w.graphs.push_back({A, n, rel, pivots, exec});
        g = &w.graphs.back();
    }
    SFC_CK(cudaGraphLaunch(g->exec, ctx->stream));
    count_launch(ctx, nlaunch);
    ++ctx->graph_replays;
    int h = 0;
    download(ctx, &h, w.word.p, 1);
    if (dropped) *dropped = h;
}

}  // namespace sfc
