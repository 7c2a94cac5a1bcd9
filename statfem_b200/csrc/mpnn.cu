// Learned preconditioner: a message-passing network on the mesh graph, its
// training on residual/error pairs from plain Jacobi-PCG, and flexible CG.
// (No reference counterpart: the reference solves with Eigen::SparseLU.)
//
// Scaled operator  Ahat = D^-1/2 S D^-1/2  (unit diagonal, FP32 CSR values on
// the matrix pattern; S is the symmetric elimination used by every solver).
// For a residual r:  rhat = D^-1/2 r,  s = rms(rhat),  x0 = rhat / s,
//   H0 = relu(E [x0, Ahat x0] + e)                    encoder, 2 -> 64
//   Hl = relu(Wl [H(l-1) ; Ahat H(l-1)] + bl)         l = 1..3, 128 -> 64
//   y  = w . H3 + c                                   decoder, 64 -> 1
//   M(r) = s D^-1/2 (x0 + y) = D^-1 r + s D^-1/2 y    Jacobi + learned correction
// (y = 0 on constrained dofs, whose rows of S are diagonal: Jacobi is exact).
// The RMS normalisation keeps the node features O(1) whatever the mesh size.
// The aggregation Ahat H is a 64-column SpMM on the operator's pattern.  The
// dense transforms run on the 5th-generation tensor cores (tcgen05.mma,
// BF16 x BF16 -> FP32 in tensor memory): k_layer_tc in inference (gather
// fused), k_dense_fwd_tc and k_dense_bwd_x_tc in training, with the inputs
// rounded to BF16 on the fly, and the weight gradient k_dense_bwd_w_tc as the
// transposed product accumulated over a CTA's node tiles; SFC_MPNN_TC=0
// selects the earlier forms (mma.sync k_layer_inf, k_dense_fwd,
// k_dense_bwd_x, and the FP32 reduction k_dense_bwd_w) for comparison.
// Activations in training, master weights, gradients and Adam state are FP32.
//
// Training pair (r, e) with S e = r: target t = D^1/2 e / s, d = x0 + y - t,
// loss L = d^T Ahat d / N (the S-norm of the error of M(r) scaled by 1/(N s^2)).
// Pairs come from x_k of Jacobi-PCG started at 0: r_k = b - S x_k,
// e_k = x* - x_k, x* the converged solution.

#include <cuda_bf16.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <new>
#include <random>
#include <vector>

#include "pcg.cuh"

namespace {

constexpr int H = 64;                 // hidden width
constexpr int LAYERS = 3;             // message-passing layers
constexpr int OFF_EW = 0;             // encoder weights [64][2]
constexpr int OFF_EB = OFF_EW + 2 * H;
constexpr int OFF_L = OFF_EB + H;     // layer l: W [64][128] then b [64]
constexpr int LSZ = H * 2 * H + H;
constexpr int OFF_DW = OFF_L + LAYERS * LSZ;
constexpr int OFF_DB = OFF_DW + H;
constexpr int NPARAM = OFF_DB + 1;

}  // namespace

struct sfc_mpnn {
    sfc_ctx *ctx = nullptr;
    int64_t step = 0;
    sfc::DBuf<float> params, grads, adam_m, adam_v;
    sfc::DBuf<__nv_bfloat16> wbf;  // LAYERS x [64][128] BF16 copies, then their transposes
    // operator-dependent data (for the system the network was last used on)
    const sfc_system *op_sys = nullptr;
    int64_t N = 0;
    sfc::DBuf<float> ahat, sdinv;
    // activations and gradients
    sfc::DBuf<float> x0, ax0, yhat, dvec, qvec, H[LAYERS + 1], Y[LAYERS + 1], dH0, dH1, dY;
    sfc::DBuf<__nv_bfloat16> hb[2];  // inference activations (BF16, ping-pong)
    sfc::DBuf<int> tc_err;           // bounded-wait status of the tensor-core layers
    sfc::DBuf<double> fcg_sc;        // flexible-CG scalars, per iteration
    sfc::DBuf<int> fcg_flags;        // done, breakdown; k_fcg: its `out`
    sfc::DBuf<float> win;            // scaled operator by windows of columns (k_fcg)
    sfc::DBuf<__nv_bfloat16> hw[2];  // activations for those, with a margin of zeros
    sfc::DBuf<double> io[2];  // operands of the host entry points, kept between calls
    sfc::DBuf<double> scal;  // [0]: N s^2 = |D^-1/2 r|^2, [1]: loss
    // training pairs (FP64, N each)
    sfc::DBuf<double> pr, pe;
    std::vector<double> pw;  // per-pair loss weights
    int npairs = 0;
};

namespace sfc {
namespace {

__device__ __forceinline__ float warp_sumf(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // .x (low half) = lo
    return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// D (16x8, f32) += A (16x16, bf16, row) * B (16x8, bf16, col)
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---- operator scaling --------------------------------------------------------
// (8 lanes per row: a thread per row followed a chain of a square root and a
// division per entry, 25 us for 15,625 nodes of a cube)
__global__ void k_scale_op(const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                           const int32_t *__restrict__ diag, const double *__restrict__ a, int64_t N,
                           float *__restrict__ ahat, float *__restrict__ sdinv)
{
    const int fl = threadIdx.x & 7;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3; i < N; i += ((int64_t)gridDim.x * blockDim.x) >> 3) {
        const double si = 1.0 / sqrt(a[diag[i]]);
        if (fl == 0) sdinv[i] = (float)si;
        for (int32_t s = rp[i] + fl; s < rp[i + 1]; s += 8) ahat[s] = (float)(a[s] * si / sqrt(a[diag[col[s]]]));
    }
}

// Ahat x (one column), warp per row, then what its value is for:
// ENC: y = Ahat x and H0 = relu(E [x, y] + e), two features per lane;
// else: y = g2 Ahat x with g2 = 2 w / N, *loss += w x . Ahat x / N
template <bool ENC>
__global__ void __launch_bounds__(256) k_spmv32(const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                                                const float *__restrict__ v, const float *__restrict__ x,
                                                float *__restrict__ y, int64_t N, const float *__restrict__ P,
                                                float *__restrict__ H0, double w, double *loss)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const float g2 = (float)(2.0 * w / (double)N);
    const double invn = w / (double)N;
    double part = 0.0;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; i < N; i += warps) {
        float s = 0.f;
        for (int32_t k = rp[i] + lane; k < rp[i + 1]; k += 32) s = fmaf(v[k], x[col[k]], s);
        s = warp_sumf(s);
        if constexpr (ENC) {
            if (lane == 0) y[i] = s;
            const float xi = x[i];
            const float *E = P + OFF_EW + 4 * lane, *e = P + OFF_EB + 2 * lane;
            *reinterpret_cast<float2 *>(H0 + i * H + 2 * lane) =
                make_float2(fmaxf(fmaf(E[0], xi, fmaf(E[1], s, e[0])), 0.f), fmaxf(fmaf(E[2], xi, fmaf(E[3], s, e[1])), 0.f));
        } else if (lane == 0) {
            part += (double)x[i] * (double)s * invn;
            y[i] = s * g2;
        }
    }
    if constexpr (!ENC) {
        __shared__ double sh[8];
        if (lane == 0) sh[threadIdx.x >> 5] = part;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < (int)(blockDim.x >> 5); ++k) part += sh[k];
            atomicAdd(loss, part);
        }
    }
}

// Y (+)= Ahat X for 64 feature columns: 16 lanes per row, four features each.
// Bound by the latency of the activation rows' loads (256 bytes each): eight
// are in flight at a time, and the next eight columns and weights on their way.
__global__ void __launch_bounds__(1024, 1) k_agg64(const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                                               const float *__restrict__ v, const float *__restrict__ X,
                                               float *__restrict__ Y, int64_t N, int accumulate)
{
    const int lane = threadIdx.x & 31, fl = lane & 15;
    // a CTA takes consecutive rows: they share most of their neighbours' lines
    const int64_t per = ((N + gridDim.x - 1) / gridDim.x + 1) / 2 * 2, row0 = blockIdx.x * per, row1 = min(N, row0 + per);
    const float4 *X4 = reinterpret_cast<const float4 *>(X);
    // both rows of a warp take every trip: the columns are shuffled
    for (int64_t base = row0 + (threadIdx.x >> 5) * 2; base < row1; base += blockDim.x >> 4) {
        const int64_t i = base + (lane >> 4);
        const int32_t b = i < row1 ? rp[i] : 0, len = i < row1 ? rp[i + 1] - b : 0;
        const int maxlen = max(len, __shfl_xor_sync(0xffffffffu, len, 16));
        float4 *out = reinterpret_cast<float4 *>(Y) + i * 16 + fl;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f), old = acc;
        if (accumulate && i < row1) old = *out;
        int32_t cv = fl < min(len, 8) ? col[b + fl] : 0;  // padding: row 0 with weight 0
        float av = fl < min(len, 8) ? v[b + fl] : 0.f;
        for (int s0 = 0; s0 < maxlen; s0 += 8) {
            const int sn = s0 + 8 + fl;
            const int32_t cvn = fl < 8 && sn < len ? col[b + sn] : 0;
            const float avn = fl < 8 && sn < len ? v[b + sn] : 0.f;
            float4 u[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) u[j] = X4[(int64_t)__shfl_sync(0xffffffffu, cv, j, 16) * 16 + fl];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float aj = __shfl_sync(0xffffffffu, av, j, 16);
                if (s0 + j < len) {
                    acc.x = fmaf(aj, u[j].x, acc.x);
                    acc.y = fmaf(aj, u[j].y, acc.y);
                    acc.z = fmaf(aj, u[j].z, acc.z);
                    acc.w = fmaf(aj, u[j].w, acc.w);
                }
            }
            cv = cvn;
            av = avn;
        }
        if (i < row1) *out = make_float4(acc.x + old.x, acc.y + old.y, acc.z + old.z, acc.w + old.w);
    }
}

// x0 = D^-1/2 r / s  (N s^2 in scal[0])
__global__ void k_x0(const double *__restrict__ r, const float *__restrict__ sdinv, const double *scal, int64_t N,
                     float *__restrict__ x0)
{
    const double inv = scal[0] > 0 ? 1.0 / sqrt(scal[0] / (double)N) : 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
        x0[i] = (float)(r[i] * (double)sdinv[i] * inv);
}

// scal[slot] += sum (D^-1/2 v)^2
// (and rhat = FP32(D^-1/2 v) when rhat != NULL)
__global__ void k_scaled_norm2(const double *__restrict__ v, const float *__restrict__ sdinv, int64_t N, double *out,
                               float *__restrict__ rhat = nullptr)
{
    __shared__ double sh[32];
    double s = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
        const double t = v[i] * (double)sdinv[i];
        s += t * t;
        if (rhat) rhat[i] = (float)t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) atomicAdd(out, s);
    }
}

// Hout = relu([Hin | Yin] W^T + b), 16 nodes per warp, BF16 mma, FP32 accumulate
__global__ void __launch_bounds__(256) k_dense_fwd(const float *__restrict__ Hin, const float *__restrict__ Yin,
                                                   const __nv_bfloat16 *__restrict__ W, const float *__restrict__ bias,
                                                   int64_t N, float *__restrict__ Hout)
{
    __shared__ __align__(16) __nv_bfloat16 sW[H * 2 * H];
    for (int t = threadIdx.x; t < H * 2 * H; t += blockDim.x) sW[t] = W[t];
    __syncthreads();
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int64_t tiles = (N + 15) / 16;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t tile = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; tile < tiles; tile += warps) {
        const int64_t r0 = tile * 16 + gid, r1 = r0 + 8;
        float acc[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[nt][q] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            const float *src = ks < 4 ? Hin : Yin;
            const int c0 = (ks & 3) * 16 + tig * 2, c1 = c0 + 8;
            float2 v00 = make_float2(0.f, 0.f), v01 = v00, v10 = v00, v11 = v00;
            if (r0 < N) {
                v00 = *reinterpret_cast<const float2 *>(src + r0 * H + c0);
                v01 = *reinterpret_cast<const float2 *>(src + r0 * H + c1);
            }
            if (r1 < N) {
                v10 = *reinterpret_cast<const float2 *>(src + r1 * H + c0);
                v11 = *reinterpret_cast<const float2 *>(src + r1 * H + c1);
            }
            const uint32_t a[4] = {pack_bf16(v00.x, v00.y), pack_bf16(v10.x, v10.y), pack_bf16(v01.x, v01.y),
                                   pack_bf16(v11.x, v11.y)};
            const int k = ks * 16 + tig * 2;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const int n = nt * 8 + gid;
                const uint32_t b0 = *reinterpret_cast<const uint32_t *>(&sW[n * 2 * H + k]);
                const uint32_t b1 = *reinterpret_cast<const uint32_t *>(&sW[n * 2 * H + k + 8]);
                mma16816(acc[nt], a, b0, b1);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int c = nt * 8 + tig * 2;
            const float b0 = bias[c], b1 = bias[c + 1];
            if (r0 < N)
                *reinterpret_cast<float2 *>(Hout + r0 * H + c) =
                    make_float2(fmaxf(acc[nt][0] + b0, 0.f), fmaxf(acc[nt][1] + b1, 0.f));
            if (r1 < N)
                *reinterpret_cast<float2 *>(Hout + r1 * H + c) =
                    make_float2(fmaxf(acc[nt][2] + b0, 0.f), fmaxf(acc[nt][3] + b1, 0.f));
        }
    }
}

// yhat = x0 + (w . H3 + c) on free dofs, x0 on constrained ones; warp per node
__global__ void k_decoder(const float *__restrict__ H3, const float *__restrict__ P, const float *__restrict__ x0,
                          const unsigned char *__restrict__ mask, int64_t N, float *__restrict__ yhat)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const float w0 = P[OFF_DW + 2 * lane], w1 = P[OFF_DW + 2 * lane + 1], c = P[OFF_DB];
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; i < N; i += warps) {
        const float2 h = *reinterpret_cast<const float2 *>(H3 + i * H + 2 * lane);
        const float s = warp_sumf(fmaf(w0, h.x, w1 * h.y));
        if (lane == 0) yhat[i] = mask[i] ? x0[i] : x0[i] + s + c;
    }
}

// d = yhat - t with the target t = D^1/2 e / s
__global__ void k_target_diff(const double *__restrict__ e, const float *__restrict__ sdinv, const double *scal,
                              const float *__restrict__ yhat, int64_t N, float *__restrict__ d)
{
    const double inv = scal[0] > 0 ? 1.0 / sqrt(scal[0] / (double)N) : 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
        d[i] = yhat[i] - (float)(e[i] / (double)sdinv[i] * inv);
}

// decoder backward: dH3 = g w ; dw += sum_i g_i H3_i ; dc += sum g_i
// (the block's sums first: an atomic per warp and parameter, on 65 addresses,
// took 101 us for 15,625 nodes)
__global__ void __launch_bounds__(256) k_decoder_bwd(const float *__restrict__ g, const float *__restrict__ H3, const float *__restrict__ P,
                              const unsigned char *__restrict__ mask, int64_t N, float *__restrict__ dH3,
                              float *__restrict__ G)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const float w0 = P[OFF_DW + 2 * lane], w1 = P[OFF_DW + 2 * lane + 1];
    float a0 = 0.f, a1 = 0.f, ac = 0.f;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; i < N; i += warps) {
        const float gi = mask[i] ? 0.f : g[i];
        const float2 h = *reinterpret_cast<const float2 *>(H3 + i * H + 2 * lane);
        *reinterpret_cast<float2 *>(dH3 + i * H + 2 * lane) = make_float2(gi * w0, gi * w1);
        a0 = fmaf(gi, h.x, a0);
        a1 = fmaf(gi, h.y, a1);
        ac += gi;
    }
    __shared__ float sh[8][H + 1];
    const int warp = threadIdx.x >> 5;
    sh[warp][2 * lane] = a0;
    sh[warp][2 * lane + 1] = a1;
    if (lane == 0) sh[warp][H] = ac;
    __syncthreads();
    static_assert(OFF_DB == OFF_DW + H, "weights, then the bias");
    if (threadIdx.x <= H) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) s += sh[k][threadIdx.x];
        atomicAdd(&G[OFF_DW + threadIdx.x], s);
    }
}

// input gradient of a dense layer: dZ = dH * (Hl > 0) (BF16),
// [dHprev | dY] = dZ W  (16 nodes per warp, mma, FP32 accumulate)
__global__ void __launch_bounds__(256) k_dense_bwd_x(const float *__restrict__ dH, const float *__restrict__ Hl,
                                                     const __nv_bfloat16 *__restrict__ W, int64_t N,
                                                     float *__restrict__ dHprev, float *__restrict__ dY)
{
    __shared__ __align__(16) __nv_bfloat16 sW[H * 2 * H];
    for (int t = threadIdx.x; t < H * 2 * H; t += blockDim.x) sW[t] = W[t];
    __syncthreads();
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int64_t tiles = (N + 15) / 16;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t tile = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; tile < tiles; tile += warps) {
        const int64_t r0 = tile * 16 + gid, r1 = r0 + 8;
        float acc[16][4];
#pragma unroll
        for (int nt = 0; nt < 16; ++nt)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[nt][q] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            const int c0 = ks * 16 + tig * 2, c1 = c0 + 8;
            float v[4][2] = {};
            if (r0 < N) {
                const float2 d0 = *reinterpret_cast<const float2 *>(dH + r0 * H + c0);
                const float2 d1 = *reinterpret_cast<const float2 *>(dH + r0 * H + c1);
                const float2 h0 = *reinterpret_cast<const float2 *>(Hl + r0 * H + c0);
                const float2 h1 = *reinterpret_cast<const float2 *>(Hl + r0 * H + c1);
                v[0][0] = h0.x > 0.f ? d0.x : 0.f;
                v[0][1] = h0.y > 0.f ? d0.y : 0.f;
                v[2][0] = h1.x > 0.f ? d1.x : 0.f;
                v[2][1] = h1.y > 0.f ? d1.y : 0.f;
            }
            if (r1 < N) {
                const float2 d0 = *reinterpret_cast<const float2 *>(dH + r1 * H + c0);
                const float2 d1 = *reinterpret_cast<const float2 *>(dH + r1 * H + c1);
                const float2 h0 = *reinterpret_cast<const float2 *>(Hl + r1 * H + c0);
                const float2 h1 = *reinterpret_cast<const float2 *>(Hl + r1 * H + c1);
                v[1][0] = h0.x > 0.f ? d0.x : 0.f;
                v[1][1] = h0.y > 0.f ? d0.y : 0.f;
                v[3][0] = h1.x > 0.f ? d1.x : 0.f;
                v[3][1] = h1.y > 0.f ? d1.y : 0.f;
            }
            const uint32_t a[4] = {pack_bf16(v[0][0], v[0][1]), pack_bf16(v[1][0], v[1][1]),
                                   pack_bf16(v[2][0], v[2][1]), pack_bf16(v[3][0], v[3][1])};
            const int k = ks * 16 + tig * 2;  // output-feature index of W rows
#pragma unroll
            for (int nt = 0; nt < 16; ++nt) {
                const int n = nt * 8 + gid;  // input-feature index (0..127)
                const uint32_t b0 = (uint32_t) * reinterpret_cast<const uint16_t *>(&sW[k * 2 * H + n]) |
                                    ((uint32_t) * reinterpret_cast<const uint16_t *>(&sW[(k + 1) * 2 * H + n]) << 16);
                const uint32_t b1 =
                    (uint32_t) * reinterpret_cast<const uint16_t *>(&sW[(k + 8) * 2 * H + n]) |
                    ((uint32_t) * reinterpret_cast<const uint16_t *>(&sW[(k + 9) * 2 * H + n]) << 16);
                mma16816(acc[nt], a, b0, b1);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 16; ++nt) {
            const int c = nt * 8 + tig * 2;
            float *dst = c < H ? dHprev : dY;
            const int cc = c < H ? c : c - H;
            if (r0 < N) *reinterpret_cast<float2 *>(dst + r0 * H + cc) = make_float2(acc[nt][0], acc[nt][1]);
            if (r1 < N) *reinterpret_cast<float2 *>(dst + r1 * H + cc) = make_float2(acc[nt][2], acc[nt][3]);
        }
    }
}

// weight gradient of a dense layer: dW[o][j] += sum_i dZ[i][o] Xc[i][j] with
// dZ and Xc = [Hin | Yin] rounded to BF16 (the operands of the tensor-core
// products), db[o] += sum_i dZ[i][o] unrounded; FP32 accumulate
constexpr int kTN = 32;
__global__ void __launch_bounds__(256) k_dense_bwd_w(const float *__restrict__ dH, const float *__restrict__ Hl,
                                                     const float *__restrict__ Hin, const float *__restrict__ Yin,
                                                     int64_t N, float *__restrict__ GW, float *__restrict__ Gb)
{
    __shared__ float sZ[kTN][H];
    __shared__ float sX[kTN][2 * H + 1];
    const int o = threadIdx.x >> 2, jq = threadIdx.x & 3;  // 64 outputs x 4 interleaved input groups
    float acc[32];
#pragma unroll
    for (int u = 0; u < 32; ++u) acc[u] = 0.f;
    float accb = 0.f;
    for (int64_t n0 = (int64_t)blockIdx.x * kTN; n0 < N; n0 += (int64_t)gridDim.x * kTN) {
        __syncthreads();
        for (int t = threadIdx.x; t < kTN * H; t += blockDim.x) {
            const int ii = t / H, k = t % H;
            const int64_t i = n0 + ii;
            float z = 0.f;
            if (i < N) z = Hl[i * H + k] > 0.f ? dH[i * H + k] : 0.f;
            sZ[ii][k] = z;
        }
        for (int t = threadIdx.x; t < kTN * 2 * H; t += blockDim.x) {
            const int ii = t / (2 * H), j = t % (2 * H);
            const int64_t i = n0 + ii;
            float x = 0.f;
            if (i < N) x = j < H ? Hin[i * H + j] : Yin[i * H + j - H];
            sX[ii][j] = bf16r(x);
        }
        __syncthreads();
        for (int ii = 0; ii < kTN; ++ii) {
            const float z0 = sZ[ii][o], z = bf16r(z0);
            if (jq == 0) accb += z0;
#pragma unroll
            for (int u = 0; u < 32; ++u) acc[u] = fmaf(z, sX[ii][u * 4 + jq], acc[u]);
        }
    }
#pragma unroll
    for (int u = 0; u < 32; ++u) atomicAdd(&GW[o * 2 * H + u * 4 + jq], acc[u]);
    if (jq == 0) atomicAdd(&Gb[o], accb);
}

// (the block's sums first, as above: 53 us with an atomic per thread)
__global__ void __launch_bounds__(256) k_encoder_bwd(const float *__restrict__ dH0, const float *__restrict__ H0, const float *__restrict__ x0,
                              const float *__restrict__ ax0, int64_t N, float *__restrict__ G)
{
    // thread owns feature k = threadIdx.x & 63 for its node stride
    const int k = threadIdx.x & (H - 1);
    float a0 = 0.f, a1 = 0.f, ab = 0.f;
    const int64_t lanes = (int64_t)gridDim.x * (blockDim.x / H);
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / H; i < N; i += lanes) {
        const float z = H0[i * H + k] > 0.f ? dH0[i * H + k] : 0.f;
        a0 = fmaf(z, x0[i], a0);
        a1 = fmaf(z, ax0[i], a1);
        ab += z;
    }
    __shared__ float sh[3][256];
    sh[0][threadIdx.x] = a0;
    sh[1][threadIdx.x] = a1;
    sh[2][threadIdx.x] = ab;
    __syncthreads();
    const int w = threadIdx.x >> 6;
    if (w < 3) {
        const float s = (sh[w][k] + sh[w][k + H]) + (sh[w][k + 2 * H] + sh[w][k + 3 * H]);
        atomicAdd(&G[w < 2 ? OFF_EW + 2 * k + w : OFF_EB + k], s);
    }
}

__global__ void k_adam(float *__restrict__ P, const float *__restrict__ G, float *__restrict__ m,
                       float *__restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2,
                       float clip)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        float g = fminf(fmaxf(G[t], -clip), clip);
        m[t] = b1 * m[t] + (1.f - b1) * g;
        v[t] = b2 * v[t] + (1.f - b2) * g * g;
        P[t] -= lr * (m[t] / c1) / (sqrtf(v[t] / c2) + eps);
    }
}

__global__ void k_to_bf16(const float *__restrict__ P, __nv_bfloat16 *__restrict__ wbf)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < LAYERS * H * 2 * H; t += gridDim.x * blockDim.x) {
        const int l = t / (H * 2 * H), r = t % (H * 2 * H);
        const __nv_bfloat16 w = __float2bfloat16_rn(P[OFF_L + l * LSZ + r]);
        wbf[t] = w;
        wbf[LAYERS * H * 2 * H + l * H * 2 * H + (r % (2 * H)) * H + r / (2 * H)] = w;  // and its transpose
    }
}

// ---- inference: BF16 activations, gather fused with the dense transform --------
// The stored activations are the BF16 values the tensor-core products round
// them to anyway; the aggregation reads them (half the gather traffic of
// FP32) and accumulates in FP32.
constexpr int kLS = 68;  // shared-memory row stride in 32-bit words (136 BF16): conflict-free fragments

__device__ __forceinline__ float2 bf16x2_to_f2(uint32_t u)
{
    __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162 *>(&u);
    return __bfloat1622float2(v);
}

// x0 = rhat / s, H0 = BF16(relu(E [x0, Ahat x0] + e)) with Ahat x0 =
// (Ahat rhat) / s; 8 lanes per node (8 features each), 4 nodes per warp trip.
// Bound by the latency of row pointer -> column -> value, so the entries of a
// row go out four per lane at a time (32 of a row in flight, the 27-entry rows
// of a 3-D mesh in one go).
__global__ void k_encoder_inf(const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                              const float *__restrict__ v, const float *__restrict__ rhat, const double *scal,
                              const float *__restrict__ P, int64_t N, float *__restrict__ x0, uint4 *__restrict__ H0)
{
    const int lane = threadIdx.x & 31, sub = lane >> 3, fl = lane & 7;
    const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const float inv = scal[0] > 0 ? (float)(1.0 / sqrt(scal[0] / (double)N)) : 0.f;
    float e0[8], e1[8], eb[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        e0[q] = P[OFF_EW + 2 * (fl * 8 + q)];
        e1[q] = P[OFF_EW + 2 * (fl * 8 + q) + 1];
        eb[q] = P[OFF_EB + fl * 8 + q];
    }
    for (int64_t base = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 4; base < N; base += nwarps * 4) {
        const int64_t i = base + sub;
        const bool valid = i < N;
        float acc = 0.f;
        const int32_t b = valid ? rp[i] : 0, e = valid ? rp[i + 1] : 0;
        for (int32_t k = b + fl; k < e; k += 32) {
            int32_t c[4];
            float a[4], x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool in = k + 8 * u < e;
                c[u] = in ? col[k + 8 * u] : -1;
                a[u] = in ? v[k + 8 * u] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = c[u] >= 0 ? rhat[c[u]] : 0.f;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c[u] >= 0) acc = fmaf(a[u], x[u], acc);
        }
        acc += __shfl_xor_sync(0xffffffffu, acc, 4);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        if (!valid) continue;
        const float xi = rhat[i] * inv, ax = acc * inv;
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            w[q] = pack_bf16(fmaxf(fmaf(e0[2 * q], xi, fmaf(e1[2 * q], ax, eb[2 * q])), 0.f),
                             fmaxf(fmaf(e0[2 * q + 1], xi, fmaf(e1[2 * q + 1], ax, eb[2 * q + 1])), 0.f));
        H0[i * 8 + fl] = make_uint4(w[0], w[1], w[2], w[3]);
        if (fl == 0) x0[i] = xi;
    }
}

// One message-passing layer, 16 nodes per warp: gather Ahat Hin for the
// tile's rows into shared memory beside the rows of Hin, then
// [Hin | Ahat Hin] W^T on BF16 mma fragments (FP32 accumulate), bias, relu.
// DECODE (last layer): instead of storing H, z = s D^-1/2 (x0 + w . H + c)
// (x0 alone on constrained dofs).
template <bool DECODE>
__global__ void __launch_bounds__(128) k_layer_inf(const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                                                   const float *__restrict__ v, const uint32_t *__restrict__ Hin,
                                                   const __nv_bfloat16 *__restrict__ W, const float *__restrict__ bias,
                                                   int64_t N, uint32_t *__restrict__ Hout,
                                                   const float *__restrict__ P, const float *__restrict__ x0,
                                                   const float *__restrict__ sdinv,
                                                   const unsigned char *__restrict__ mask, const double *scal,
                                                   double *__restrict__ z)
{
    __shared__ __align__(16) uint32_t sW[H * kLS];
    __shared__ __align__(16) uint32_t sA[4][16 * kLS];
    const uint32_t *W32 = reinterpret_cast<const uint32_t *>(W);
    for (int t = threadIdx.x; t < H * H; t += blockDim.x) sW[(t / H) * kLS + (t % H)] = W32[t];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    uint32_t *tileA = sA[warp];
    const int64_t tiles = (N + 15) / 16;
    const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t tile = blockIdx.x * (int64_t)(blockDim.x >> 5) + warp; tile < tiles; tile += nwarps) {
        // gather: 8 lanes per row (8 features = 16 bytes each), 4 rows at a
        // time, 8 neighbours per trip with independent loads
        const int sub = lane >> 3, fl = lane & 7;
        const uint4 *Hin4 = reinterpret_cast<const uint4 *>(Hin);
        for (int pass = 0; pass < 4; ++pass) {
            const int rr = pass * 4 + sub;
            const int64_t i = tile * 16 + rr;
            const bool valid = i < N;
            const int32_t b = valid ? rp[i] : 0;
            const int len = valid ? rp[i + 1] - b : 0;
            int maxlen = len;
            maxlen = max(maxlen, __shfl_xor_sync(0xffffffffu, maxlen, 8));
            maxlen = max(maxlen, __shfl_xor_sync(0xffffffffu, maxlen, 16));
            float acc[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[q] = 0.f;
            for (int s0 = 0; s0 < maxlen; s0 += 8) {
                const int sl = s0 + fl;
                const int32_t cv = sl < len ? col[b + sl] : 0;  // padding: row 0 with weight 0
                const float av = sl < len ? v[b + sl] : 0.f;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int32_t cj = __shfl_sync(0xffffffffu, cv, j, 8);
                    const float aj = __shfl_sync(0xffffffffu, av, j, 8);
                    const uint4 u = Hin4[(int64_t)cj * 8 + fl];
                    const float2 f0 = bf16x2_to_f2(u.x), f1 = bf16x2_to_f2(u.y), f2 = bf16x2_to_f2(u.z),
                                 f3 = bf16x2_to_f2(u.w);
                    acc[0] = fmaf(aj, f0.x, acc[0]);
                    acc[1] = fmaf(aj, f0.y, acc[1]);
                    acc[2] = fmaf(aj, f1.x, acc[2]);
                    acc[3] = fmaf(aj, f1.y, acc[3]);
                    acc[4] = fmaf(aj, f2.x, acc[4]);
                    acc[5] = fmaf(aj, f2.y, acc[5]);
                    acc[6] = fmaf(aj, f3.x, acc[6]);
                    acc[7] = fmaf(aj, f3.y, acc[7]);
                }
            }
            const uint4 hv = valid ? Hin4[i * 8 + fl] : make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4 *>(&tileA[rr * kLS + fl * 4]) = hv;
            *reinterpret_cast<uint4 *>(&tileA[rr * kLS + 32 + fl * 4]) =
                make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]),
                           pack_bf16(acc[6], acc[7]));
        }
        __syncwarp();
        float acc[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[nt][q] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            const int kw = ks * 8 + tig;  // 32-bit word of columns (k, k+1), k = ks*16 + 2*tig
            const uint32_t a[4] = {tileA[gid * kLS + kw], tileA[(gid + 8) * kLS + kw], tileA[gid * kLS + kw + 4],
                                   tileA[(gid + 8) * kLS + kw + 4]};
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const int n = nt * 8 + gid;
                mma16816(acc[nt], a, sW[n * kLS + kw], sW[n * kLS + kw + 4]);
            }
        }
        __syncwarp();
        if constexpr (!DECODE) {
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const int c = nt * 8 + tig * 2;
                const float b0 = bias[c], b1 = bias[c + 1];
                tileA[gid * kLS + c / 2] = pack_bf16(fmaxf(acc[nt][0] + b0, 0.f), fmaxf(acc[nt][1] + b1, 0.f));
                tileA[(gid + 8) * kLS + c / 2] = pack_bf16(fmaxf(acc[nt][2] + b0, 0.f), fmaxf(acc[nt][3] + b1, 0.f));
            }
            __syncwarp();
            for (int rr = 0; rr < 16; ++rr) {
                const int64_t i = tile * 16 + rr;
                if (i < N) Hout[i * (H / 2) + lane] = tileA[rr * kLS + lane];
            }
            __syncwarp();
        } else {
            float y0 = 0.f, y1 = 0.f;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const int c = nt * 8 + tig * 2;
                const float b0 = bias[c], b1 = bias[c + 1], w0 = P[OFF_DW + c], w1 = P[OFF_DW + c + 1];
                y0 = fmaf(w0, fmaxf(acc[nt][0] + b0, 0.f), fmaf(w1, fmaxf(acc[nt][1] + b1, 0.f), y0));
                y1 = fmaf(w0, fmaxf(acc[nt][2] + b0, 0.f), fmaf(w1, fmaxf(acc[nt][3] + b1, 0.f), y1));
            }
            y0 += __shfl_xor_sync(0xffffffffu, y0, 1);
            y0 += __shfl_xor_sync(0xffffffffu, y0, 2);
            y1 += __shfl_xor_sync(0xffffffffu, y1, 1);
            y1 += __shfl_xor_sync(0xffffffffu, y1, 2);
            if (tig == 0) {
                const double sc = sqrt(scal[0] / (double)N);
                const float c0 = P[OFF_DB];
                const int64_t i0 = tile * 16 + gid, i1 = i0 + 8;
                if (i0 < N) z[i0] = sc * (double)sdinv[i0] * (double)(mask[i0] ? x0[i0] : x0[i0] + y0 + c0);
                if (i1 < N) z[i1] = sc * (double)sdinv[i1] * (double)(mask[i1] ? x0[i1] : x0[i1] + y1 + c0);
            }
        }
    }
}

// ---- inference on the 5th-generation tensor cores (tcgen05) ---------------------
// A CTA of eight warps takes up to 128 nodes at a time: the warps gather the tile's
// [Hin | Ahat Hin] rows (BF16, K = 128) into shared memory in the canonical
// K-major layout without swizzle (8-row x 16-byte core matrices: core (row
// group g, K chunk c) at byte (16 g + c) * 128, so the next K chunk is 128
// bytes on (LBO) and the next 8-row group 2,048 bytes on (SBO)); W (64 x 128,
// K-major) sits beside it in the same layout for the whole kernel.  One thread
// issues eight tcgen05.mma (M = 128, N = 64, K = 16, BF16 x BF16 -> FP32)
// into a 64-column accumulator in tensor memory and commits them to an
// mbarrier; warps w and w + 4 then read the 32 rows of TMEM lanes 32 (w % 4)
// .. with tcgen05.ld, columns 0-31 and 32-63 respectively, add the bias, apply
// relu and store BF16 rows (or, DECODE, the decoded correction z).  The mbarrier wait is bounded: on a timeout the
// kernel sets *err, waits once more (bounded) for the MMAs in flight, frees
// its tensor memory and leaves.  Bound by the gather: 128 bytes per matrix
// entry through L1, about half of it from L2 (39,304 nodes of a cube, a layer
// 32.6 -> 25.6 us with the next trip's indices prefetched, packed FP32 FMAs,
// the tiles spread over all CTAs and neighbouring tiles on one SM).
constexpr int kTcRows = 128;           // nodes per tile (MMA M)
constexpr uint32_t kTcCols = 64;       // accumulator columns (MMA N), tensor-memory columns allocated
constexpr int kTcBBytes = H * 2 * H * 2;      // W: 16 KiB
constexpr int kTcABytes = kTcRows * 2 * H * 2;  // A tile: 32 KiB
// k_layer_tc: bytes from the tile's first row to W, and of the whole (+ mbarrier + tensor-memory address).  A tile of
// fewer rows leaves the rest to L1, but W's end has to lie behind 128 rows
__host__ __device__ constexpr int tc_layer_a(int rows)
{
    return (rows < kTcRows / 2 ? kTcRows / 2 : rows) * 2 * H * 2;
}
constexpr size_t tc_layer_smem(int rows) { return (size_t)tc_layer_a(rows) + kTcBBytes + 16; }
static_assert(tc_layer_a(8) + kTcBBytes >= kTcABytes, "128 rows lie within the tile and W");
constexpr uint32_t kTcWaitTries = 1u << 22;
// instruction descriptor: FP32 accumulator (bits 4-5 = 1), A and B BF16 (bits
// 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
constexpr uint32_t kTcIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kTcCols >> 3) << 17) | ((uint32_t)(kTcRows >> 4) << 24);
static_assert(kTcIdesc == (1u << 4) + (1u << 7) + (1u << 10) + (8u << 17) + (8u << 24), "M = 128, N = 64");

// byte offset of the 16-byte piece (row, K chunk) of a K-major operand with KC
// chunks of 8 BF16 per row in the canonical layout (core matrix = 8 rows of
// one chunk, 128 bytes; next chunk +128 B; next 8-row group + 128 KC B)
template <int KC = 16>
__device__ __forceinline__ uint32_t tc_off(int row, int chunk)
{
    return (uint32_t)(((row >> 3) * KC + chunk) * 128 + (row & 7) * 16);
}

// shared-memory matrix descriptor: start address, LBO = 128 B (next K chunk),
// SBO = 128 KC B (next 8-row group), all in 16-byte units; descriptor version
// 1, no swizzle
template <int KC = 16>
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) |
           ((uint64_t)((128u * KC) >> 4) << 32) | (1ull << 46);
}

// instruction descriptor of a BF16 x BF16 -> FP32 MMA, both operands K-major
constexpr uint32_t tc_idesc(uint32_t M, uint32_t N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity)
{
    for (uint32_t i = 0; i < kTcWaitTries; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t u[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
          "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
        : "r"(taddr));
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(u[j]);
}

// two FP32 values in a 64-bit register (fma.rn.f32x2: each half rounds as fmaf)
__device__ __forceinline__ unsigned long long f2_pack(float a)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}

__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b, unsigned long long c)
{
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ unsigned long long bf16x2_to_f2b(uint32_t u)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(u << 16), "r"(u & 0xffff0000u));
    return r;
}

__device__ __forceinline__ uint32_t f2_bf16(unsigned long long a)
{
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a));
    return pack_bf16(lo, hi);
}

template <bool DECODE>
__global__ void __launch_bounds__(256, 4) k_layer_tc(const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                                                     const float *__restrict__ v, const uint32_t *__restrict__ Hin,
                                                     const __nv_bfloat16 *__restrict__ W,
                                                     const float *__restrict__ bias, int64_t N, int rows, int sms,
                                                     uint32_t *__restrict__ Hout, const float *__restrict__ P,
                                                     const float *__restrict__ x0, const float *__restrict__ sdinv,
                                                     const unsigned char *__restrict__ mask, const double *scal,
                                                     double *__restrict__ z, int *err)
{
    extern __shared__ __align__(1024) unsigned char tsm[];
    // the tile's rows, then W: the MMA's M = 128 reads on past `rows` into W,
    // results that nobody takes
    unsigned char *sA = tsm, *sB = tsm + tc_layer_a(rows);
    uint64_t *bar = reinterpret_cast<uint64_t *>(sB + kTcBBytes);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(sB + kTcBBytes + 8);
    __shared__ __align__(16) float sbias[H], sdec[H];
    if (threadIdx.x < H) {
        sbias[threadIdx.x] = bias[threadIdx.x];
        if constexpr (DECODE) sdec[threadIdx.x] = P[OFF_DW + threadIdx.x];
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t sA_u = (uint32_t)__cvta_generic_to_shared(sA), sB_u = (uint32_t)__cvta_generic_to_shared(sB);
    const uint32_t bar_u = (uint32_t)__cvta_generic_to_shared(bar);
    // W (row n = output feature, 16 chunks of 8 K values) into the canonical layout
    const uint4 *W4 = reinterpret_cast<const uint4 *>(W);
    for (int t = threadIdx.x; t < H * 16; t += blockDim.x) {
        const int n = (t >> 7) * 8 + (t & 7), c = (t >> 3) & 15;
        *reinterpret_cast<uint4 *>(sB + tc_off(n, c)) = W4[n * 16 + c];
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(tslot)),
                     "r"(kTcCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_u) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // W visible to the tensor cores
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __shared__ float ypart[kTcRows];  // DECODE: the upper 32 columns' share of each row's w . H
    const uint32_t tmem = *tslot;
    // warps w and w + 4 share TMEM lanes 32 (w % 4) ..: w < 4 reads columns 0-31, w >= 4 columns 32-63
    const int quad = warp & 3, half = warp >> 2;
    const uint32_t trow = tmem + ((uint32_t)(32 * quad) << 16) + 32u * half;
    const int64_t tiles = (N + rows - 1) / rows;
    const int passes = rows >> 2;
    const uint4 *Hin4 = reinterpret_cast<const uint4 *>(Hin);
    const int sub = lane >> 3, fl = lane & 7;
    uint32_t parity = 0;
    bool ok = !(*err), pending = false;  // pending: MMAs committed and not yet waited for
    // consecutive tiles to the CTAs that the first wave puts on one SM: they
    // share most of their neighbours' lines in L1
    const int64_t per = gridDim.x / sms;  // the grid is a multiple of sms
    for (int64_t t0 = 0; t0 < tiles && ok; t0 += gridDim.x) {
        const int64_t tile = t0 + (blockIdx.x % sms) * per + blockIdx.x / sms;
        if (tile >= tiles) break;
        // gather: passes of four rows, 8 lanes per row, dealt to the warps in turn.
        // A trip takes 8 neighbours: their 8 loads are independent, and the
        // next trip's columns and weights (at a row's end the next pass's) are
        // already on their way.
        const int64_t first = tile * rows;
        int32_t b, len;
        auto row_at = [&](int pass, int32_t &rb, int32_t &rl) {
            const int64_t i = first + 4 * pass + sub;
            const bool in = pass < passes && i < N;
            rb = in ? rp[i] : 0;
            rl = in ? rp[i + 1] - rb : 0;
        };
        row_at(warp, b, len);
        int32_t cv = fl < len ? col[b + fl] : 0;  // padding: row 0 with weight 0
        float av = fl < len ? v[b + fl] : 0.f;
        for (int pass = warp; pass < passes; pass += 8) {
            const int rr = 4 * pass + sub;
            const int64_t i = first + rr;
            int32_t bn, lenn;
            row_at(pass + 8, bn, lenn);
            int maxlen = max(len, 1);
            maxlen = max(maxlen, __shfl_xor_sync(0xffffffffu, maxlen, 8));
            maxlen = max(maxlen, __shfl_xor_sync(0xffffffffu, maxlen, 16));
            unsigned long long acc[4] = {0ull, 0ull, 0ull, 0ull};  // pairs of FP32 sums
            for (int s0 = 0; s0 < maxlen; s0 += 8) {
                const bool more = s0 + 8 < maxlen;
                const int sn = more ? s0 + 8 + fl : fl;
                const int32_t nb = more ? b : bn, nl = more ? len : lenn;
                const int32_t cvn = sn < nl ? col[nb + sn] : 0;
                const float avn = sn < nl ? v[nb + sn] : 0.f;
                uint4 u[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) u[j] = Hin4[(int64_t)__shfl_sync(0xffffffffu, cv, j, 8) * 8 + fl];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const unsigned long long aj = f2_pack(__shfl_sync(0xffffffffu, av, j, 8));
                    acc[0] = f2_fma(aj, bf16x2_to_f2b(u[j].x), acc[0]);
                    acc[1] = f2_fma(aj, bf16x2_to_f2b(u[j].y), acc[1]);
                    acc[2] = f2_fma(aj, bf16x2_to_f2b(u[j].z), acc[2]);
                    acc[3] = f2_fma(aj, bf16x2_to_f2b(u[j].w), acc[3]);
                }
                cv = cvn;
                av = avn;
            }
            const uint4 hv = i < N ? Hin4[i * 8 + fl] : make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4 *>(sA + tc_off(rr, fl)) = hv;
            *reinterpret_cast<uint4 *>(sA + tc_off(rr, 8 + fl)) =
                make_uint4(f2_bf16(acc[0]), f2_bf16(acc[1]), f2_bf16(acc[2]), f2_bf16(acc[3]));
            b = bn;
            len = lenn;
        }
        // the tile is visible to the tensor cores, and every warp has read the
        // previous tile's accumulator
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (threadIdx.x == 0) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                const uint64_t da = tc_desc(sA_u + 256u * ks), db = tc_desc(sB_u + 256u * ks);
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                    :
                    : "r"(tmem), "l"(da), "l"(db), "r"(kTcIdesc), "r"(ks), "r"(0u)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_u)
                         : "memory");
        }
        pending = true;
        ok = __syncthreads_and(tc_wait(bar_u, parity));
        if (!ok) break;
        pending = false;
        parity ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int64_t i = first + 32 * quad + lane;  // this thread's row
        const bool mine = 32 * quad + lane < rows && i < N;
        const int c0 = 32 * half;                              // and its first column
        float y = 0.f;
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            float d[16];
            tc_ld16(trow + 16u * part, d);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int cb = c0 + 16 * part;
            if constexpr (!DECODE) {
                uint32_t w[8];
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    w[j] = pack_bf16(fmaxf(d[2 * j] + sbias[cb + 2 * j], 0.f),
                                     fmaxf(d[2 * j + 1] + sbias[cb + 2 * j + 1], 0.f));
                if (mine) {
                    uint4 *dst = reinterpret_cast<uint4 *>(Hout + i * (H / 2) + cb / 2);
                    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
                    dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) y = fmaf(sdec[cb + j], fmaxf(d[j] + sbias[cb + j], 0.f), y);
            }
        }
        if constexpr (DECODE) {
            if (half) ypart[32 * quad + lane] = y;
            __syncthreads();
            if (!half && mine) {
                y += ypart[32 * quad + lane];
                const double sc = sqrt(scal[0] / (double)N);
                z[i] = sc * (double)sdinv[i] * (double)(mask[i] ? x0[i] : x0[i] + y + P[OFF_DB]);
            }
        }
    }
    if (!ok && pending) {
        // a wait gave up: record it and let the MMAs in flight finish (bounded)
        if (threadIdx.x == 0) atomicExch(err, 1);
        tc_wait(bar_u, parity);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols));
}

// ---- training products on tcgen05 --------------------------------------------------
// Shared steps of the tensor-core kernels below: warp 0 allocates NCOLS
// tensor-memory columns and thread 0 initialises the mbarrier; tc_product
// makes the staged operands visible to the tensor cores, lets thread 0 issue
// the KS K-steps (16 each) and commit them, and waits for them (bounded);
// tc_finish frees the tensor memory after a last bounded wait when a product
// is still in flight.
template <uint32_t NCOLS>
__device__ __forceinline__ uint32_t tc_setup(uint32_t *tslot, uint32_t bar_u)
{
    if ((threadIdx.x >> 5) == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(tslot)),
                     "r"(NCOLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_u) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return *tslot;
}

template <int KCA, int KCB, int KS, uint32_t IDESC>
__device__ __forceinline__ bool tc_product(uint32_t sA_u, uint32_t sB_u, uint32_t tmem, uint32_t bar_u,
                                           uint32_t parity)
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (threadIdx.x == 0) {
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            const uint64_t da = tc_desc<KCA>(sA_u + 256u * ks), db = tc_desc<KCB>(sB_u + 256u * ks);
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                :
                : "r"(tmem), "l"(da), "l"(db), "r"(IDESC), "r"(ks), "r"(0u)
                : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_u)
                     : "memory");
    }
    const bool ok = __syncthreads_and(tc_wait(bar_u, parity));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return ok;
}

template <uint32_t NCOLS>
__device__ __forceinline__ void tc_finish(uint32_t tmem, uint32_t bar_u, uint32_t parity, bool ok, bool pending,
                                          int *err)
{
    if (!ok && pending) {
        if (threadIdx.x == 0) atomicExch(err, 1);
        tc_wait(bar_u, parity);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if ((threadIdx.x >> 5) == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOLS));
}

// Hout = relu([Hin | Yin] W^T + b) on tcgen05: 128 nodes per tile, the FP32
// inputs rounded to BF16 into the canonical K-major layout (K = 128), W
// (64 x 128) staged once; M = 128, N = 64, eight K-steps into 64 TMEM columns.
// A CTA takes `rows` <= 128 nodes at a time (tc_layer_rows): the time is that
// of one tile's loads, so small meshes are spread over all CTAs.
// Sixteen warps; warp w reads back TMEM lanes 32 (w % 4) .., columns 16 (w / 4) ...
constexpr size_t kTcFwdSmem = (size_t)kTcABytes + kTcBBytes + 16;

__global__ void __launch_bounds__(512, 2) k_dense_fwd_tc(const float *__restrict__ Hin, const float *__restrict__ Yin,
                                                         const __nv_bfloat16 *__restrict__ W,
                                                         const float *__restrict__ bias, int64_t N, int rows,
                                                         float *__restrict__ Hout, int *err)
{
    extern __shared__ __align__(1024) unsigned char tsm[];
    unsigned char *sA = tsm, *sB = tsm + tc_layer_a(rows);
    uint64_t *bar = reinterpret_cast<uint64_t *>(sB + kTcBBytes);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(sB + kTcBBytes + 8);
    const uint32_t sA_u = (uint32_t)__cvta_generic_to_shared(sA), sB_u = (uint32_t)__cvta_generic_to_shared(sB);
    const uint32_t bar_u = (uint32_t)__cvta_generic_to_shared(bar);
    const uint4 *W4 = reinterpret_cast<const uint4 *>(W);
    for (int t = threadIdx.x; t < H * 16; t += blockDim.x) {
        const int n = (t >> 7) * 8 + (t & 7), c = (t >> 3) & 15;
        *reinterpret_cast<uint4 *>(sB + tc_off(n, c)) = W4[n * 16 + c];
    }
    const uint32_t tmem = tc_setup<64>(tslot, bar_u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3, quarter = warp >> 2;
    const uint32_t trow = tmem + ((uint32_t)(32 * quad) << 16) + 16u * quarter;
    const int64_t tiles = (N + rows - 1) / rows;
    uint32_t parity = 0;
    bool ok = !(*err), pending = false;
    for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        // rows x 16 pieces of 8 inputs, eight rows to eight lanes: their
        // pieces lie side by side in shared memory
        for (int t = threadIdx.x; t < rows * 16; t += blockDim.x) {
            const int rr = (t >> 7) * 8 + (t & 7), c = (t >> 3) & 15;
            const int64_t i = tile * rows + rr;
            uint4 u = make_uint4(0, 0, 0, 0);
            if (i < N) {
                const float4 *src = reinterpret_cast<const float4 *>((c < 8 ? Hin : Yin) + i * H + (c & 7) * 8);
                const float4 a = src[0], b = src[1];
                u = make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
            }
            *reinterpret_cast<uint4 *>(sA + tc_off(rr, c)) = u;
        }
        pending = true;
        ok = tc_product<16, 16, 8, tc_idesc(128, 64)>(sA_u, sB_u, tmem, bar_u, parity);
        if (!ok) break;
        pending = false;
        parity ^= 1u;
        const int64_t i = tile * rows + 32 * quad + lane;
        const bool mine = 32 * quad + lane < rows && i < N;
        float d[16];
        tc_ld16(trow, d);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const int cb = 16 * quarter;
        if (mine) {
            float4 *dst = reinterpret_cast<float4 *>(Hout + i * H + cb);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                dst[q] = make_float4(fmaxf(d[4 * q] + bias[cb + 4 * q], 0.f), fmaxf(d[4 * q + 1] + bias[cb + 4 * q + 1], 0.f),
                                     fmaxf(d[4 * q + 2] + bias[cb + 4 * q + 2], 0.f),
                                     fmaxf(d[4 * q + 3] + bias[cb + 4 * q + 3], 0.f));
        }
    }
    tc_finish<64>(tmem, bar_u, parity, ok, pending, err);
}

// [dHprev | dY] = dZ W with dZ = dH * (Hl > 0) on tcgen05: A = dZ rounded to
// BF16 (128 x 64, K = 64 over the layer's outputs), B = W^T (128 x 64, staged
// once from W's transposed copy); M = 128, N = 128, four K-steps into 128 TMEM
// columns.  Warp w reads back TMEM lanes 32 (w % 4) .., columns 32 (w / 4) ..
// (0-63: dHprev, 64-127: dY).
constexpr int kTcXABytes = kTcRows * H * 2;   // 16 KiB
constexpr int kTcXBBytes = 2 * H * H * 2;     // 16 KiB
constexpr size_t kTcBwdSmem = (size_t)kTcXABytes + kTcXBBytes + 16;  // of 128 rows
static_assert(kTcXBBytes >= kTcXABytes, "128 rows of A lie within a shorter tile and B");

__global__ void __launch_bounds__(512, 2) k_dense_bwd_x_tc(const float *__restrict__ dH, const float *__restrict__ Hl,
                                                           const __nv_bfloat16 *__restrict__ Wt, int64_t N, int rows,
                                                           float *__restrict__ dHprev, float *__restrict__ dY,
                                                           int *err)
{
    extern __shared__ __align__(1024) unsigned char tsm[];
    unsigned char *sA = tsm, *sB = tsm + rows * H * 2;  // the MMA's 128 rows reach into B at most
    uint64_t *bar = reinterpret_cast<uint64_t *>(sB + kTcXBBytes);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(sB + kTcXBBytes + 8);
    const uint32_t sA_u = (uint32_t)__cvta_generic_to_shared(sA), sB_u = (uint32_t)__cvta_generic_to_shared(sB);
    const uint32_t bar_u = (uint32_t)__cvta_generic_to_shared(bar);
    // B[j][o] = W[o][j]: 128 rows j x 8 pieces of 8 outputs o, from the transposed copy
    const uint4 *Wt4 = reinterpret_cast<const uint4 *>(Wt);
    for (int t = threadIdx.x; t < 2 * H * 8; t += blockDim.x) {
        const int j = (t >> 6) * 8 + (t & 7), c = (t >> 3) & 7;
        *reinterpret_cast<uint4 *>(sB + tc_off<8>(j, c)) = Wt4[j * 8 + c];
    }
    const uint32_t tmem = tc_setup<128>(tslot, bar_u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3, quarter = warp >> 2;
    const uint32_t trow = tmem + ((uint32_t)(32 * quad) << 16) + 32u * quarter;
    float *out = quarter >= 2 ? dY : dHprev;
    const int64_t tiles = (N + rows - 1) / rows;
    uint32_t parity = 0;
    bool ok = !(*err), pending = false;
    for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        // rows x 8 pieces of 8 outputs, eight rows to eight lanes
        for (int t = threadIdx.x; t < rows * 8; t += blockDim.x) {
            const int rr = (t >> 6) * 8 + (t & 7), c = (t >> 3) & 7;
            const int64_t i = tile * rows + rr;
            uint4 u = make_uint4(0, 0, 0, 0);
            if (i < N) {
                const float4 *d4 = reinterpret_cast<const float4 *>(dH + i * H + 8 * c);
                const float4 *h4 = reinterpret_cast<const float4 *>(Hl + i * H + 8 * c);
                const float4 a = d4[0], b = d4[1], ha = h4[0], hb = h4[1];
                u = make_uint4(pack_bf16(ha.x > 0.f ? a.x : 0.f, ha.y > 0.f ? a.y : 0.f),
                               pack_bf16(ha.z > 0.f ? a.z : 0.f, ha.w > 0.f ? a.w : 0.f),
                               pack_bf16(hb.x > 0.f ? b.x : 0.f, hb.y > 0.f ? b.y : 0.f),
                               pack_bf16(hb.z > 0.f ? b.z : 0.f, hb.w > 0.f ? b.w : 0.f));
            }
            *reinterpret_cast<uint4 *>(sA + tc_off<8>(rr, c)) = u;
        }
        pending = true;
        ok = tc_product<8, 8, 4, tc_idesc(128, 128)>(sA_u, sB_u, tmem, bar_u, parity);
        if (!ok) break;
        pending = false;
        parity ^= 1u;
        const int64_t i = tile * rows + 32 * quad + lane;
        const bool mine = 32 * quad + lane < rows && i < N;
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            float d[16];
            tc_ld16(trow + 16u * part, d);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (mine) {
                float4 *dst = reinterpret_cast<float4 *>(out + i * H + 32 * (quarter & 1) + 16 * part);
#pragma unroll
                for (int q = 0; q < 4; ++q) dst[q] = make_float4(d[4 * q], d[4 * q + 1], d[4 * q + 2], d[4 * q + 3]);
            }
        }
    }
    tc_finish<128>(tmem, bar_u, parity, ok, pending, err);
}

// dW[o][j] += sum_i dZ[i][o] Xc[i][j] (Xc = [Hin | Yin]) and db[o] += sum_i
// dZ[i][o] on tcgen05: the transposed product dW^T = Xc^T dZ with M = 128 (the
// inputs j), N = 64 (the outputs o) and K = the 128 nodes of a tile, both
// operands MN-major as they lie in memory (a node's 8 consecutive features
// are one 16-byte piece: piece (feature group g, node group kg) at byte
// (16 g + kg) * 128 + (node % 8) * 16, so the next node group is 128 B on
// (LBO) and the next feature group 2,048 B on (SBO)), rounded to BF16 like
// the forward products.  A CTA accumulates all its tiles in 64 TMEM columns
// and adds the result to GW once; db (unrounded dZ) is summed on the way.
constexpr uint32_t kTcIdescWgrad = tc_idesc(128, 64) | (1u << 15) | (1u << 16);  // A and B MN-major

__global__ void __launch_bounds__(256, 4) k_dense_bwd_w_tc(const float *__restrict__ dH, const float *__restrict__ Hl,
                                                           const float *__restrict__ Hin,
                                                           const float *__restrict__ Yin, int64_t N,
                                                           float *__restrict__ GW, float *__restrict__ Gb, int *err)
{
    extern __shared__ __align__(1024) unsigned char tsm[];
    unsigned char *sA = tsm, *sB = tsm + kTcABytes;  // Xc^T: 128 x 128 (32 KiB); dZ^T: 64 x 128 (16 KiB)
    uint64_t *bar = reinterpret_cast<uint64_t *>(tsm + kTcABytes + kTcBBytes);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(tsm + kTcABytes + kTcBBytes + 8);
    __shared__ float sdb[8][H];
    const uint32_t sA_u = (uint32_t)__cvta_generic_to_shared(sA), sB_u = (uint32_t)__cvta_generic_to_shared(sB);
    const uint32_t bar_u = (uint32_t)__cvta_generic_to_shared(bar);
    const uint32_t tmem = tc_setup<64>(tslot, bar_u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3, half = warp >> 2;
    const int64_t tiles = (N + kTcRows - 1) / kTcRows;
    uint32_t parity = 0;
    bool ok = !(*err), pending = false, any = false;
    float db[8] = {};
    for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        // Xc: 128 nodes x 16 feature groups; dZ: 128 nodes x 8 output groups;
        // eight nodes to eight lanes (their pieces lie side by side)
        auto piece = [&](unsigned char *dst, int g, int node, const float4 &a, const float4 &b) {
            *reinterpret_cast<uint4 *>(dst + (g * 16 + (node >> 3)) * 128 + (node & 7) * 16) =
                make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
        };
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int t = threadIdx.x; t < kTcRows * 16; t += 256) {
            const int node = (t >> 7) * 8 + (t & 7), g = (t >> 3) & 15;
            const int64_t i = tile * kTcRows + node;
            const float4 *src = reinterpret_cast<const float4 *>((g < 8 ? Hin : Yin) + i * H + (g & 7) * 8);
            piece(sA, g, node, i < N ? src[0] : zero, i < N ? src[1] : zero);
        }
#pragma unroll
        for (int t = threadIdx.x; t < kTcRows * 8; t += 256) {
            const int node = (t >> 6) * 8 + (t & 7), g = (t >> 3) & 7;  // g is the thread's in every trip
            const int64_t i = tile * kTcRows + node;
            float4 a = zero, b = zero;
            if (i < N) {
                const float4 *d4 = reinterpret_cast<const float4 *>(dH + i * H + g * 8);
                const float4 *h4 = reinterpret_cast<const float4 *>(Hl + i * H + g * 8);
                const float4 da = d4[0], dbv = d4[1], ha = h4[0], hb = h4[1];
                a = make_float4(ha.x > 0.f ? da.x : 0.f, ha.y > 0.f ? da.y : 0.f, ha.z > 0.f ? da.z : 0.f,
                                ha.w > 0.f ? da.w : 0.f);
                b = make_float4(hb.x > 0.f ? dbv.x : 0.f, hb.y > 0.f ? dbv.y : 0.f, hb.z > 0.f ? dbv.z : 0.f,
                                hb.w > 0.f ? dbv.w : 0.f);
            }
            const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int q = 0; q < 8; ++q) db[q] += v[q];  // unrounded
            piece(sB, g, node, a, b);
        }
        pending = true;
        // K-steps of 16 nodes: the descriptors advance by two node groups (256 B);
        // the first tile's first step overwrites the accumulator
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (threadIdx.x == 0) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                const uint64_t da = tc_desc<16>(sA_u + 256u * ks), dbd = tc_desc<16>(sB_u + 256u * ks);
                const uint32_t acc = (any || ks > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                    :
                    : "r"(tmem), "l"(da), "l"(dbd), "r"(kTcIdescWgrad), "r"(acc), "r"(0u)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_u)
                         : "memory");
        }
        ok = __syncthreads_and(tc_wait(bar_u, parity));
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!ok) break;
        pending = false;
        any = true;
        parity ^= 1u;
    }
    if (ok && any) {
        // D[j][o]: warps w and w + 4 hold inputs j = 32 (w % 4) + lane, outputs 0-31 / 32-63
        const int j = 32 * quad + lane;
        const uint32_t trow = tmem + ((uint32_t)(32 * quad) << 16) + 32u * half;
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            float d[16];
            tc_ld16(trow + 16u * part, d);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int q = 0; q < 16; ++q) atomicAdd(&GW[(32 * half + 16 * part + q) * 2 * H + j], d[q]);
        }
    }
    // db: the eight lanes of an output group, then the warps (group 4 (warp % 2) + lane / 8)
#pragma unroll
    for (int q = 0; q < 8; ++q) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) db[q] += __shfl_xor_sync(0xffffffffu, db[q], o);
        if ((lane & 7) == 0) sdb[warp][(4 * (warp & 1) + (lane >> 3)) * 8 + q] = db[q];
    }
    __syncthreads();
    if (ok && any && threadIdx.x < H) {
        const int w0 = threadIdx.x >> 5;  // warps of this group's parity
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) s += sdb[2 * w + w0][threadIdx.x];
        atomicAdd(&Gb[threadIdx.x], s);
    }
    tc_finish<64>(tmem, bar_u, parity, ok, pending, err);
}

__device__ double block_sum_d(double v, double *sh)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    v = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
    if (threadIdx.x < 32) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    return v;  // valid in thread 0
}

// *out += a . b
__global__ void k_fdot(const double *__restrict__ a, const double *__restrict__ b, int64_t n, double *out)
{
    __shared__ double sh[32];
    double v = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        v += a[i] * b[i];
    v = block_sum_d(v, sh);
    if (threadIdx.x == 0) atomicAdd(out, v);
}

// ---- flexible CG with the network: one persistent kernel -------------------------
// As launches an iteration took seven (24.0 ms for the 221 iterations of a
// 33^3 cube), and of a layer's 23 us ten went into starting its CTAs: tensor
// memory, W, first loads.  Here one CTA per SM, of a cooperative launch, keeps
// all three W and its tensor memory, owns a run of consecutive rows and goes
// through the phases of an iteration behind grid barriers (pcg.cuh; every wait
// has a limit):
//   x, r update with |r|^2, D^-1/2 r and its norm | encoder | layer | layer |
//   layer and decoder with z.q | p update with p.r | q = S p with p.q
//
// A layer takes 320 rows a round (three MMA tiles of 128, the last one partly
// behind the rows).  Its gather is the bulk of an iteration.  On meshes
// numbered along a lattice (WIN) the columns of a row are runs of consecutive
// nodes, the same for every row, so 8 lanes take four rows together: a window
// of 6 activation rows serves 12 entries, no indices, the weights 16 bytes at
// a time.  Sums stay in the order of the columns, as in k_layer_tc.
constexpr int kFcgThreads = 640, kFcgWarps = kFcgThreads / 32;
constexpr int kFcgRows = 4 * 4 * kFcgWarps;  // rows of a round: four per 8 lanes
constexpr int kFcgABytes = kFcgRows * 2 * H * 2;
constexpr size_t kFcgSmem = (size_t)kFcgABytes + LAYERS * kTcBBytes + 16;
constexpr int kFcgTiles = (kFcgRows + kTcRows - 1) / kTcRows;
constexpr uint32_t kFcgCols = 256;  // tensor-memory columns: kFcgTiles x 64, a power of two
static_assert(kFcgTiles * kTcABytes <= kFcgABytes + LAYERS * kTcBBytes, "the last tile's 128 rows lie within A and W");
static_assert(kFcgTiles * kTcCols <= kFcgCols, "accumulators");

struct FcgArgs {
    PcgArgs op;  // x, r, p, q; sums: p.q, p.r, r.r, z.q, |D^-1/2 r|^2; out: iterations, why, error, (barrier), mark_it
    const int32_t *rp, *col;
    const float *ahat;
    const float4 *win;  // [run][quad of rows][3][4 rows]
    int runs, woff[kDiaMax];
    const float *sdinv;
    const unsigned char *mask;
    const __nv_bfloat16 *W;
    const float *P;
    float *rhat, *x0;
    uint32_t *hb0, *hb1;  // WIN: with rows of zeros before and behind, for the windows that reach out of the matrix
    double *z, *mark;  // mark: rr at the last 100-fold reduction
    int64_t per;       // rows of a CTA, a multiple of 4
    int it0, check, stall, mark_it;
    double thr;
};
enum FcgWhy { FCG_CAP = 0, FCG_DONE = 1, FCG_BREAKDOWN = 2, FCG_STALL = 3 };

struct FcgShared {
    CommShared comm;
    alignas(16) float bias[LAYERS][H];
    alignas(16) float dec[H];
    alignas(16) float enc[3][H];
    float ypart[kFcgRows];
};

// rows r0 .. of the round -> [Hin | Ahat Hin] in sA
template <bool WIN>
__device__ __forceinline__ void fcg_gather(const FcgArgs &g, unsigned char *sA, const uint4 *Hin4, int64_t r0, int64_t row1)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane >> 3, fl = lane & 7;
    const int64_t N = g.op.N;
    if constexpr (WIN) {
        const int rr = 4 * (4 * warp + sub);
        const int64_t i = r0 + rr;
        if (i >= row1) return;
        unsigned long long acc[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[k][c] = 0ull;
        const int64_t step = ((N + 3) >> 2) * 3;
        const float4 *w4 = g.win + (i >> 2) * 3;
        float w[3][4];
        uint4 h[6];
        const uint4 *row = Hin4 + i * 8 + fl, *hp = row + (int64_t)g.woff[0] * 8;
#pragma unroll
        for (int j = 0; j < 6; ++j) h[j] = hp[8 * j];
#pragma unroll
        for (int u = 0; u < 3; ++u) *reinterpret_cast<float4 *>(w[u]) = w4[u];
#pragma unroll 1
        for (int s = 1; s <= g.runs; ++s) {
            // the next run's values are fetched as this run's are used up
            const int sn = min(s, g.runs - 1);
            w4 += s < g.runs ? step : 0;
            hp = row + (int64_t)g.woff[sn] * 8;
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                const unsigned long long f[4] = {bf16x2_to_f2b(h[j].x), bf16x2_to_f2b(h[j].y), bf16x2_to_f2b(h[j].z),
                                                 bf16x2_to_f2b(h[j].w)};
                h[j] = hp[8 * j];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (j - k >= 0 && j - k < 3) {
                        const unsigned long long a = f2_pack(w[j - k < 0 || j - k > 2 ? 0 : j - k][k]);
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[k][c] = f2_fma(a, f[c], acc[k][c]);
                    }
                if (j >= 3) *reinterpret_cast<float4 *>(w[j >= 3 ? j - 3 : 0]) = w4[j - 3];
            }
        }
        // lane fl stores the rows in the order k ^ (fl & 3): the pieces of one
        // row lie 128 bytes apart, in the same banks
        uint4 y[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = make_uint4(f2_bf16(acc[k][0]), f2_bf16(acc[k][1]), f2_bf16(acc[k][2]), f2_bf16(acc[k][3]));
        auto swap_if = [](bool c, uint4 &a, uint4 &b) {
            const uint4 t = c ? b : a;
            b = c ? a : b;
            a = t;
        };
        swap_if(fl & 1, y[0], y[1]);
        swap_if(fl & 1, y[2], y[3]);
        swap_if(fl & 2, y[0], y[2]);
        swap_if(fl & 2, y[1], y[3]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int kk = k ^ (fl & 3);
            *reinterpret_cast<uint4 *>(sA + tc_off(rr + kk, fl)) = row[8 * kk];
            *reinterpret_cast<uint4 *>(sA + tc_off(rr + kk, 8 + fl)) = y[k];
        }
    } else {
        const int passes = (int)(min((int64_t)kFcgRows, row1 - r0) + 3) >> 2;
        for (int pass = warp; pass < passes; pass += kFcgWarps) {
            const int rr = 4 * pass + sub;
            const int64_t i = r0 + rr;
            const int32_t b = i < row1 ? g.rp[i] : 0;
            const int len = i < row1 ? g.rp[i + 1] - b : 0;
            int maxlen = len;
            maxlen = max(maxlen, __shfl_xor_sync(0xffffffffu, maxlen, 8));
            maxlen = max(maxlen, __shfl_xor_sync(0xffffffffu, maxlen, 16));
            unsigned long long acc[4] = {0ull, 0ull, 0ull, 0ull};
            int32_t cv = fl < len ? g.col[b + fl] : 0;  // padding: row 0 with weight 0
            float av = fl < len ? g.ahat[b + fl] : 0.f;
            for (int s0 = 0; s0 < maxlen; s0 += 8) {
                const int sn = s0 + 8 + fl;
                const int32_t cvn = sn < len ? g.col[b + sn] : 0;
                const float avn = sn < len ? g.ahat[b + sn] : 0.f;
                uint4 u[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) u[j] = Hin4[(int64_t)__shfl_sync(0xffffffffu, cv, j, 8) * 8 + fl];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const unsigned long long aj = f2_pack(__shfl_sync(0xffffffffu, av, j, 8));
                    acc[0] = f2_fma(aj, bf16x2_to_f2b(u[j].x), acc[0]);
                    acc[1] = f2_fma(aj, bf16x2_to_f2b(u[j].y), acc[1]);
                    acc[2] = f2_fma(aj, bf16x2_to_f2b(u[j].z), acc[2]);
                    acc[3] = f2_fma(aj, bf16x2_to_f2b(u[j].w), acc[3]);
                }
                cv = cvn;
                av = avn;
            }
            const uint4 hv = i < row1 ? Hin4[i * 8 + fl] : make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4 *>(sA + tc_off(rr, fl)) = hv;
            *reinterpret_cast<uint4 *>(sA + tc_off(rr, 8 + fl)) =
                make_uint4(f2_bf16(acc[0]), f2_bf16(acc[1]), f2_bf16(acc[2]), f2_bf16(acc[3]));
        }
    }
}

// one layer on the CTA's rows; false when a wait for the MMAs gave up (they
// may still be in flight).  DECODE: z and this thread's share of z.q.
template <bool WIN, bool DECODE>
__device__ bool fcg_layer(const FcgArgs &g, FcgShared &sh, unsigned char *sA, uint32_t sB_u, uint32_t bar_u, uint32_t tmem,
                          uint32_t &parity, const uint32_t *Hin, uint32_t *Hout, const float *bias, int64_t row0,
                          int64_t row1, double nn, double &dot)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3;
    const uint32_t sA_u = (uint32_t)__cvta_generic_to_shared(sA);
    for (int64_t r0 = row0; r0 < row1; r0 += kFcgRows) {
        const int rows = (int)min((int64_t)kFcgRows, row1 - r0), tiles = (rows + kTcRows - 1) / kTcRows;
        fcg_gather<WIN>(g, sA, reinterpret_cast<const uint4 *>(Hin), r0, row1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (threadIdx.x == 0) {
            for (int tile = 0; tile < tiles; ++tile)
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    const uint64_t da = tc_desc(sA_u + (uint32_t)kTcABytes * tile + 256u * ks), db = tc_desc(sB_u + 256u * ks);
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                        :
                        : "r"(tmem + kTcCols * tile), "l"(da), "l"(db), "r"(kTcIdesc), "r"(ks), "r"(0u)
                        : "memory");
                }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_u)
                         : "memory");
        }
        if (!__syncthreads_and(tc_wait(bar_u, parity))) return false;
        parity ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // warps of one quarter of the TMEM lanes share out the tiles' halves of 32 columns
        // (five such warps: a warp has at most one half of either parity)
        static_assert(kFcgWarps / 4 % 2 == 1 && 2 * kFcgTiles <= kFcgWarps / 2, "one lower half to a warp");
        float yown = 0.f;
        int rown = rows;
        for (int task = warp >> 2; task < 2 * tiles; task += kFcgWarps / 4) {
            const int tile = task >> 1, half = task & 1, rr = kTcRows * tile + 32 * quad + lane;
            const int64_t i = r0 + rr;
            float y = 0.f;
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                float d[16];
                const int cb = 32 * half + 16 * part;
                float bv[16];
#pragma unroll
                for (int j = 0; j < 4; ++j) *reinterpret_cast<float4 *>(bv + 4 * j) = *reinterpret_cast<const float4 *>(bias + cb + 4 * j);
                tc_ld16(tmem + ((uint32_t)(32 * quad) << 16) + kTcCols * tile + cb, d);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if constexpr (!DECODE) {
                    uint32_t w[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        w[j] = pack_bf16(fmaxf(d[2 * j] + bv[2 * j], 0.f),
                                         fmaxf(d[2 * j + 1] + bv[2 * j + 1], 0.f));
                    if (rr < rows) {
                        uint4 *dst = reinterpret_cast<uint4 *>(Hout + i * (H / 2) + cb / 2);
                        dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
                        dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 w = *reinterpret_cast<const float4 *>(sh.dec + cb + 4 * j);
                        y = fmaf(w.x, fmaxf(d[4 * j] + bv[4 * j], 0.f), y);
                        y = fmaf(w.y, fmaxf(d[4 * j + 1] + bv[4 * j + 1], 0.f), y);
                        y = fmaf(w.z, fmaxf(d[4 * j + 2] + bv[4 * j + 2], 0.f), y);
                        y = fmaf(w.w, fmaxf(d[4 * j + 3] + bv[4 * j + 3], 0.f), y);
                    }
                }
            }
            if constexpr (DECODE) {
                if (half && rr < rows) sh.ypart[rr] = y;
                if (!half) {
                    yown = y;
                    rown = rr;
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if constexpr (DECODE) {
            __syncthreads();
            const double sc = sqrt(nn / (double)g.op.N);
            if (rown < rows) {
                const int64_t i = r0 + rown;
                const float y = yown + sh.ypart[rown];
                const double zi = sc * (double)g.sdinv[i] * (double)(g.mask[i] ? g.x0[i] : g.x0[i] + y + g.P[OFF_DB]);
                g.z[i] = zi;
                dot += zi * g.op.q[i];
            }
        }
    }
    return true;
}

template <int F, bool WIN>
__global__ void __launch_bounds__(kFcgThreads, 1) k_fcg(const __grid_constant__ FcgArgs g)
{
    extern __shared__ __align__(1024) unsigned char tsm[];
    __shared__ __align__(16) FcgShared sh;
    unsigned char *sA = tsm, *sB = tsm + kFcgABytes;
    uint64_t *bar = reinterpret_cast<uint64_t *>(sB + LAYERS * kTcBBytes);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(sB + LAYERS * kTcBBytes + 8);
    const uint32_t sB_u = (uint32_t)__cvta_generic_to_shared(sB), bar_u = (uint32_t)__cvta_generic_to_shared(bar);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int t = tid; t < LAYERS * H * 16; t += kFcgThreads) {
        const int l = t >> 10, u = t & 1023, n = (u >> 7) * 8 + (u & 7), c = (u >> 3) & 15;
        *reinterpret_cast<uint4 *>(sB + l * kTcBBytes + tc_off(n, c)) = reinterpret_cast<const uint4 *>(g.W)[l * H * 16 + n * 16 + c];
    }
    if (tid < H) {
        for (int l = 0; l < LAYERS; ++l) sh.bias[l][tid] = g.P[OFF_L + l * LSZ + H * 2 * H + tid];
        sh.dec[tid] = g.P[OFF_DW + tid];
        sh.enc[0][tid] = g.P[OFF_EW + 2 * tid];
        sh.enc[1][tid] = g.P[OFF_EW + 2 * tid + 1];
        sh.enc[2][tid] = g.P[OFF_EB + tid];
    }
    const uint32_t tmem = tc_setup<kFcgCols>(tslot, bar_u);
    uint32_t parity = 0;
    bool tc_ok = true;
    Comm<false> comm{g.op, sh.comm};
    enum { PQ, PR, RR, ZQ, NN, SUMS };
    const int64_t N = g.op.N, row0 = min(N, (int64_t)blockIdx.x * g.per), row1 = min(N, row0 + g.per);
    const bool first = blockIdx.x == 0 && tid == 0;
    double pq = g.op.sums[sum_slot(PQ, g.it0)], pr = g.op.sums[sum_slot(PR, g.it0)], mark = *g.mark, none = 0.0;
    int mark_it = g.mark_it, it = g.it0, why = FCG_CAP;
    while (it < g.op.max_iter) {
        if (!(pq > 0.0)) {
            why = FCG_BREAKDOWN;
            ++it;
            break;
        }
        const double alpha = pr / pq;
        double rr = 0.0, nn = 0.0;
        for (int64_t i = row0 + tid; i < row1; i += kFcgThreads) {
            g.op.x[i] += alpha * g.op.p[i];
            const double ri = g.op.r[i] - alpha * g.op.q[i];
            g.op.r[i] = ri;
            rr += ri * ri;
            const double t = ri * (double)g.sdinv[i];
            nn += t * t;
            g.rhat[i] = (float)t;
        }
        if (!comm.sum<2>(rr, nn, sum_slot(RR, it + 1), sum_slot(NN, it + 1))) break;
        if (first) clear_slots<SUMS>(g.op.sums, it);
        if (rr <= g.thr) {
            why = FCG_DONE;
            ++it;
            break;
        }
        if ((it + 1) % g.check == 0) {  // no 10-fold reduction of |r| within `stall` iterations
            if (rr < 0.01 * mark) {
                mark = rr;
                mark_it = it + 1;
            } else if (it + 1 - mark_it > g.stall) {
                why = FCG_STALL;
                ++it;
                break;
            }
        }
        {  // encoder, 8 lanes per row
            const int sub = lane >> 3, fl = lane & 7;
            const float inv = nn > 0 ? (float)(1.0 / sqrt(nn / (double)N)) : 0.f;
            constexpr int R = 4;  // rows of a lane group at a time: their chains of loads overlap
            for (int64_t base = row0 + 4 * warp; base < row1; base += 4 * kFcgWarps * R) {
                int32_t k0[R], e[R];
                float acc[R], own[R];
                int len = 0;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int64_t i = base + sub + 4 * kFcgWarps * r;
                    k0[r] = i < row1 ? g.rp[i] + fl : 0;
                    e[r] = i < row1 ? g.rp[i + 1] : 0;
                    own[r] = i < row1 ? g.rhat[i] : 0.f;
                    acc[r] = 0.f;
                }
#pragma unroll
                for (int r = 0; r < R; ++r) len = max(len, e[r] - k0[r]);
                for (int k = 0; k < len; k += 32) {
                    int32_t c[R][4];
                    float a[R][4], x[R][4];
#pragma unroll
                    for (int r = 0; r < R; ++r)
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int32_t at = k0[r] + k + 8 * u;
                            c[r][u] = at < e[r] ? g.col[at] : -1;
                            a[r][u] = at < e[r] ? g.ahat[at] : 0.f;
                        }
#pragma unroll
                    for (int r = 0; r < R; ++r)
#pragma unroll
                        for (int u = 0; u < 4; ++u) x[r][u] = c[r][u] >= 0 ? g.rhat[c[r][u]] : 0.f;
#pragma unroll
                    for (int r = 0; r < R; ++r)
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (c[r][u] >= 0) acc[r] = fmaf(a[r][u], x[r][u], acc[r]);
                }
                __syncwarp();
                float ev[3][8];
#pragma unroll
                for (int w = 0; w < 3; ++w)
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        *reinterpret_cast<float4 *>(ev[w] + 4 * q) = *reinterpret_cast<const float4 *>(&sh.enc[w][fl * 8 + 4 * q]);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    float s = acc[r];
                    s += __shfl_xor_sync(0xffffffffu, s, 4);
                    s += __shfl_xor_sync(0xffffffffu, s, 2);
                    s += __shfl_xor_sync(0xffffffffu, s, 1);
                    const int64_t i = base + sub + 4 * kFcgWarps * r;
                    if (i < row1) {
                        const float xi = own[r] * inv, ax = s * inv;
                        uint32_t w[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            w[q] = pack_bf16(
                                fmaxf(fmaf(ev[0][2 * q], xi, fmaf(ev[1][2 * q], ax, ev[2][2 * q])), 0.f),
                                fmaxf(fmaf(ev[0][2 * q + 1], xi, fmaf(ev[1][2 * q + 1], ax, ev[2][2 * q + 1])), 0.f));
                        reinterpret_cast<uint4 *>(g.hb0)[i * 8 + fl] = make_uint4(w[0], w[1], w[2], w[3]);
                        if (fl == 0) g.x0[i] = xi;
                    }
                }
            }
        }
        if (!comm.barrier()) break;
        double zq = 0.0;
        tc_ok = fcg_layer<WIN, false>(g, sh, sA, sB_u, bar_u, tmem, parity, g.hb0, g.hb1, sh.bias[0], row0, row1, nn, zq);
        if (!tc_ok || !comm.barrier()) break;
        tc_ok = fcg_layer<WIN, false>(g, sh, sA, sB_u + kTcBBytes, bar_u, tmem, parity, g.hb1, g.hb0, sh.bias[1], row0, row1, nn, zq);
        if (!tc_ok || !comm.barrier()) break;
        tc_ok = fcg_layer<WIN, true>(g, sh, sA, sB_u + 2 * kTcBBytes, bar_u, tmem, parity, g.hb0, nullptr, sh.bias[2], row0, row1, nn, zq);
        if (!tc_ok || !comm.sum<1>(zq, none, sum_slot(ZQ, it), 0)) break;
        const double beta = -zq / pq;
        pr = 0.0;
        for (int64_t i = row0 + tid; i < row1; i += kFcgThreads) {
            const double pi = g.z[i] + beta * g.op.p[i];
            g.op.p[i] = pi;
            pr += pi * g.op.r[i];
        }
        if (!comm.barrier()) break;
        pq = product<F>(g.op, g.op.p, g.op.q);
        if (!comm.sum<2>(pq, pr, sum_slot(PQ, it + 1), sum_slot(PR, it + 1))) break;
        ++it;
    }
    if (first) {
        g.op.out[0] = it;
        g.op.out[1] = why;
        g.op.out[4] = mark_it;
        *g.mark = mark;
    }
    tc_finish<kFcgCols>(tmem, bar_u, parity, tc_ok, true, g.op.out + 5);
}

// windows of the layers' gather: runs of up to three consecutive columns
struct FcgRuns {
    int runs, off[kDiaMax];
};

__global__ void k_fcg_window(const __grid_constant__ FcgRuns o, const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                             const float *__restrict__ ahat, int64_t N, float *__restrict__ win)
{
    const int64_t quads = (N + 3) >> 2;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 4 * quads; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t k = i < N ? rp[i] : 0;
        const int32_t e = i < N ? rp[i + 1] : 0;
        for (int s = 0; s < o.runs; ++s)
            for (int u = 0; u < 3; ++u) {
                const bool hit = k < e && col[k] - (int)i == o.off[s] + u;
                win[((s * quads + (i >> 2)) * 3 + u) * 4 + (i & 3)] = hit ? ahat[k] : 0.f;
                k += hit;
            }
    }
}

// ---- host side -------------------------------------------------------------------
// the tensor-core (tcgen05) kernels unless SFC_MPNN_TC=0 selects the mma.sync ones
bool use_tc()
{
    static int m = -1;
    if (m < 0) {
        const char *e = std::getenv("SFC_MPNN_TC");
        m = (e && e[0] == '0') ? 0 : 1;
    }
    return m == 1;
}

// grid of the tensor-core kernels (four CTAs per SM by their resources, at
// most 4 x 128 tensor-memory columns; the grid-stride loops take any number of
// tiles); sets their attributes and the error word on first use
unsigned tc_grid(sfc_mpnn *m, int64_t N)
{
    sfc_ctx *ctx = m->ctx;
    if (!m->tc_err.p) {
        m->tc_err.alloc(1);
        SFC_CK(cudaMemsetAsync(m->tc_err.p, 0, sizeof(int), ctx->stream));
    }
    static bool attr = false;
    if (!attr) {
        const std::pair<const void *, size_t> ks[] = {{(const void *)k_layer_tc<false>, tc_layer_smem(kTcRows)},
                                                      {(const void *)k_layer_tc<true>, tc_layer_smem(kTcRows)},
                                                      {(const void *)k_dense_fwd_tc, kTcFwdSmem},
                                                      {(const void *)k_dense_bwd_x_tc, kTcBwdSmem},
                                                      {(const void *)k_dense_bwd_w_tc, kTcFwdSmem}};
        for (const auto &k : ks) {
            SFC_CK(cudaFuncSetAttribute(k.first, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.second));
            const bool layer = k.first == (const void *)k_layer_tc<false> || k.first == (const void *)k_layer_tc<true>;
            if (!layer) SFC_CK(cudaFuncSetAttribute(k.first, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        }
        attr = true;
    }
    return (unsigned)std::min<int64_t>((N + kTcRows - 1) / kTcRows, (int64_t)ctx->sm_count * 4);
}

// nodes per CTA of k_layer_tc: the MMA takes 128, but with N below 128 x the
// CTAs the GPU holds (four per SM) tiles of 128 leave some SMs an extra tile,
// and each warp a chain of four passes of gathers, so the nodes are spread
// over all of them (a multiple of 8; at least 32, one pass per warp).  39,304
// nodes, 27 entries per row: 32.6 us per layer with 128 (308 tiles), 25.6 with 72.
int tc_layer_rows(const sfc_ctx *ctx, int64_t N)
{
    const int64_t slots = (int64_t)ctx->sm_count * 4, even = ((N + slots - 1) / slots + 7) / 8 * 8;
    return (int)std::max<int64_t>(32, std::min<int64_t>(kTcRows, even));
}

// nodes per tile of k_dense_fwd_tc and k_dense_bwd_x_tc, and the CTAs (two fit
// an SM): as few rounds of one tile per SM as 128 nodes a tile allow, of equal
// size.  More and smaller CTAs cost more to start (four per SM: 6 us until the
// last one runs) than their loads take.
int tc_dense_rows(const sfc_ctx *ctx, int64_t N)
{
    const int64_t sm = ctx->sm_count, rounds = (N + kTcRows * sm - 1) / (kTcRows * sm);
    return (int)std::max<int64_t>(32, ((N + sm * rounds - 1) / (sm * rounds) + 7) / 8 * 8);
}
unsigned tc_tiles(sfc_mpnn *m, int64_t N, int rows)
{
    tc_grid(m, N);
    return (unsigned)std::min<int64_t>((N + rows - 1) / rows, (int64_t)m->ctx->sm_count * 2);
}

// after a batch of applications: a tensor-core layer whose bounded wait gave
// up fails the call
void check_tc(sfc_mpnn *m)
{
    if (!m->tc_err.p) return;
    int h = 0;
    download(m->ctx, &h, m->tc_err.p, 1);
    if (h) {
        SFC_CK(cudaMemsetAsync(m->tc_err.p, 0, sizeof(int), m->ctx->stream));
        fail(SFC_ERR_TIMEOUT, "learned preconditioner: a bounded wait for the tensor-core products gave up");
    }
}

void refresh_bf16(sfc_mpnn *m)
{
    k_to_bf16<<<64, 256, 0, m->ctx->stream>>>(m->params.p, m->wbf.p);
    count_launch(m->ctx);
}

// bind the network to a system's operator (scaled copy of its FP64 values)
void bind(sfc_mpnn *m, sfc_system *s)
{
    sfc_ctx *ctx = m->ctx;
    flush_staged(s);
    build_operator(s);
    const int64_t N = s->N;
    if (m->N != N) {
        m->N = N;
        m->sdinv.alloc(N);
        m->x0.alloc(N);
        m->ax0.alloc(N);
        m->yhat.alloc(N);
        m->dvec.alloc(N);
        m->qvec.alloc(N);
        for (int l = 0; l <= LAYERS; ++l) {
            m->H[l].alloc(N * H);
            m->Y[l].alloc(N * H);
        }
        m->hb[0].alloc(N * H);
        m->hb[1].alloc(N * H);
        m->dH0.alloc(N * H);
        m->dH1.alloc(N * H);
        m->dY.alloc(N * H);
    }
    m->ahat.reserve(s->nnz);
    k_scale_op<<<grid_for(8 * N, 256, ctx->sm_count * 16), 256, 0, ctx->stream>>>(s->row_ptr.p, s->col.p, s->diag.p, s->a_op.p, N, m->ahat.p,
                                                         m->sdinv.p);
    count_launch(ctx);
    m->op_sys = s;
}

unsigned gwarp(sfc_ctx *ctx) { return (unsigned)(ctx->sm_count * 8); }

// forward pass on residual r (device FP64): fills x0, ax0, H[], Y[], yhat
void forward(sfc_mpnn *m, const double *r)
{
    sfc_ctx *ctx = m->ctx;
    const sfc_system *s = m->op_sys;
    const int64_t N = m->N;
    const int rows = tc_dense_rows(ctx, N);
    ProfScope ps(ctx, "mpnn_forward", 0.0);
    SFC_CK(cudaMemsetAsync(m->scal.p, 0, sizeof(double), ctx->stream));
    k_scaled_norm2<<<grid_for(N, 256, ctx->sm_count * 4), 256, 0, ctx->stream>>>(r, m->sdinv.p, N, m->scal.p);
    count_launch(ctx);
    k_x0<<<grid_for(N, 256), 256, 0, ctx->stream>>>(r, m->sdinv.p, m->scal.p, N, m->x0.p);
    k_spmv32<true><<<gwarp(ctx), 256, 0, ctx->stream>>>(s->row_ptr.p, s->col.p, m->ahat.p, m->x0.p, m->ax0.p, N,
                                                       m->params.p, m->H[0].p, 0.0, nullptr);
    count_launch(ctx, 2);
    for (int l = 1; l <= LAYERS; ++l) {
        k_agg64<<<ctx->sm_count, 1024, 0, ctx->stream>>>(s->row_ptr.p, s->col.p, m->ahat.p, m->H[l - 1].p, m->Y[l].p, N, 0);
        if (use_tc())
            k_dense_fwd_tc<<<tc_tiles(m, N, rows), 512, tc_layer_smem(rows), ctx->stream>>>(
                m->H[l - 1].p, m->Y[l].p, m->wbf.p + (l - 1) * H * 2 * H, m->params.p + OFF_L + (l - 1) * LSZ + H * 2 * H,
                N, rows, m->H[l].p, m->tc_err.p);
        else
            k_dense_fwd<<<gwarp(ctx), 256, 0, ctx->stream>>>(m->H[l - 1].p, m->Y[l].p, m->wbf.p + (l - 1) * H * 2 * H,
                                                            m->params.p + OFF_L + (l - 1) * LSZ + H * 2 * H, N,
                                                            m->H[l].p);
        count_launch(ctx, 2);
    }
    k_decoder<<<gwarp(ctx), 256, 0, ctx->stream>>>(m->H[LAYERS].p, m->params.p, m->x0.p, s->mask.p, N, m->yhat.p);
    count_launch(ctx);
}

// residual-dependent quantities of a pair: s, x0, target t, d = yhat - t,
// q = 2 w Ahat d / N (the gradient w.r.t. yhat) and the weighted loss in
// scal[1]; yhat is the network output, or x0 alone for the Jacobi loss
void pair_residual(sfc_mpnn *m, const double *e, const float *yhat, double w)
{
    sfc_ctx *ctx = m->ctx;
    const sfc_system *s = m->op_sys;
    const int64_t N = m->N;
    SFC_CK(cudaMemsetAsync(m->scal.p + 1, 0, sizeof(double), ctx->stream));
    k_target_diff<<<grid_for(N, 256), 256, 0, ctx->stream>>>(e, m->sdinv.p, m->scal.p, yhat, N, m->dvec.p);
    k_spmv32<false><<<gwarp(ctx), 256, 0, ctx->stream>>>(s->row_ptr.p, s->col.p, m->ahat.p, m->dvec.p, m->qvec.p, N,
                                                        nullptr, nullptr, w, m->scal.p + 1);
    count_launch(ctx, 2);
}

// loss of the Jacobi preconditioner (zero network output) for pair (r, e)
double jacobi_loss(sfc_mpnn *m, const double *r, const double *e)
{
    sfc_ctx *ctx = m->ctx;
    const int64_t N = m->N;
    SFC_CK(cudaMemsetAsync(m->scal.p, 0, sizeof(double), ctx->stream));
    k_scaled_norm2<<<grid_for(N, 256, ctx->sm_count * 4), 256, 0, ctx->stream>>>(r, m->sdinv.p, N, m->scal.p);
    k_x0<<<grid_for(N, 256), 256, 0, ctx->stream>>>(r, m->sdinv.p, m->scal.p, N, m->x0.p);
    count_launch(ctx, 2);
    pair_residual(m, e, m->x0.p, 1.0);
    double hl = 0;
    download(ctx, &hl, m->scal.p + 1, 1);
    check_tc(m);
    return hl;
}

// weighted loss w * L and its parameter gradient for pair (r, e) (device
// FP64); gradients accumulate into grads; returns w * L
double loss_grad(sfc_mpnn *m, const double *r, const double *e, double w)
{
    sfc_ctx *ctx = m->ctx;
    const sfc_system *s = m->op_sys;
    const int64_t N = m->N;
    forward(m, r);
    const int rows = tc_dense_rows(ctx, N);
    ProfScope ps(ctx, "mpnn_backward", 0.0);
    pair_residual(m, e, m->yhat.p, w);
    // qvec = dL/dyhat
    float *dHa = m->dH0.p, *dHb = m->dH1.p;
    k_decoder_bwd<<<grid_for(N * 32, 256, ctx->sm_count * 4), 256, 0, ctx->stream>>>(m->qvec.p, m->H[LAYERS].p, m->params.p, s->mask.p, N, dHa,
                                                       m->grads.p);
    count_launch(ctx);
    for (int l = LAYERS; l >= 1; --l) {
        const __nv_bfloat16 *W = m->wbf.p + (l - 1) * H * 2 * H;
        float *GW = m->grads.p + OFF_L + (l - 1) * LSZ;
        if (use_tc())
            k_dense_bwd_w_tc<<<tc_grid(m, N), 256, kTcFwdSmem, ctx->stream>>>(dHa, m->H[l].p, m->H[l - 1].p,
                                                                               m->Y[l].p, N, GW, GW + H * 2 * H,
                                                                               m->tc_err.p);
        else
            k_dense_bwd_w<<<(unsigned)(ctx->sm_count * 2), 256, 0, ctx->stream>>>(dHa, m->H[l].p, m->H[l - 1].p,
                                                                                  m->Y[l].p, N, GW, GW + H * 2 * H);
        if (use_tc())
            k_dense_bwd_x_tc<<<tc_tiles(m, N, rows), 512, (size_t)rows * H * 2 + kTcXBBytes + 16, ctx->stream>>>(
                dHa, m->H[l].p, W + LAYERS * H * 2 * H, N, rows, dHb, m->dY.p, m->tc_err.p);
        else
            k_dense_bwd_x<<<gwarp(ctx), 256, 0, ctx->stream>>>(dHa, m->H[l].p, W, N, dHb, m->dY.p);
        // dH(l-1) += Ahat^T dY (Ahat is symmetric)
        k_agg64<<<ctx->sm_count, 1024, 0, ctx->stream>>>(s->row_ptr.p, s->col.p, m->ahat.p, m->dY.p, dHb, N, 1);
        count_launch(ctx, 3);
        std::swap(dHa, dHb);
    }
    k_encoder_bwd<<<grid_for(N * H, 256, ctx->sm_count * 4), 256, 0, ctx->stream>>>(dHa, m->H[0].p, m->x0.p,
                                                                                     m->ax0.p, N, m->grads.p);
    count_launch(ctx);
    double hl = 0;
    download(ctx, &hl, m->scal.p + 1, 1);
    check_tc(m);
    return hl;
}

// z = M(r) (device FP64 vectors): the inference kernels, no host
// synchronisation.  With `scaled`, scal[0] and ax0 already hold |D^-1/2 r|^2
// and FP32(D^-1/2 r).
void apply(sfc_mpnn *m, const double *r, double *z, bool scaled = false)
{
    sfc_ctx *ctx = m->ctx;
    const sfc_system *s = m->op_sys;
    const int64_t N = m->N;
    ProfScope ps(ctx, "mpnn_apply", 0.0);
    if (!scaled) {
        SFC_CK(cudaMemsetAsync(m->scal.p, 0, sizeof(double), ctx->stream));
        k_scaled_norm2<<<grid_for(N, 256, ctx->sm_count * 4), 256, 0, ctx->stream>>>(r, m->sdinv.p, N, m->scal.p,
                                                                                       m->ax0.p);
        count_launch(ctx);
    }
    k_encoder_inf<<<gwarp(ctx), 256, 0, ctx->stream>>>(s->row_ptr.p, s->col.p, m->ahat.p, m->ax0.p, m->scal.p,
                                                       m->params.p, N, m->x0.p, reinterpret_cast<uint4 *>(m->hb[0].p));
    count_launch(ctx);
    if (use_tc()) {
        tc_grid(m, N);
        const int rows = tc_layer_rows(ctx, N);
        const int64_t tiles = (N + rows - 1) / rows;
        const unsigned gt =
            (unsigned)(std::min<int64_t>((tiles + ctx->sm_count - 1) / ctx->sm_count, 4) * ctx->sm_count);
        for (int l = 0; l < LAYERS; ++l) {
            const uint32_t *hin = reinterpret_cast<const uint32_t *>(m->hb[l & 1].p);
            uint32_t *hout = reinterpret_cast<uint32_t *>(m->hb[(l + 1) & 1].p);
            const __nv_bfloat16 *W = m->wbf.p + l * H * 2 * H;
            const float *b = m->params.p + OFF_L + l * LSZ + H * 2 * H;
            if (l + 1 < LAYERS)
                k_layer_tc<false><<<gt, 256, tc_layer_smem(rows), ctx->stream>>>(s->row_ptr.p, s->col.p, m->ahat.p, hin, W, b, N,
                                                                     rows, ctx->sm_count, hout, m->params.p, m->x0.p, m->sdinv.p,
                                                                     s->mask.p, m->scal.p, nullptr, m->tc_err.p);
            else
                k_layer_tc<true><<<gt, 256, tc_layer_smem(rows), ctx->stream>>>(s->row_ptr.p, s->col.p, m->ahat.p, hin, W, b, N,
                                                                    rows, ctx->sm_count, nullptr, m->params.p, m->x0.p, m->sdinv.p,
                                                                    s->mask.p, m->scal.p, z, m->tc_err.p);
            count_launch(ctx);
        }
        return;
    }
    const unsigned g = (unsigned)std::min<int64_t>((N + 63) / 64, (int64_t)ctx->sm_count * 12);
    for (int l = 0; l < LAYERS; ++l) {
        const uint32_t *hin = reinterpret_cast<const uint32_t *>(m->hb[l & 1].p);
        uint32_t *hout = reinterpret_cast<uint32_t *>(m->hb[(l + 1) & 1].p);
        const __nv_bfloat16 *W = m->wbf.p + l * H * 2 * H;
        const float *b = m->params.p + OFF_L + l * LSZ + H * 2 * H;
        if (l + 1 < LAYERS)
            k_layer_inf<false><<<g, 128, 0, ctx->stream>>>(s->row_ptr.p, s->col.p, m->ahat.p, hin, W, b, N, hout,
                                                           m->params.p, m->x0.p, m->sdinv.p, s->mask.p, m->scal.p,
                                                           nullptr);
        else
            k_layer_inf<true><<<g, 128, 0, ctx->stream>>>(s->row_ptr.p, s->col.p, m->ahat.p, hin, W, b, N, nullptr,
                                                          m->params.p, m->x0.p, m->sdinv.p, s->mask.p, m->scal.p, z);
        count_launch(ctx);
    }
}

void adam_step(sfc_mpnn *m, double lr)
{
    ++m->step;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
    k_adam<<<64, 256, 0, m->ctx->stream>>>(m->params.p, m->grads.p, m->adam_m.p, m->adam_v.p, NPARAM, (float)lr, b1, b2,
                                           1e-8f, c1, c2, 1.0f);
    count_launch(m->ctx);
    refresh_bf16(m);
}

__global__ void k_resid_pair(const double *__restrict__ b, const double *__restrict__ Sx, const double *__restrict__ xs,
                             const double *__restrict__ x, int64_t N, double *__restrict__ r, double *__restrict__ e)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
        r[i] = b[i] - Sx[i];
        e[i] = xs[i] - x[i];
    }
}

// Residual/error pairs from Jacobi-PCG on the system's right-hand side b:
// x* converged to 1e-12; x_k = k iterations of PCG from 0, for k = 0 and
// max_pairs - 1 values spaced geometrically up to the iteration at which
// |r_k| / |b| first drops below `floor` (later iterates carry too few digits
// of their error).  Each pair's weight is 1 / (its Jacobi loss) when
// `normalize`, else 1.
void make_pairs(sfc_mpnn *m, sfc_system *s, int max_pairs, double floor, bool normalize)
{
    sfc_ctx *ctx = m->ctx;
    const int64_t N = s->N;
    DBuf<double> b, xs, xk, t;
    b.alloc(N);
    xs.alloc(N);
    xk.alloc(N);
    t.alloc(N);
    lifted_rhs(s, b.p);
    const PcgStats ref = pcg64(s, b.p, xs.p, 1e-12, 200000, false);
    SFC_REQUIRE(ref.converged, "Jacobi-PCG did not converge while generating training pairs");
    const PcgStats fl = pcg64(s, b.p, xk.p, floor, 200000, false);
    const int kmax = std::max(1, fl.iters);
    std::vector<int> ks{0};
    for (int j = 1; j < max_pairs; ++j) {
        const int k = (int)std::lround(std::pow((double)kmax, (double)j / (double)std::max(1, max_pairs - 1)));
        if (k > ks.back()) ks.push_back(k);
    }
    const int np = (int)ks.size();
    m->pr.reserve(N * np);
    m->pe.reserve(N * np);
    m->pw.assign(np, 1.0);
    for (int j = 0; j < np; ++j) {
        if (ks[j] == 0)
            SFC_CK(cudaMemsetAsync(xk.p, 0, N * 8, ctx->stream));
        else
            pcg64(s, b.p, xk.p, 1e-300, ks[j], false);
        spmv_op64(s, xk.p, t.p);
        k_resid_pair<<<grid_for(N, 256), 256, 0, ctx->stream>>>(b.p, t.p, xs.p, xk.p, N, m->pr.p + j * N,
                                                               m->pe.p + j * N);
        count_launch(ctx);
        if (normalize) {
            const double lj = jacobi_loss(m, m->pr.p + j * N, m->pe.p + j * N);
            m->pw[j] = lj > 0 ? 1.0 / lj : 1.0;
        }
    }
    m->npairs = np;
    SFC_CK(cudaStreamSynchronize(ctx->stream));
}

__global__ void k_resid(const double *__restrict__ b, const double *__restrict__ Sx, int64_t n, double *__restrict__ r)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        r[i] = b[i] - Sx[i];
}

__global__ void k_axpy(double *__restrict__ y, const double *__restrict__ x, double a, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] += a * x[i];
}

// alpha = (p.r)/(p.q); x += alpha p; r -= alpha q; rr' += r.r; and the
// network's input: rhat = FP32(D^-1/2 r), scal += |D^-1/2 r|^2
__global__ void k_fcg_update(double *__restrict__ x, double *__restrict__ r, const double *__restrict__ p,
                             const double *__restrict__ q, int64_t n, const double *pq, const double *pr,
                             double *rr_next, const float *__restrict__ sdinv, float *__restrict__ rhat, double *scal,
                             const int *done, int *err)
{
    __shared__ double sh[32];
    if (*done) return;
    const double den = *pq;
    if (!(den > 0.0)) {
        if (threadIdx.x == 0) atomicExch(err, 1);
        return;
    }
    const double alpha = *pr / den;
    double c = 0, c2 = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        x[i] += alpha * p[i];
        const double ri = r[i] - alpha * q[i];
        r[i] = ri;
        c += ri * ri;
        const double t = ri * (double)sdinv[i];
        c2 += t * t;
        rhat[i] = (float)t;
    }
    c = block_sum_d(c, sh);
    if (threadIdx.x == 0) atomicAdd(rr_next, c);
    c2 = block_sum_d(c2, sh);
    if (threadIdx.x == 0) atomicAdd(scal, c2);
}

// beta = -(z.q)/(p.q); p = z + beta p; pr' += p.r; clears scal for the next
// update.  Where the update brought rr to the threshold: *done = it instead.
__global__ void k_fcg_pupdate(double *__restrict__ p, const double *__restrict__ z, const double *__restrict__ r,
                              int64_t n, const double *zq, const double *pq, double *pr_next, const double *rr,
                              double thr, int it, double *scal, int *done, const int *err)
{
    __shared__ double sh[32];
    if (*done || *err) return;
    const bool last = *rr <= thr;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *scal = 0.0;
        if (last) *done = it;
    }
    if (last) return;
    const double beta = -*zq / *pq;
    double c = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double pi = z[i] + beta * p[i];
        p[i] = pi;
        c += pi * r[i];
    }
    c = block_sum_d(c, sh);
    if (threadIdx.x == 0) atomicAdd(pr_next, c);
}

struct FcgRun {
    double *x, *r, *z, *p, *q, *mark;
    int it, max_iter, check, stall, mark_it;
    double thr, mark_rr;
};

// k_fcg from slot run.it on
FcgWhy fcg_run(sfc_mpnn *m, sfc_system *s, FcgRun &run)
{
    sfc_ctx *ctx = s->ctx;
    const int64_t N = s->N;
    FcgArgs g{};
    const Format f = grid_operator(s, g.op, false);
    FcgRuns o{};
    // rows of a window outside the matrix, at most: its reach, and the rest of the four rows and the run
    const int64_t margin = f == DIA ? s->dia_off[s->dia_nd - 1] + 8 : 0;
    if (f == DIA) {
        for (int d = 0; d < s->dia_nd;) {
            const int first = s->dia_off[d];
            o.off[o.runs++] = first;
            while (d < s->dia_nd && s->dia_off[d] < first + 3) ++d;
        }
        const size_t rows = (size_t)(N + 2 * margin) * H;
        // without room the gather reads the rows
        if (!reserve_spare(spare(m->win, (size_t)o.runs * 3 * ((N + 3) / 4 * 4)), spare(m->hw[0], rows), spare(m->hw[1], rows)))
            o.runs = 0;
    }
    if (o.runs) {
        k_fcg_window<<<grid_for(N, 256), 256, 0, ctx->stream>>>(o, s->row_ptr.p, s->col.p, m->ahat.p, N, m->win.p);
        count_launch(ctx);
        g.win = reinterpret_cast<const float4 *>(m->win.p);
        g.runs = o.runs;
        std::copy(o.off, o.off + o.runs, g.woff);
    }
    g.op.x = run.x;
    g.op.r = run.r;
    g.op.p = run.p;
    g.op.q = run.q;
    g.op.sums = m->fcg_sc.p;
    g.op.max_iter = run.max_iter;
    g.op.out = m->fcg_flags.p;
    g.op.bar = reinterpret_cast<unsigned *>(m->fcg_flags.p + 3);
    g.rp = s->row_ptr.p;
    g.col = s->col.p;
    g.ahat = m->ahat.p;
    g.sdinv = m->sdinv.p;
    g.mask = s->mask.p;
    g.W = m->wbf.p;
    g.P = m->params.p;
    g.rhat = m->ax0.p;
    g.x0 = m->x0.p;
    __nv_bfloat16 *hb[2] = {m->hb[0].p, m->hb[1].p};
    if (o.runs)
        for (int k = 0; k < 2; ++k) {
            hb[k] = m->hw[k].p + margin * H;
            SFC_CK(cudaMemsetAsync(m->hw[k].p, 0, margin * H * 2, ctx->stream));
            SFC_CK(cudaMemsetAsync(hb[k] + N * H, 0, margin * H * 2, ctx->stream));
        }
    g.hb0 = reinterpret_cast<uint32_t *>(hb[0]);
    g.hb1 = reinterpret_cast<uint32_t *>(hb[1]);
    g.z = run.z;
    g.mark = run.mark;
    g.it0 = run.it;
    g.check = run.check;
    g.stall = run.stall;
    g.mark_it = run.mark_it;
    g.thr = run.thr;
    // one CTA per SM, of at least 64 rows
    const int64_t ctas = std::max<int64_t>(1, std::min<int64_t>(ctx->sm_count, N / 64));
    g.per = ((N + ctas - 1) / ctas + 3) / 4 * 4;
    using Kernel = void (*)(FcgArgs);
    const Kernel kernel = f == CSR    ? k_fcg<CSR, false>
                          : f == BSR  ? k_fcg<BSR, false>
                          : f == BDIA ? k_fcg<BDIA, false>
                          : o.runs    ? k_fcg<DIA, true>
                                      : k_fcg<DIA, false>;
    SFC_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFcgSmem));
    SFC_CK(cudaMemsetAsync(g.op.out, 0, 8 * sizeof(int), ctx->stream));
    SFC_CK(cudaMemcpyAsync(run.mark, &run.mark_rr, sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.stream = ctx->stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3((unsigned)((N + g.per - 1) / g.per));
    cfg.blockDim = dim3(kFcgThreads);
    cfg.dynamicSmemBytes = kFcgSmem;
    SFC_CK(cudaLaunchKernelEx(&cfg, kernel, g));
    count_launch(ctx);
    int h[6];
    download(ctx, h, g.op.out, 6);
    if (h[2]) fail(SFC_ERR_TIMEOUT, "learned preconditioner: a grid barrier gave up");
    if (h[5]) fail(SFC_ERR_TIMEOUT, "learned preconditioner: a bounded wait for the tensor-core products gave up");
    download(ctx, &run.mark_rr, run.mark, 1);
    run.it = h[0];
    run.mark_it = h[4];
    return (FcgWhy)h[1];
}

}  // namespace

// Flexible CG (FCG(1), Notay 2000) with z = M(r) from the network, with
// plain Jacobi-PCG as the fallback when the network stalls or breaks down:
// alpha = p.r / p.Sp, p' = z - (z.Sp / p.Sp) p.  The iterations are one
// persistent kernel (k_fcg); with SFC_MPNN_TC=0 they are launches whose scalars
// live on the device, one slot per iteration, and whose flags the host reads
// every check_every iterations.  When the recurrence residual meets tol, the
// true FP64 residual ||b - S x|| is computed; if it misses tol, the method
// restarts from it.
void solve_forward_fcg(sfc_system *s)
{
    sfc_ctx *ctx = s->ctx;
    SFC_REQUIRE(s->mpnn, "no learned preconditioner set (sfc_system_set_mpnn)");
    sfc_mpnn *m = s->mpnn;
    bind(m, s);  // the operator's values may have changed since the last use
    dia_ensure(s);
    const int64_t N = s->N;
    const auto &o = s->opt;
    const int max_iter = o.max_iter > 0 ? o.max_iter : 20000;
    const int check = o.check_every > 0 ? o.check_every : 8;
    const double tol = o.tol > 0 ? o.tol : 1e-8;
    s->X.alloc(N);
    s->blk64.reserve(6 * N);
    double *b = s->blk64.p, *r = b + N, *z = r + N, *p = z + N, *q = p + N, *t = q + N;
    // a slot per iteration for the launches; the persistent kernel goes round a few
    const bool ring = use_tc();
    const int64_t slots = ring ? kSumRing : (int64_t)max_iter + 2;
    m->fcg_sc.reserve(5 * slots + 1);
    double *pq = m->fcg_sc.p, *pr = pq + slots, *rr = pr + slots, *zq = rr + slots, *mark = zq + 2 * slots;
    m->fcg_flags.reserve(8);
    int *done = m->fcg_flags.p, *err = done + 1;
    cudaEvent_t e0, e1;
    SFC_CK(cudaEventCreate(&e0));
    SFC_CK(cudaEventCreate(&e1));
    SFC_CK(cudaEventRecord(e0, ctx->stream));
    SFC_CK(cudaMemsetAsync(m->fcg_sc.p, 0, (5 * slots + 1) * sizeof(double), ctx->stream));
    lifted_rhs(s, b);
    SFC_CK(cudaMemsetAsync(s->X.p, 0, N * 8, ctx->stream));
    SFC_CK(cudaMemcpyAsync(r, b, N * 8, cudaMemcpyDeviceToDevice, ctx->stream));
    const double bb = device_dot(ctx, b, b, N);
    const double thr = tol * tol * bb;
    const unsigned g = grid_for(N, 256, ctx->sm_count * 4);
    auto true_residual = [&]() {  // r = b - S x, returns |r| / |b|
        spmv_op64(s, s->X.p, t);
        k_resid<<<grid_for(N, 256), 256, 0, ctx->stream>>>(b, t, N, r);
        count_launch(ctx);
        return std::sqrt(device_dot(ctx, r, r, N) / bb);
    };
    auto start = [&](int at) {  // direction from the current residual
        const int64_t slot = ring ? at % kSumRing : at;
        if (ring) SFC_CK(cudaMemsetAsync(m->fcg_sc.p, 0, 5 * slots * sizeof(double), ctx->stream));
        apply(m, r, z);
        SFC_CK(cudaMemcpyAsync(p, z, N * 8, cudaMemcpyDeviceToDevice, ctx->stream));
        spmv_op64_dot(s, p, q, pq + slot, nullptr);
        k_fdot<<<g, 256, 0, ctx->stream>>>(p, r, N, pr + slot);
        count_launch(ctx);
    };
    int it = 0, iters = 0, fallback = 0, mark_it = 0;
    constexpr int kStall = 400;
    double mark_rr = bb;
    bool conv = bb == 0.0;
    double rel = 0.0;
    // iterations from slot `it` on to convergence of the recurrence, breakdown
    // (p.Sp <= 0), a stall or the cap; `it` ends at the iteration reached
    auto iterate = [&]() -> FcgWhy {
        if (use_tc()) {
            FcgRun run{s->X.p, r, z, p, q, mark, it, max_iter, check, kStall, mark_it, thr, mark_rr};
            const FcgWhy why = fcg_run(m, s, run);
            it = run.it;
            mark_it = run.mark_it;
            mark_rr = run.mark_rr;
            return why;
        }
        SFC_CK(cudaMemsetAsync(done, 0, 2 * sizeof(int), ctx->stream));
        SFC_CK(cudaMemsetAsync(m->scal.p, 0, sizeof(double), ctx->stream));  // for the next k_fcg_update
        for (; it < max_iter; ++it) {
            k_fcg_update<<<g, 256, 0, ctx->stream>>>(s->X.p, r, p, q, N, pq + it, pr + it, rr + it + 1, m->sdinv.p,
                                                    m->ax0.p, m->scal.p, done, err);
            apply(m, r, z, true);
            k_fdot<<<g, 256, 0, ctx->stream>>>(z, q, N, zq + it);
            k_fcg_pupdate<<<g, 256, 0, ctx->stream>>>(p, z, r, N, zq + it, pq + it, pr + it + 1, rr + it + 1, thr,
                                                      it + 1, m->scal.p, done, err);
            count_launch(ctx, 3);
            spmv_op64_dot(s, p, q, pq + it + 1, done);
            if ((it + 1) % check == 0 || it + 1 == max_iter) {
                int hf[2];
                download(ctx, hf, done, 2);
                if (hf[1]) {
                    ++it;
                    return FCG_BREAKDOWN;
                }
                if (hf[0]) {
                    it = hf[0];
                    return FCG_DONE;
                }
                // stagnation: no 100-fold reduction of the recurrence
                // residual^2 (10-fold of the residual) within kStall iterations
                double rr_now = 0;
                download(ctx, &rr_now, rr + it + 1, 1);
                if (rr_now < 0.01 * mark_rr) {
                    mark_rr = rr_now;
                    mark_it = it + 1;
                } else if (it + 1 - mark_it > kStall) {
                    ++it;
                    return FCG_STALL;
                }
            }
        }
        return FCG_CAP;
    };
    if (!conv) {
        ProfScope ps(ctx, "fcg_iterations", 0.0);
        start(0);
        while (iterate() == FCG_DONE) {
            iters = it;
            rel = true_residual();
            conv = rel <= tol;
            // counts go on from the end of the check interval
            it = (int)std::min<int64_t>(max_iter, ((int64_t)it + check - 1) / check * check);
            if (conv || it >= max_iter) break;
            // the recurrence drifted: restart from the true residual
            start(it);
            mark_it = it;
        }
        if (!conv) {
            // the network failed this system (stagnation, breakdown or the
            // iteration cap): plain FP64 Jacobi-PCG finishes from the current
            // x on the true residual, S d = b - S x, x += d
            it = (int)std::min<int64_t>(max_iter, ((int64_t)it + check - 1) / check * check);
            iters = std::max(iters, it);
            rel = true_residual();
            if (rel > tol) {
                fallback = 1;
                const PcgStats pr = pcg64(s, r, z, tol / rel, max_iter, false);
                k_axpy<<<g, 256, 0, ctx->stream>>>(s->X.p, z, 1.0, N);
                count_launch(ctx);
                iters += pr.iters;
                rel = true_residual();
            }
            conv = rel <= tol * (1.0 + 1e-9);
        }
    }
    SFC_CK(cudaEventRecord(e1, ctx->stream));
    float ms = 0;
    SFC_CK(cudaEventSynchronize(e1));
    SFC_CK(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    check_tc(m);
    s->stats = {};
    s->stats.iterations = iters;
    s->stats.num_rhs = 1;
    s->stats.converged = conv ? 1 : 0;
    s->stats.max_rel_residual = rel;
    s->stats.device_ms = ms;
    s->stats.fallback_columns = fallback;
    if (!conv) fail(SFC_ERR_NOT_CONVERGED, "flexible CG (and the Jacobi-PCG fallback) did not converge within max_iter");
}

}  // namespace sfc

using namespace sfc;

namespace {
int mguard(sfc_ctx *ctx, const std::function<void()> &fn)
{
    try {
        SFC_CK(cudaSetDevice(ctx->device));
        fn();
        return SFC_OK;
    } catch (const Error &e) {
        ctx->err = e.msg;
        if (e.code == SFC_ERR_CUDA) cudaGetLastError();
        return e.code;
    } catch (const std::exception &e) {
        ctx->err = e.what();
        return SFC_ERR_BAD_ARG;
    }
}
}  // namespace

extern "C" {

int64_t sfc_mpnn_num_params(void) { return NPARAM; }

int32_t sfc_mpnn_create(sfc_ctx_t *ctx, uint64_t seed, sfc_mpnn_t **out)
{
    if (!ctx || !out) return SFC_ERR_BAD_ARG;
    *out = nullptr;
    sfc_mpnn *m = new (std::nothrow) sfc_mpnn();
    if (!m) return SFC_ERR_NO_MEMORY;
    int rc = mguard(ctx, [&] {
        m->ctx = ctx;
        std::vector<float> p(NPARAM, 0.f);
        std::mt19937_64 gen(seed);
        std::normal_distribution<float> nd(0.f, 1.f);
        for (int k = 0; k < 2 * H; ++k) p[OFF_EW + k] = nd(gen) * 0.7f;
        for (int k = 0; k < H; ++k) p[OFF_EB + k] = 0.05f;
        for (int l = 0; l < LAYERS; ++l)
            for (int k = 0; k < H * 2 * H; ++k) p[OFF_L + l * LSZ + k] = nd(gen) * std::sqrt(2.f / (2 * H));
        // decoder starts at zero: the untrained network is exactly Jacobi
        m->params.alloc(NPARAM);
        m->grads.alloc(NPARAM);
        m->adam_m.alloc(NPARAM);
        m->adam_v.alloc(NPARAM);
        m->wbf.alloc(2 * LAYERS * H * 2 * H);
        m->scal.alloc(4);
        upload(ctx, m->params, p.data(), NPARAM);
        SFC_CK(cudaMemsetAsync(m->adam_m.p, 0, NPARAM * 4, ctx->stream));
        SFC_CK(cudaMemsetAsync(m->adam_v.p, 0, NPARAM * 4, ctx->stream));
        refresh_bf16(m);
        SFC_CK(cudaStreamSynchronize(ctx->stream));
    });
    if (rc != SFC_OK) {
        delete m;
        return rc;
    }
    *out = m;
    return SFC_OK;
}

int32_t sfc_mpnn_destroy(sfc_mpnn_t *m)
{
    if (!m) return SFC_OK;
    cudaSetDevice(m->ctx->device);
    cudaStreamSynchronize(m->ctx->stream);
    delete m;
    return SFC_OK;
}

int32_t sfc_mpnn_get_params(const sfc_mpnn_t *m, float *out, int64_t n)
{
    if (!m || !out || n != NPARAM) return SFC_ERR_BAD_ARG;
    return mguard(m->ctx, [&] { download(m->ctx, out, m->params.p, NPARAM); });
}

int32_t sfc_mpnn_set_params(sfc_mpnn_t *m, const float *in, int64_t n)
{
    if (!m || !in || n != NPARAM) return SFC_ERR_BAD_ARG;
    return mguard(m->ctx, [&] {
        upload(m->ctx, m->params, in, NPARAM);
        refresh_bf16(m);
        SFC_CK(cudaStreamSynchronize(m->ctx->stream));
    });
}

int32_t sfc_mpnn_save(const sfc_mpnn_t *m, const char *path)
{
    if (!m || !path) return SFC_ERR_BAD_ARG;
    return mguard(m->ctx, [&] {
        std::vector<float> buf(3 * (size_t)NPARAM);
        download(m->ctx, buf.data(), m->params.p, NPARAM);
        download(m->ctx, buf.data() + NPARAM, m->adam_m.p, NPARAM);
        download(m->ctx, buf.data() + 2 * NPARAM, m->adam_v.p, NPARAM);
        FILE *f = std::fopen(path, "wb");
        SFC_REQUIRE(f, std::string("cannot open ") + path);
        const int64_t hdr[3] = {0x53464d50, NPARAM, m->step};  // "SFMP"
        bool ok = std::fwrite(hdr, sizeof hdr, 1, f) == 1 && std::fwrite(buf.data(), 4, buf.size(), f) == buf.size();
        std::fclose(f);
        SFC_REQUIRE(ok, "checkpoint write failed");
    });
}

int32_t sfc_mpnn_load(sfc_mpnn_t *m, const char *path)
{
    if (!m || !path) return SFC_ERR_BAD_ARG;
    return mguard(m->ctx, [&] {
        FILE *f = std::fopen(path, "rb");
        SFC_REQUIRE(f, std::string("cannot open ") + path);
        int64_t hdr[3] = {};
        std::vector<float> buf(3 * (size_t)NPARAM);
        bool ok = std::fread(hdr, sizeof hdr, 1, f) == 1 && hdr[0] == 0x53464d50 && hdr[1] == NPARAM &&
                  std::fread(buf.data(), 4, buf.size(), f) == buf.size();
        std::fclose(f);
        SFC_REQUIRE(ok, "not a checkpoint of this network");
        upload(m->ctx, m->params, buf.data(), NPARAM);
        upload(m->ctx, m->adam_m, buf.data() + NPARAM, NPARAM);
        upload(m->ctx, m->adam_v, buf.data() + 2 * NPARAM, NPARAM);
        m->step = hdr[2];
        refresh_bf16(m);
        SFC_CK(cudaStreamSynchronize(m->ctx->stream));
    });
}

int32_t sfc_mpnn_loss_grad(sfc_mpnn_t *m, sfc_system_t *s, const double *r, const double *e, double *loss,
                           float *grad)
{
    if (!m || !s || !r || !e) return SFC_ERR_BAD_ARG;
    return mguard(m->ctx, [&] {
        bind(m, s);
        DBuf<double> &dr = m->io[0], &de = m->io[1];
        upload(m->ctx, dr, r, s->N);
        upload(m->ctx, de, e, s->N);
        SFC_CK(cudaMemsetAsync(m->grads.p, 0, NPARAM * 4, m->ctx->stream));
        const double l = loss_grad(m, dr.p, de.p, 1.0);
        if (loss) *loss = l;
        if (grad) download(m->ctx, grad, m->grads.p, NPARAM);
    });
}

int32_t sfc_mpnn_apply(sfc_mpnn_t *m, sfc_system_t *s, const double *r, double *z)
{
    if (!m || !s || !r || !z) return SFC_ERR_BAD_ARG;
    return mguard(m->ctx, [&] {
        bind(m, s);
        DBuf<double> &dr = m->io[0], &dz = m->io[1];
        upload(m->ctx, dr, r, s->N);
        dz.reserve(s->N);
        apply(m, dr.p, dz.p);
        download(m->ctx, z, dz.p, s->N);
        check_tc(m);
    });
}

int32_t sfc_mpnn_default_train_options(sfc_mpnn_train_options_t *o)
{
    if (!o) return SFC_ERR_BAD_ARG;
    o->steps = 500;
    o->batch = 4;
    o->max_pairs = 16;
    o->normalize = 1;
    o->lr = 1e-3;
    o->pair_floor = 1e-6;
    o->seed = 0;
    return SFC_OK;
}

int32_t sfc_mpnn_train(sfc_mpnn_t *m, sfc_system_t *s, const sfc_mpnn_train_options_t *o, double *loss_history)
{
    if (!m || !s || !o || o->steps < 0 || o->batch < 1 || o->max_pairs < 1 || o->max_pairs > 64 || !(o->lr > 0) ||
        !(o->pair_floor > 0 && o->pair_floor < 1)) {
        if (m) m->ctx->err = "invalid training options";
        return SFC_ERR_BAD_ARG;
    }
    return mguard(m->ctx, [&] {
        bind(m, s);
        make_pairs(m, s, o->max_pairs, o->pair_floor, o->normalize != 0);
        const int64_t N = s->N;
        std::mt19937_64 gen(o->seed ^ (uint64_t)(m->step * 0x9E3779B97F4A7C15ull));
        std::uniform_int_distribution<int> pick(0, m->npairs - 1);
        for (int t = 0; t < o->steps; ++t) {
            SFC_CK(cudaMemsetAsync(m->grads.p, 0, NPARAM * 4, m->ctx->stream));
            double acc = 0;
            for (int j = 0; j < o->batch; ++j) {
                const int k = pick(gen);
                acc += loss_grad(m, m->pr.p + k * N, m->pe.p + k * N, m->pw[k] / o->batch);
            }
            adam_step(m, o->lr);
            if (loss_history) loss_history[t] = acc;
        }
        SFC_CK(cudaStreamSynchronize(m->ctx->stream));
    });
}

int32_t sfc_system_set_mpnn(sfc_system_t *s, sfc_mpnn_t *m)
{
    if (!s) return SFC_ERR_BAD_ARG;
    s->mpnn = m;
    if (m) m->op_sys = nullptr;  // rebind on next use
    return SFC_OK;
}

}  // extern "C"
