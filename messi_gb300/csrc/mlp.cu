// mlp.cu -- the learned MCMC proposal network (HP3): a BF16 MLP with a
// Gaussian-mixture head, trained and evaluated on the GPU.
//
// The reference's MCMC moves (src/MCMC.jl:1307-1674) have no learned part;
// this network is the proposal described for the learned chain: input = the
// current model parameters (transformed) + alignment summary statistics,
// output = a K-component diagonal Gaussian mixture over the free parameters.
//
// Layout: three linear layers in -> H -> H -> out with SiLU after the first
// two.  Weights are kept in FP32 (Adam master copy) and BF16 (the copy the
// forward/backward kernels read); activations are BF16, and so are the
// gradient operands of the backward GEMMs (rounded while a tile is staged);
// every product is accumulated in FP32.  Every GEMM runs on the tensor cores
// (gemm_bf16_kernel: 32 x 32 CTA tiles, four warps of 16 x 16, BF16
// mma.sync m16n8k16 with FP32 accumulators) with its epilogue fused: bias,
// bias + SiLU (writing the FP32 pre-activation and the BF16 activation), or
// the SiLU derivative of the backward pass.  The network is small (batch a
// few hundred, width 256), so a GEMM is latency bound: small tiles for more
// CTAs, a 256-wide K chunk staged per barrier, and the fused epilogues
// remove the elementwise launches between the GEMMs.
//
// Networks whose activations of 16 rows fit half an SM's shared memory (widths
// up to about 350) run in two kernels instead: mlp_rows_kernel takes 16 rows of
// the batch through forward, loss and the backward data path, mlp_wgrad_kernel
// forms all weight and bias gradients.  The GEMM per layer remains for wider
// networks.
//
// Head per sample: [K logits | K*D means | K*D log-sd]; the loss is the
// negative log-likelihood of a target vector under the mixture.
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "internal.h"

struct messi_mlp {
    int in = 0, H = 0, out = 0, K = 0, D = 0;
    int cap = 0;                       // batch capacity of the activation buffers
    // parameters: W1[H][in] b1[H] W2[H][H] b2[H] W3[out][H] b3[out]
    int nparam = 0;
    float* p32 = nullptr;              // FP32 master
    __nv_bfloat16* p16 = nullptr;      // BF16 copy (GEMM per layer only)
    float* grad = nullptr;
    float* m1 = nullptr;               // Adam moments
    float* m2 = nullptr;
    int64_t steps = 0;
    // activations
    __nv_bfloat16 *x = nullptr, *a1 = nullptr, *a2 = nullptr;   // inputs / post-SiLU (BF16)
    float *z1 = nullptr, *z2 = nullptr, *y = nullptr;           // pre-activations, head (FP32)
    float *dy = nullptr, *d2 = nullptr, *d1 = nullptr;          // gradients w.r.t. y, a2/z2, a1/z1
    float* target = nullptr;
    float* loss = nullptr;             // [cap]
    float* stage = nullptr;            // host-pinned staging
    // two-kernel form (fused): weights as BF16 with K padded to 32 and zero
    // filled, W1 W2 W3 W2^T W3^T; the batch's operands of the weight gradients,
    // feature-major; per-CTA column sums for the bias gradients
    bool fused = false;
    __nv_bfloat16* w16 = nullptr;
    __nv_bfloat16 *xT = nullptr, *a1T = nullptr, *a2T = nullptr, *dyT = nullptr, *d2T = nullptr, *d1T = nullptr;
    float* colsum = nullptr;
};

namespace messi {

namespace {

__device__ __forceinline__ float silu(float z);
__device__ __forceinline__ float dsilu(float z);

__device__ __forceinline__ __nv_bfloat16 to_bf(float v) { return __float2bfloat16(v); }
__device__ __forceinline__ __nv_bfloat16 to_bf(__nv_bfloat16 v) { return v; }


// CTA tile 32 x 32 (four warps of 16 x 16), the K extent staged in chunks of
// kBK: the GEMMs of this network are a few hundred rows, so the CTA count,
// not the per-CTA rate, bounds them; a whole chunk's loads are issued before
// the one CTA barrier, so a chunk costs one memory round trip.
constexpr int kBM = 32, kBN = 32, kBK = 256, kPad = 8;

// Four consecutive elements (16 B of FP32 or 8 B of BF16), rounded to BF16.
__device__ __forceinline__ void load4_bf(const float* p, __nv_bfloat16 (&o)[4])
{
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = __float2bfloat16(v.x);
    o[1] = __float2bfloat16(v.y);
    o[2] = __float2bfloat16(v.z);
    o[3] = __float2bfloat16(v.w);
}
__device__ __forceinline__ void load4_bf(const __nv_bfloat16* p, __nv_bfloat16 (&o)[4])
{
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
    const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&v);
    o[0] = b[0];
    o[1] = b[1];
    o[2] = b[2];
    o[3] = b[3];
}

// Stage rows r0.. of one operand tile, [rows][k] in shared memory (rows of
// kBK + kPad): X(r, k) = X[r*srow + k*sk].  With vec (unit stride along the
// fast index, the other stride a multiple of 4, the base aligned), four
// consecutive elements of the fast index come in one load.
template <int ROWS, typename T>
__device__ __forceinline__ void stage_tile(__nv_bfloat16 (*dst)[kBK + 8], const T* __restrict__ X, long long srow,
                                           long long sk, int r0, int nrows, int k0, int kc, int kc16, bool vec)
{
    const bool k_fast = (sk == 1);
    if (vec) {
        for (int e = threadIdx.x; e < ROWS * kBK / 4; e += blockDim.x) {
            // groups of four along the fast index
            const int r = k_fast ? e / (kBK / 4) : 4 * (e % (ROWS / 4));
            const int c = k_fast ? 4 * (e % (kBK / 4)) : e / (ROWS / 4);
            if (c >= kc16) continue;
            __nv_bfloat16 v[4];
            const int rr = r0 + r, kk = k0 + c;
            if (k_fast) {
                if (rr < nrows && c + 3 < kc) load4_bf(X + rr * srow + kk, v);
                else
                    for (int q = 0; q < 4; q++)
                        v[q] = (rr < nrows && c + q < kc) ? to_bf(X[rr * srow + kk + q]) : __float2bfloat16(0.f);
                for (int q = 0; q < 4; q++) dst[r][c + q] = v[q];
            } else {
                if (rr + 3 < nrows && c < kc) load4_bf(X + rr + kk * sk, v);
                else
                    for (int q = 0; q < 4; q++)
                        v[q] = (rr + q < nrows && c < kc) ? to_bf(X[(rr + q) + kk * sk]) : __float2bfloat16(0.f);
                for (int q = 0; q < 4; q++) dst[r + q][c] = v[q];
            }
        }
    } else {
        for (int e = threadIdx.x; e < ROWS * kBK; e += blockDim.x) {
            const int r = k_fast ? e / kBK : e % ROWS, c = k_fast ? e % kBK : e / ROWS;
            if (c >= kc16) continue;
            const int rr = r0 + r, kk = k0 + c;
            dst[r][c] = (rr < nrows && c < kc) ? to_bf(X[rr * srow + kk * sk]) : __float2bfloat16(0.f);
        }
    }
}

template <typename T>
__host__ __device__ inline bool vec_ok(const T* p, long long srow, long long sk)
{
    const size_t align = sizeof(T) * 4;
    const bool unit = (srow == 1) != (sk == 1) && (srow == 1 || sk == 1);
    const long long other = (sk == 1) ? srow : sk;
    return unit && other % 4 == 0 && (reinterpret_cast<size_t>(p) % align) == 0;
}

// GEMM epilogues
enum GemmMode {
    kStoreBias = 0,  // C = acc + bias[n]
    kAccumulate = 1, // C += acc
    kBiasSilu = 2,   // z = acc + bias[n]; C = z (FP32); act = bf16(silu(z))
    kDsilu = 3       // C = acc * dsilu(z[m][n])
};

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// C[m][n] (row stride scm) = epilogue(sum_k A(m, k) * B(k, n)) with
// A(m,k) = A[m*sam + k*sak], B(k,n) = B[k*sbk + n*sbn]; operands are rounded
// to BF16 as they are staged in shared memory ([row][k], k contiguous, rows
// padded by 8 so the fragment loads hit 32 distinct banks).
template <typename TA, typename TB>
__global__ void __launch_bounds__(128) gemm_bf16_kernel(int M, int N, int K, const TA* __restrict__ A, long long sam,
                                                        long long sak, const TB* __restrict__ B, long long sbk,
                                                        long long sbn, const float* __restrict__ bias,
                                                        float* __restrict__ C, long long scm, int mode,
                                                        const float* __restrict__ z, __nv_bfloat16* __restrict__ act)
{
    __shared__ __align__(16) __nv_bfloat16 As[kBM][kBK + kPad];
    __shared__ __align__(16) __nv_bfloat16 Bs[kBN][kBK + kPad];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * 16;
    const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
    float acc[2][4];
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[j][q] = 0.f;
    // consecutive threads walk the operand's unit-stride index (coalesced)
    const bool va = vec_ok(A, sam, sak), vb = vec_ok(B, sbn, sbk);
    for (int k0 = 0; k0 < K; k0 += kBK) {
        const int kc = min(kBK, K - k0);
        const int kc16 = (kc + 15) & ~15;  // chunk rounded up to whole k16 steps (zero padded)
        if (k0 > 0) __syncthreads();
        stage_tile<kBM>(As, A, sam, sak, m0, M, k0, kc, kc16, va);
        stage_tile<kBN>(Bs, B, sbn, sbk, n0, N, k0, kc, kc16, vb);
        __syncthreads();
        for (int ks = 0; ks < kc16; ks += 16) {
            uint32_t af[4], bf[2][2];
            const int r = wm + g;
            af[0] = *reinterpret_cast<const uint32_t*>(&As[r][ks + 2 * t]);
            af[1] = *reinterpret_cast<const uint32_t*>(&As[r + 8][ks + 2 * t]);
            af[2] = *reinterpret_cast<const uint32_t*>(&As[r][ks + 2 * t + 8]);
            af[3] = *reinterpret_cast<const uint32_t*>(&As[r + 8][ks + 2 * t + 8]);
#pragma unroll
            for (int nt = 0; nt < 2; nt++) {
                const int c = wn + nt * 8 + g;
                bf[nt][0] = *reinterpret_cast<const uint32_t*>(&Bs[c][ks + 2 * t]);
                bf[nt][1] = *reinterpret_cast<const uint32_t*>(&Bs[c][ks + 2 * t + 8]);
            }
#pragma unroll
            for (int nt = 0; nt < 2; nt++) mma_bf16(acc[nt], af, bf[nt][0], bf[nt][1]);
        }
    }
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int m = m0 + wm + g + 8 * (q >> 1);
            const int n = n0 + wn + nt * 8 + 2 * t + (q & 1);
            if (m >= M || n >= N) continue;
            const long long o = m * scm + n;
            const float v = acc[nt][q];
            if (mode == kStoreBias) {
                C[o] = v + (bias ? bias[n] : 0.f);
            } else if (mode == kAccumulate) {
                C[o] += v;
            } else if (mode == kBiasSilu) {
                const float zz = v + (bias ? bias[n] : 0.f);
                C[o] = zz;
                act[o] = __float2bfloat16(silu(zz));
            } else {
                C[o] = v * dsilu(z[o]);
            }
        }
}

template <typename TA, typename TB>
int gemm(messi_ctx* ctx, int M, int N, int K, const TA* A, long long sam, long long sak, const TB* B, long long sbk,
         long long sbn, const float* bias, float* C, long long scm, int mode, const float* z = nullptr,
         __nv_bfloat16* act = nullptr)
{
    dim3 grid((N + kBN - 1) / kBN, (M + kBM - 1) / kBM);
    gemm_bf16_kernel<TA, TB><<<grid, 128, 0, ctx->stream>>>(M, N, K, A, sam, sak, B, sbk, sbn, bias, C, scm, mode, z,
                                                            act);
    LAUNCH_CHECK(ctx, "gemm_bf16_kernel");
    return MESSI_OK;
}

__device__ __forceinline__ float silu(float z) { return z / (1.f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z)
{
    const float s = 1.f / (1.f + __expf(-z));
    return s * (1.f + z * (1.f - s));
}

__global__ void to_bf16_kernel(const float* __restrict__ s, __nv_bfloat16* __restrict__ d, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) d[i] = __float2bfloat16(s[i]);
}

__global__ void colsum_kernel(const float* __restrict__ dY, int M, int N, float* __restrict__ db)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    float s = 0.f;
    for (int m = 0; m < M; m++) s += dY[(long long)m * N + n];
    db[n] += s;
}

// Mixture negative log-likelihood per sample and its gradient w.r.t. the head.
// y: [K logits | K*D means | K*D log-sd], log-sd clamped to [-7, 5].
__global__ void mixture_nll_kernel(const float* __restrict__ y, const float* __restrict__ tgt, int M, int K, int D,
                                   float* __restrict__ loss, float* __restrict__ dy, float inv_batch)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    const int O = K + 2 * K * D;
    const float* ym = y + (long long)m * O;
    const float* x = tgt + (long long)m * D;
    float* g = dy + (long long)m * O;
    float lw[8], lp[8];
    float mx = -INFINITY;
    for (int k = 0; k < K; k++) mx = fmaxf(mx, ym[k]);
    float se = 0.f;
    for (int k = 0; k < K; k++) se += __expf(ym[k] - mx);
    const float lse_w = mx + __logf(se);
    const float c = -0.91893853320467274f * D;  // -D/2 log(2 pi)
    float best = -INFINITY;
    for (int k = 0; k < K; k++) {
        lw[k] = ym[k] - lse_w;
        float s = c;
        for (int d = 0; d < D; d++) {
            const float ls = fminf(fmaxf(ym[K + K * D + k * D + d], -7.f), 5.f);
            const float r = (x[d] - ym[K + k * D + d]) * __expf(-ls);
            s += -0.5f * r * r - ls;
        }
        lp[k] = lw[k] + s;
        best = fmaxf(best, lp[k]);
    }
    float tot = 0.f;
    for (int k = 0; k < K; k++) tot += __expf(lp[k] - best);
    const float ll = best + __logf(tot);
    loss[m] = -ll;
    for (int k = 0; k < K; k++) {
        const float r_k = __expf(lp[k] - ll);        // responsibility
        const float w_k = __expf(lw[k]);
        g[k] = (w_k - r_k) * inv_batch;              // d(-ll)/d logit
        for (int d = 0; d < D; d++) {
            const float raw = ym[K + K * D + k * D + d];
            const float ls = fminf(fmaxf(raw, -7.f), 5.f);
            const float iv = __expf(-2.f * ls);
            const float diff = x[d] - ym[K + k * D + d];
            g[K + k * D + d] = -r_k * diff * iv * inv_batch;
            const float gls = -r_k * (diff * diff * iv - 1.f);
            g[K + K * D + k * D + d] = (raw > -7.f && raw < 5.f) ? gls * inv_batch : 0.f;
        }
    }
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ gr, float* __restrict__ m1,
                            float* __restrict__ m2, __nv_bfloat16* __restrict__ p16, int n, float lr, float b1,
                            float b2, float c1, float c2, float eps, float clip_scale)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float g = gr[i] * clip_scale;
    const float a = b1 * m1[i] + (1.f - b1) * g;
    const float b = b2 * m2[i] + (1.f - b2) * g * g;
    m1[i] = a;
    m2[i] = b;
    const float v = p[i] - lr * (a / c1) / (sqrtf(b / c2) + eps);
    p[i] = v;
    if (p16) p16[i] = __float2bfloat16(v);
}

__global__ void sumsq_kernel(const float* __restrict__ g, int n, float* __restrict__ out)
{
    __shared__ float red[256];
    float s = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s += g[i] * g[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(out, red[0]);
}

// ---------------------------------------------------------------------------
// Two-kernel form.  The network is tiny (44 -> 256 -> 256 -> 92), so a launch
// per GEMM was latency: 16-25 us each for a few dozen CTAs, 13 launches per
// gradient.  Here a CTA keeps 16 rows in shared memory through every layer and
// streams the weights (200 KB) from L2 as MMA fragments, 16 bytes per lane:
// every contraction index is stored permuted within its 32 (kpos) so that a
// lane's 16 bytes are its fragments of two m16n8k16 MMAs, the same products in
// the same order as the GEMM per layer.  The weight gradients contract over
// the batch: the row kernel leaves its operands feature-major, so their
// fragments are 16-byte loads too.  One draw (batch 1): three GEMM launches 49 us ->
// 16 us; gradients at batch 256: 210 us of kernels -> 40 us.
// ---------------------------------------------------------------------------
constexpr int kRows = 16;         // batch rows per CTA: one MMA tile
constexpr size_t kRowsMaxSmem = 110 * 1024;
constexpr int kRowThreads = 512;  // 16 warps

__host__ __device__ inline int pad32(int k) { return (k + 31) & ~31; }

// Place of contraction index k within its 32: lane t of an MMA quad holds
// indices 2t, 2t+1, 2t+8, 2t+9 of both halves at places 8t .. 8t+7; kat is the
// inverse.
__host__ __device__ constexpr int kpos(int k)
{
    return (k & ~31) | (((k & 7) >> 1) << 3) | (((k >> 4) & 1) << 2) | (((k >> 3) & 1) << 1) | (k & 1);
}
__host__ __device__ constexpr int kat(int p)
{
    return (p & ~31) | (((p >> 2) & 1) << 4) | (((p >> 1) & 1) << 3) | (((p >> 3) & 3) << 1) | (p & 1);
}
constexpr bool kpos_ok()
{
    for (int k = 0; k < 64; k++)
        if (kat(kpos(k)) != k || (kpos(k) ^ k) >= 32) return false;
    return true;
}
static_assert(kpos_ok(), "kat inverts kpos within each 32");

// Element offsets of the padded BF16 weights.
struct PackedW {
    size_t w1, w2, w3, w2t, w3t, total;
};
__host__ __device__ inline PackedW packed_layout(int in, int H, int out)
{
    PackedW p;
    p.w1 = 0;
    p.w2 = p.w1 + (size_t)H * pad32(in);
    p.w3 = p.w2 + (size_t)H * pad32(H);
    p.w2t = p.w3 + (size_t)out * pad32(H);
    p.w3t = p.w2t + (size_t)H * pad32(H);
    p.total = p.w3t + (size_t)H * pad32(out);
    return p;
}

__global__ void pack_weights_kernel(const float* __restrict__ p32, __nv_bfloat16* __restrict__ w, int in, int H, int out)
{
    const PackedW L = packed_layout(in, H, out);
    const size_t o1 = 0, o2 = (size_t)H * in + H, o3 = o2 + (size_t)H * H + H;  // W1, W2, W3 in p32
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < L.total; e += (size_t)gridDim.x * blockDim.x) {
        float v = 0.f;
        if (e < L.w2) {
            const int K = pad32(in), n = (int)(e / K), k = kat((int)(e % K));
            if (k < in) v = p32[o1 + (size_t)n * in + k];
        } else if (e < L.w3) {
            const int K = pad32(H), n = (int)((e - L.w2) / K), k = kat((int)((e - L.w2) % K));
            if (k < H) v = p32[o2 + (size_t)n * H + k];
        } else if (e < L.w2t) {
            const int K = pad32(H), n = (int)((e - L.w3) / K), k = kat((int)((e - L.w3) % K));
            if (k < H) v = p32[o3 + (size_t)n * H + k];
        } else if (e < L.w3t) {
            const int K = pad32(H), n = (int)((e - L.w2t) / K), k = kat((int)((e - L.w2t) % K));
            if (k < H) v = p32[o2 + (size_t)k * H + n];
        } else {
            const int K = pad32(out), n = (int)((e - L.w3t) / K), k = kat((int)((e - L.w3t) % K));
            if (k < out) v = p32[o3 + (size_t)k * H + n];
        }
        w[e] = __float2bfloat16(v);
    }
}

// epi(n0, acc): acc = X W^T for the CTA's 16 rows and columns n0 .. n0 + 15, in
// the accumulator layout of two N tiles; X in shared memory (row stride ld, a
// multiple of 8 whose eighth is odd: conflict-free 16-byte reads), W in global
// memory (row stride K = pad32), both with kpos order along k.  A warp takes
// 16 columns at a time and loads 256 wide steps of both tiles at once.
template <typename Epi>
__device__ __forceinline__ void rows_layer(const __nv_bfloat16* X, int ld, int K, const __nv_bfloat16* __restrict__ W,
                                           int N, Epi epi)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    for (int n0 = 16 * warp; n0 < N; n0 += 16 * nw) {
        float acc[2][4] = {};
        const uint4* w0 = reinterpret_cast<const uint4*>(W + (size_t)min(n0 + g, N - 1) * K) + t;
        const uint4* w1 = reinterpret_cast<const uint4*>(W + (size_t)min(n0 + 8 + g, N - 1) * K) + t;
        for (int kb = 0; kb < K; kb += 256) {
            uint4 b[8][2];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const bool on = kb + 32 * u < K;
                b[u][0] = on ? __ldg(w0 + (kb >> 3) + 4 * u) : make_uint4(0, 0, 0, 0);
                b[u][1] = on ? __ldg(w1 + (kb >> 3) + 4 * u) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (kb + 32 * u >= K) break;
                const uint4 lo = *reinterpret_cast<const uint4*>(X + g * ld + kb + 32 * u + 8 * t);
                const uint4 hi = *reinterpret_cast<const uint4*>(X + (8 + g) * ld + kb + 32 * u + 8 * t);
                const uint32_t f0[4] = {lo.x, hi.x, lo.y, hi.y}, f1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    mma_bf16(acc[j], f0, b[u][j].x, b[u][j].y);
                    mma_bf16(acc[j], f1, b[u][j].z, b[u][j].w);
                }
            }
        }
        epi(n0, acc);
    }
}

// Shared memory of a row CTA, in bytes; grad: with what the backward pass keeps.
struct RowsLayout {
    int ldx, ldh, ldo;  // row strides (elements)
    size_t x, a1, a2, z1, z2, y, dyf, dy, d2, comp, total;
};
__host__ __device__ inline RowsLayout rows_layout(int in, int H, int out, int D, bool grad)
{
    RowsLayout r;
    r.ldx = pad32(in) + 8;
    r.ldh = pad32(H) + 8;
    r.ldo = pad32(out) + 8;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 15) & ~size_t(15);
        return at;
    };
    r.x = take(sizeof(__nv_bfloat16) * kRows * r.ldx);
    r.a1 = take(sizeof(__nv_bfloat16) * kRows * r.ldh);
    r.a2 = take(sizeof(__nv_bfloat16) * kRows * r.ldh);
    r.z1 = r.z2 = r.y = r.dyf = r.dy = r.d2 = r.comp = 0;
    if (grad) {
        r.z1 = take(sizeof(float) * kRows * H);
        r.z2 = take(sizeof(float) * kRows * H);
        r.y = take(sizeof(float) * kRows * out);
        r.dyf = take(sizeof(float) * kRows * out);
        r.dy = take(sizeof(__nv_bfloat16) * kRows * r.ldo);
        r.d2 = take(sizeof(__nv_bfloat16) * kRows * r.ldh);
        r.comp = take(sizeof(float) * kRows * (17 + D));
    }
    r.total = o;
    return r;
}

struct RowsArgs {
    int B, BP, in, H, out, K, D;
    const float *x, *target;          // [B][in], [B][D] (host-pinned)
    const float* p32;                 // biases
    const __nv_bfloat16* w;
    float* y;                         // [B][out] (host-pinned; forward only)
    float* loss;                      // [B] (host-pinned)
    __nv_bfloat16 *xT, *a1T, *a2T, *dyT, *d2T, *d1T;  // [feature][BP]
    float* colsum;                    // [CTAs][out + 2 H]: sums of dy, d2, d1 over the CTA's rows
};

// Sum over the CTA's 16 rows of one column pair of a layer's epilogue: v[q]
// of lane (g, t) as in the accumulators; every lane ends with columns 2t, 2t+1.
__device__ __forceinline__ float2 rows_colsum(const float (&v)[4])
{
    float2 s = make_float2(v[0] + v[2], v[1] + v[3]);
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, off);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, off);
    }
    return s;
}

// [16 rows][n] of shared memory (kpos order along n) to the CTA's half of a
// 32-row group of [n][BP] in global memory (kpos order along the rows), 8
// bytes of a feature per thread.
__device__ __forceinline__ void rows_transpose(const __nv_bfloat16* S, int ld, int n, __nv_bfloat16* __restrict__ T,
                                               int BP, int row0)
{
    const int base = row0 & ~31, half = (row0 >> 4) & 1;
    for (int e = threadIdx.x; e < n * 4; e += blockDim.x) {
        const int f = e >> 2, t = e & 3, c = kpos(f);
        __align__(8) __nv_bfloat16 v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] = S[(2 * t + (q & 1) + 8 * (q >> 1)) * ld + c];
        *reinterpret_cast<uint2*>(T + (size_t)f * BP + base + 8 * t + 4 * half) = *reinterpret_cast<const uint2*>(v);
    }
}

template <bool GRAD>
__global__ void __launch_bounds__(kRowThreads) mlp_rows_kernel(const RowsArgs A)
{
    extern __shared__ uint4 rows_smem[];
    char* base = reinterpret_cast<char*>(rows_smem);
    const RowsLayout R = rows_layout(A.in, A.H, A.out, A.D, GRAD);
    const PackedW L = packed_layout(A.in, A.H, A.out);
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(base + R.x);
    __nv_bfloat16* a1 = reinterpret_cast<__nv_bfloat16*>(base + R.a1);
    __nv_bfloat16* a2 = reinterpret_cast<__nv_bfloat16*>(base + R.a2);
    float* z1 = reinterpret_cast<float*>(base + R.z1);
    float* z2 = reinterpret_cast<float*>(base + R.z2);
    float* ys = reinterpret_cast<float*>(base + R.y);
    float* dyf = reinterpret_cast<float*>(base + R.dyf);
    __nv_bfloat16* dys = reinterpret_cast<__nv_bfloat16*>(base + R.dy);
    __nv_bfloat16* d2s = reinterpret_cast<__nv_bfloat16*>(base + R.d2);
    float* comp = reinterpret_cast<float*>(base + R.comp);
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int row0 = blockIdx.x * kRows, H = A.H, out = A.out;
    const float* b1 = A.p32 + (size_t)H * A.in;
    const float* b2 = b1 + H + (size_t)H * H;
    const float* b3 = b2 + H + (size_t)out * H;
    // inputs rounded to BF16, zero beyond the batch and the input size; the
    // padding of the activations is zero too (it meets zero weights)
    for (int e = tid; e < kRows * R.ldx; e += kRowThreads) {
        const int r = e / R.ldx, k = e % R.ldx;
        if (k >= pad32(A.in)) continue;
        xs[r * R.ldx + kpos(k)] =
            __float2bfloat16((row0 + r < A.B && k < A.in) ? A.x[(size_t)(row0 + r) * A.in + k] : 0.f);
    }
    float* tgt = comp + kRows * 17;  // [16][D]
    if (GRAD)
        for (int e = tid; e < kRows * A.D; e += kRowThreads)
            tgt[e] = (row0 + e / A.D < A.B) ? A.target[(size_t)row0 * A.D + e] : 0.f;
    const int padH = pad32(H) - H;
    for (int e = tid; e < kRows * padH; e += kRowThreads) {
        const int r = e / padH, k = kpos(H + e % padH);
        a1[r * R.ldh + k] = a2[r * R.ldh + k] = __float2bfloat16(0.f);
        if (GRAD) d2s[r * R.ldh + k] = __float2bfloat16(0.f);
    }
    __syncthreads();
    auto hidden = [&](const float* b, __nv_bfloat16* a, float* z) {
        return [=](int n0, float (&acc)[2][4]) {
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int n = n0 + 8 * j + 2 * t + (q & 1), r = 8 * (q >> 1) + g;
                    if (n >= H) continue;
                    const float zz = acc[j][q] + __ldg(b + n);
                    if (GRAD) z[r * H + n] = zz;
                    a[r * R.ldh + kpos(n)] = __float2bfloat16(silu(zz));
                }
        };
    };
    rows_layer(xs, R.ldx, pad32(A.in), A.w + L.w1, H, hidden(b1, a1, z1));
    __syncthreads();
    rows_layer(a1, R.ldh, pad32(H), A.w + L.w2, H, hidden(b2, a2, z2));
    __syncthreads();
    rows_layer(a2, R.ldh, pad32(H), A.w + L.w3, out, [&](int n0, float (&acc)[2][4]) {
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int n = n0 + 8 * j + 2 * t + (q & 1), r = 8 * (q >> 1) + g;
                if (n >= out) continue;
                const float v = acc[j][q] + __ldg(b3 + n);
                if (GRAD) ys[r * out + n] = v;
                else if (row0 + r < A.B) A.y[(size_t)(row0 + r) * out + n] = v;
            }
    });
    if (!GRAD) return;
    __syncthreads();
    // mixture negative log-likelihood (mixture_nll_kernel's formulas) and its
    // gradient: a lane per component, then the lanes over the outputs
    const int K = A.K, D = A.D, KD = K * D;
    {
        const int r = tid >> 5, k = tid & 31;  // a warp per row
        const float* ym = ys + r * out;
        const bool on = row0 + r < A.B;
        if (on && k < K) {
            float mx = -INFINITY;
            for (int q = 0; q < K; q++) mx = fmaxf(mx, ym[q]);
            float se = 0.f;
            for (int q = 0; q < K; q++) se += __expf(ym[q] - mx);
            const float lw = ym[k] - (mx + __logf(se));
            float sl = -0.91893853320467274f * D;  // -D/2 log(2 pi)
            const float* x = tgt + r * D;
            for (int d = 0; d < D; d++) {
                const float ls = fminf(fmaxf(ym[K + KD + k * D + d], -7.f), 5.f);
                const float rr = (x[d] - ym[K + k * D + d]) * __expf(-ls);
                sl += -0.5f * rr * rr - ls;
            }
            comp[r * 17 + k] = lw;
            comp[r * 17 + 8 + k] = lw + sl;
        }
        __syncwarp();
        float ll = 0.f;
        if (on) {
            float best = -INFINITY, tot = 0.f;
            for (int q = 0; q < K; q++) best = fmaxf(best, comp[r * 17 + 8 + q]);
            for (int q = 0; q < K; q++) tot += __expf(comp[r * 17 + 8 + q] - best);
            ll = best + __logf(tot);
            if (k == 0) A.loss[row0 + r] = -ll;
        }
        const float inv = 1.f / (float)A.B;
        for (int o = k; o < pad32(out); o += 32) {
            float v = 0.f;
            if (on && o < out) {
                const int q = (o < K) ? o : ((o - K) % KD) / D;
                const float rk = __expf(comp[r * 17 + 8 + q] - ll);  // responsibility
                if (o < K) {
                    v = (__expf(comp[r * 17 + q]) - rk) * inv;  // d(-ll)/d logit
                } else {
                    const int d = (o - K) % D;
                    const float raw = ym[K + KD + q * D + d];
                    const float ls = fminf(fmaxf(raw, -7.f), 5.f);
                    const float iv = __expf(-2.f * ls);
                    const float diff = tgt[r * D + d] - ym[K + q * D + d];
                    if (o < K + KD) v = -rk * diff * iv * inv;
                    else if (raw > -7.f && raw < 5.f) v = (-rk * (diff * diff * iv - 1.f)) * inv;
                }
            }
            dys[r * R.ldo + kpos(o)] = __float2bfloat16(v);
            if (o < out) dyf[r * out + o] = v;
        }
    }
    __syncthreads();
    float* sums = A.colsum + (size_t)blockIdx.x * (out + 2 * H);
    for (int o = tid; o < out; o += kRowThreads) {
        float v = 0.f;
        for (int r = 0; r < kRows; r++) v += dyf[r * out + o];
        sums[o] = v;
    }
    rows_transpose(xs, R.ldx, A.in, A.xT, A.BP, row0);
    rows_transpose(a1, R.ldh, H, A.a1T, A.BP, row0);
    rows_transpose(a2, R.ldh, H, A.a2T, A.BP, row0);
    rows_transpose(dys, R.ldo, out, A.dyT, A.BP, row0);
    // backward data path: d = (d_next W) * silu'(z), rounded to BF16 for the
    // next product, its FP32 column sums for the bias gradient
    auto back = [&](__nv_bfloat16* d, const float* z, float* cs) {
        return [=](int n0, float (&acc)[2][4]) {
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int n = n0 + 8 * j + 2 * t;
                float v[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int r = 8 * (q >> 1) + g, nn = n + (q & 1);
                    v[q] = (nn < H) ? acc[j][q] * dsilu(z[r * H + nn]) : 0.f;
                    if (nn < H) d[r * R.ldh + kpos(nn)] = __float2bfloat16(v[q]);
                }
                const float2 cv = rows_colsum(v);
                if (g == 0) {
                    if (n < H) cs[n] = cv.x;
                    if (n + 1 < H) cs[n + 1] = cv.y;
                }
            }
        };
    };
    rows_layer(dys, R.ldo, pad32(out), A.w + L.w3t, H, back(d2s, z2, sums + out));
    __syncthreads();  // d2 complete; a2 has been copied out and its place is free for d1
    rows_transpose(d2s, R.ldh, H, A.d2T, A.BP, row0);
    rows_layer(d2s, R.ldh, pad32(H), A.w + L.w2t, H, back(a2, z1, sums + out + H));
    __syncthreads();
    rows_transpose(a2, R.ldh, H, A.d1T, A.BP, row0);
}

// Weight gradients dW[m][n] = sum_b U[m][b] V[n][b] for the three layers, one
// 32 x 32 tile per CTA (four warps of 16 x 16), both operands feature-major;
// the last CTAs add the bias column sums of the row CTAs in order.
struct WgradArgs {
    int BP, in, H, out, nrows;  // nrows: row CTAs
    const __nv_bfloat16 *xT, *a1T, *a2T, *dyT, *d2T, *d1T;
    const float* colsum;
    float* grad;
};

__global__ void __launch_bounds__(128) mlp_wgrad_kernel(const WgradArgs A)
{
    const int tO = (A.out + 31) / 32, tH = (A.H + 31) / 32, tI = (A.in + 31) / 32;
    const size_t o1 = 0, ob1 = (size_t)A.H * A.in, o2 = ob1 + A.H, ob2 = o2 + (size_t)A.H * A.H, o3 = ob2 + A.H,
                 ob3 = o3 + (size_t)A.out * A.H;
    int job = blockIdx.x;
    const __nv_bfloat16 *U, *V;
    int M, N, tn;
    float* C;
    if (job < tH * tH) {
        U = A.d2T, V = A.a1T, M = A.H, N = A.H, tn = tH, C = A.grad + o2;
    } else if ((job -= tH * tH) < tO * tH) {
        U = A.dyT, V = A.a2T, M = A.out, N = A.H, tn = tH, C = A.grad + o3;
    } else if ((job -= tO * tH) < tH * tI) {
        U = A.d1T, V = A.xT, M = A.H, N = A.in, tn = tI, C = A.grad + o1;
    } else {
        const int f = (job - tH * tI) * 128 + threadIdx.x, F = A.out + 2 * A.H;
        if (f >= F) return;
        float v = 0.f;
        for (int c = 0; c < A.nrows; c++) v += A.colsum[(size_t)c * F + f];
        A.grad[f < A.out ? ob3 + f : (f < A.out + A.H ? ob2 + f - A.out : ob1 + f - A.out - A.H)] = v;
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int m0 = (job / tn) * 32 + 16 * (warp >> 1), n0 = (job % tn) * 32 + 16 * (warp & 1);
    const uint4* u0 = reinterpret_cast<const uint4*>(U + (size_t)min(m0 + g, M - 1) * A.BP) + t;
    const uint4* u1 = reinterpret_cast<const uint4*>(U + (size_t)min(m0 + 8 + g, M - 1) * A.BP) + t;
    const uint4* v0 = reinterpret_cast<const uint4*>(V + (size_t)min(n0 + g, N - 1) * A.BP) + t;
    const uint4* v1 = reinterpret_cast<const uint4*>(V + (size_t)min(n0 + 8 + g, N - 1) * A.BP) + t;
    float acc[2][4] = {};
    for (int kb = 0; kb < A.BP; kb += 128) {
        uint4 a[4][2], b[4][2];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const bool on = kb + 32 * u < A.BP;
            const int at = (kb >> 3) + 4 * u;
            const uint4 zero = make_uint4(0, 0, 0, 0);
            a[u][0] = on ? __ldg(u0 + at) : zero;
            a[u][1] = on ? __ldg(u1 + at) : zero;
            b[u][0] = on ? __ldg(v0 + at) : zero;
            b[u][1] = on ? __ldg(v1 + at) : zero;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t f0[4] = {a[u][0].x, a[u][1].x, a[u][0].y, a[u][1].y};
            const uint32_t f1[4] = {a[u][0].z, a[u][1].z, a[u][0].w, a[u][1].w};
#pragma unroll
            for (int j = 0; j < 2; j++) {
                mma_bf16(acc[j], f0, b[u][j].x, b[u][j].y);
                mma_bf16(acc[j], f1, b[u][j].z, b[u][j].w);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int m = m0 + g + 8 * (q >> 1), n = n0 + 8 * j + 2 * t + (q & 1);
            if (m < M && n < N) C[(size_t)m * N + n] = acc[j][q];
        }
}

}  // namespace

static int mlp_offsets(const messi_mlp* m, size_t off[6])
{
    off[0] = 0;                                    // W1
    off[1] = off[0] + (size_t)m->H * m->in;        // b1
    off[2] = off[1] + m->H;                        // W2
    off[3] = off[2] + (size_t)m->H * m->H;         // b2
    off[4] = off[3] + m->H;                        // W3
    off[5] = off[4] + (size_t)m->out * m->H;       // b3
    return (int)(off[5] + m->out);
}

static int mlp_reserve(messi_ctx* ctx, messi_mlp* m, int batch)
{
    if (batch <= m->cap) return MESSI_OK;
    void** act[] = {(void**)&m->x,  (void**)&m->a1, (void**)&m->a2, (void**)&m->z1,  (void**)&m->z2,  (void**)&m->y,
                    (void**)&m->dy, (void**)&m->d2, (void**)&m->d1, (void**)&m->target, (void**)&m->loss,
                    (void**)&m->xT, (void**)&m->a1T, (void**)&m->a2T, (void**)&m->dyT, (void**)&m->d2T,
                    (void**)&m->d1T, (void**)&m->colsum};
    for (void** p : act) {
        cudaFree(*p);
        *p = nullptr;
    }
    cudaFreeHost(m->stage);
    m->stage = nullptr;
    m->cap = 0;
    const size_t B = (size_t)batch;
    cudaError_t e = cudaSuccess;
    auto al = [&](void** p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMalloc(p, bytes);
    };
    if (m->fused) {
        const size_t BP = (size_t)pad32(batch);
        al((void**)&m->xT, BP * m->in * 2);
        al((void**)&m->a1T, BP * m->H * 2);
        al((void**)&m->a2T, BP * m->H * 2);
        al((void**)&m->dyT, BP * m->out * 2);
        al((void**)&m->d2T, BP * m->H * 2);
        al((void**)&m->d1T, BP * m->H * 2);
        al((void**)&m->colsum, BP / kRows * (m->out + 2 * m->H) * 4);
    } else {
        al((void**)&m->x, B * m->in * 2);
        al((void**)&m->a1, B * m->H * 2);
        al((void**)&m->a2, B * m->H * 2);
        al((void**)&m->z1, B * m->H * 4);
        al((void**)&m->z2, B * m->H * 4);
        al((void**)&m->y, B * m->out * 4);
        al((void**)&m->dy, B * m->out * 4);
        al((void**)&m->d2, B * m->H * 4);
        al((void**)&m->d1, B * m->H * 4);
        al((void**)&m->target, B * m->D * 4);
        al((void**)&m->loss, B * 4 + 64);
    }
    if (e == cudaSuccess) e = cudaMallocHost((void**)&m->stage, B * (m->in + m->out + m->D + 2) * 4 + 64);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp activations");
    m->cap = batch;
    return MESSI_OK;
}

static inline unsigned blocks(long long n) { return (unsigned)((n + 255) / 256); }

// ---- two-kernel form, host side ----
// The packed BF16 weights from the FP32 master copy (queued on the stream).
static int fused_pack(messi_ctx* ctx, messi_mlp* m)
{
    pack_weights_kernel<<<152, 256, 0, ctx->stream>>>(m->p32, m->w16, m->in, m->H, m->out);
    LAUNCH_CHECK(ctx, "pack_weights_kernel");
    return MESSI_OK;
}

// Host staging (pinned, read and written by the kernels): x, target, y, loss.
static float* stage_target(messi_mlp* m) { return m->stage + (size_t)m->cap * m->in; }
static float* stage_y(messi_mlp* m) { return stage_target(m) + (size_t)m->cap * m->D; }
static float* stage_loss(messi_mlp* m) { return stage_y(m) + (size_t)m->cap * m->out; }

static RowsArgs rows_args(messi_mlp* m, int batch)
{
    RowsArgs a{};
    a.B = batch;
    a.BP = pad32(batch);
    a.in = m->in;
    a.H = m->H;
    a.out = m->out;
    a.K = m->K;
    a.D = m->D;
    a.x = m->stage;
    a.target = stage_target(m);
    a.p32 = m->p32;
    a.w = m->w16;
    a.y = stage_y(m);
    a.loss = stage_loss(m);
    a.xT = m->xT;
    a.a1T = m->a1T;
    a.a2T = m->a2T;
    a.dyT = m->dyT;
    a.d2T = m->d2T;
    a.d1T = m->d1T;
    a.colsum = m->colsum;
    return a;
}

static int fused_rows(messi_ctx* ctx, messi_mlp* m, int batch, bool grad)
{
    const size_t smem = rows_layout(m->in, m->H, m->out, m->D, grad).total;
    const void* kernel = grad ? (const void*)mlp_rows_kernel<true> : (const void*)mlp_rows_kernel<false>;
    const cudaError_t e = allow_smem(ctx->device, kernel, smem);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp_rows_kernel attributes");
    // the gradients' operands are whole groups of 32 rows
    const int grid = grad ? pad32(batch) / kRows : (batch + kRows - 1) / kRows;
    if (grad) mlp_rows_kernel<true><<<grid, kRowThreads, smem, ctx->stream>>>(rows_args(m, batch));
    else mlp_rows_kernel<false><<<grid, kRowThreads, smem, ctx->stream>>>(rows_args(m, batch));
    LAUNCH_CHECK(ctx, "mlp_rows_kernel");
    return MESSI_OK;
}

// loss in the staging buffer, gradients in m->grad
static int fused_gradients(messi_ctx* ctx, messi_mlp* m, int batch, const float* x, const float* target)
{
    std::memcpy(m->stage, x, sizeof(float) * batch * m->in);
    std::memcpy(stage_target(m), target, sizeof(float) * batch * m->D);
    int rc;
    if ((rc = fused_rows(ctx, m, batch, true))) return rc;
    WgradArgs w{pad32(batch), m->in, m->H, m->out, pad32(batch) / kRows, m->xT, m->a1T, m->a2T, m->dyT, m->d2T,
                m->d1T, m->colsum, m->grad};
    const int tO = (m->out + 31) / 32, tH = (m->H + 31) / 32, tI = (m->in + 31) / 32;
    const int jobs = tH * tH + tO * tH + tH * tI + (m->out + 2 * m->H + 127) / 128;
    mlp_wgrad_kernel<<<jobs, 128, 0, ctx->stream>>>(w);
    LAUNCH_CHECK(ctx, "mlp_wgrad_kernel");
    return MESSI_OK;
}

// The weights as the network's form reads them, from the FP32 master copy.
static int refresh_weights(messi_ctx* ctx, messi_mlp* m)
{
    if (m->fused) return fused_pack(ctx, m);
    to_bf16_kernel<<<blocks(m->nparam), 256, 0, ctx->stream>>>(m->p32, m->p16, m->nparam);
    LAUNCH_CHECK(ctx, "to_bf16_kernel");
    return MESSI_OK;
}

// forward pass on the batch already in m->x (BF16)
static int mlp_forward_dev(messi_ctx* ctx, messi_mlp* m, int Bn)
{
    size_t off[6];
    mlp_offsets(m, off);
    const __nv_bfloat16* W1 = m->p16 + off[0];
    const __nv_bfloat16* W2 = m->p16 + off[2];
    const __nv_bfloat16* W3 = m->p16 + off[4];
    int rc;
    // z1 = x W1^T + b1 : A = x [B x in], B(k, n) = W1[n][k]
    // (z1, a1) = (x W1^T + b1, silu); the same for layer 2; y = a2 W3^T + b3
    if ((rc = gemm(ctx, Bn, m->H, m->in, m->x, m->in, 1, W1, 1, m->in, m->p32 + off[1], m->z1, m->H, kBiasSilu,
                   nullptr, m->a1)))
        return rc;
    if ((rc = gemm(ctx, Bn, m->H, m->H, m->a1, m->H, 1, W2, 1, m->H, m->p32 + off[3], m->z2, m->H, kBiasSilu,
                   nullptr, m->a2)))
        return rc;
    return gemm(ctx, Bn, m->out, m->H, m->a2, m->H, 1, W3, 1, m->H, m->p32 + off[5], m->y, m->out, kStoreBias);
}

// loss + gradients into m->grad (zeroed first); returns via m->loss
static int mlp_backward_dev(messi_ctx* ctx, messi_mlp* m, int Bn)
{
    size_t off[6];
    mlp_offsets(m, off);
    const __nv_bfloat16* W2 = m->p16 + off[2];
    const __nv_bfloat16* W3 = m->p16 + off[4];
    cudaError_t e = cudaMemsetAsync(m->grad, 0, sizeof(float) * m->nparam, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "grad reset");
    mixture_nll_kernel<<<blocks(Bn), 256, 0, ctx->stream>>>(m->y, m->target, Bn, m->K, m->D, m->loss, m->dy,
                                                            1.f / (float)Bn);
    LAUNCH_CHECK(ctx, "mixture_nll_kernel");
    int rc;
    // layer 3: dW3[o][h] = sum_b dy[b][o] a2[b][h]; db3 = colsum dy; d2 = dy W3
    if ((rc = gemm(ctx, m->out, m->H, Bn, m->dy, 1, m->out, m->a2, m->H, 1, nullptr, m->grad + off[4], m->H,
                   kAccumulate)))
        return rc;
    colsum_kernel<<<blocks(m->out), 256, 0, ctx->stream>>>(m->dy, Bn, m->out, m->grad + off[5]);
    LAUNCH_CHECK(ctx, "colsum_kernel");
    // d2 = (dy W3) * silu'(z2)
    if ((rc = gemm(ctx, Bn, m->H, m->out, m->dy, m->out, 1, W3, m->H, 1, nullptr, m->d2, m->H, kDsilu, m->z2)))
        return rc;
    // layer 2
    if ((rc = gemm(ctx, m->H, m->H, Bn, m->d2, 1, m->H, m->a1, m->H, 1, nullptr, m->grad + off[2], m->H,
                   kAccumulate)))
        return rc;
    colsum_kernel<<<blocks(m->H), 256, 0, ctx->stream>>>(m->d2, Bn, m->H, m->grad + off[3]);
    LAUNCH_CHECK(ctx, "colsum_kernel");
    if ((rc = gemm(ctx, Bn, m->H, m->H, m->d2, m->H, 1, W2, m->H, 1, nullptr, m->d1, m->H, kDsilu, m->z1)))
        return rc;
    // layer 1
    if ((rc = gemm(ctx, m->H, m->in, Bn, m->d1, 1, m->H, m->x, m->in, 1, nullptr, m->grad + off[0], m->in,
                   kAccumulate)))
        return rc;
    colsum_kernel<<<blocks(m->H), 256, 0, ctx->stream>>>(m->d1, Bn, m->H, m->grad + off[1]);
    LAUNCH_CHECK(ctx, "colsum_kernel");
    return MESSI_OK;
}

static int upload_batch(messi_ctx* ctx, messi_mlp* m, int Bn, const float* x, const float* target)
{
    int rc;
    if ((rc = mlp_reserve(ctx, m, Bn))) return rc;
    float* st = m->stage;
    std::memcpy(st, x, sizeof(float) * Bn * m->in);
    cudaError_t e = cudaMemcpyAsync(m->z1, st, sizeof(float) * Bn * m->in, cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp input upload");
    // inputs to BF16 (z1 is free at this point and large enough: H >= in)
    to_bf16_kernel<<<blocks((long long)Bn * m->in), 256, 0, ctx->stream>>>(m->z1, m->x, (long long)Bn * m->in);
    LAUNCH_CHECK(ctx, "to_bf16_kernel");
    if (target) {
        float* sp = st + (size_t)Bn * m->in;
        std::memcpy(sp, target, sizeof(float) * Bn * m->D);
        e = cudaMemcpyAsync(m->target, sp, sizeof(float) * Bn * m->D, cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp target upload");
    }
    return MESSI_OK;
}

}  // namespace messi

using namespace messi;

extern "C" {

int messi_mlp_create(messi_ctx* ctx, int32_t in_dim, int32_t width, int32_t ncomp, int32_t dim, uint64_t seed,
                     messi_mlp** out)
{
    if (!ctx || !out || in_dim < 1 || width < 1 || ncomp < 1 || ncomp > 8 || dim < 1) return MESSI_EINVAL;
    if (width < in_dim) return fail(ctx, MESSI_EINVAL, "mlp: width must be >= input size");
    cudaSetDevice(ctx->device);
    messi_mlp* m = new messi_mlp();
    m->in = in_dim;
    m->H = width;
    m->K = ncomp;
    m->D = dim;
    m->out = ncomp + 2 * ncomp * dim;
    size_t off[6];
    m->nparam = mlp_offsets(m, off);
    // He-style initialisation from a splitmix64 stream (deterministic in seed)
    std::vector<float> p(m->nparam, 0.f);
    uint64_t st = seed ? seed : 0x9E3779B97F4A7C15ull;
    auto next = [&]() {
        st += 0x9E3779B97F4A7C15ull;
        uint64_t z = st;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](size_t o, size_t n, double scale) {
        for (size_t i = 0; i < n; i++) p[o + i] = (float)((2.0 * next() - 1.0) * scale);
    };
    fill(off[0], (size_t)m->H * m->in, std::sqrt(3.0 / m->in));
    fill(off[2], (size_t)m->H * m->H, std::sqrt(3.0 / m->H));
    fill(off[4], (size_t)m->out * m->H, 0.1 * std::sqrt(3.0 / m->H));
    cudaError_t e = cudaMalloc((void**)&m->p32, sizeof(float) * m->nparam);
    if (e == cudaSuccess) e = cudaMalloc((void**)&m->grad, sizeof(float) * (m->nparam + 16));
    if (e == cudaSuccess) e = cudaMalloc((void**)&m->m1, sizeof(float) * m->nparam);
    if (e == cudaSuccess) e = cudaMalloc((void**)&m->m2, sizeof(float) * m->nparam);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(m->p32, p.data(), sizeof(float) * m->nparam, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->m1, 0, sizeof(float) * m->nparam, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->m2, 0, sizeof(float) * m->nparam, ctx->stream);
    if (e != cudaSuccess) {
        messi_mlp_destroy(m);
        return cuda_fail(ctx, e, "mlp parameters");
    }
    // two-kernel form where 16 rows of activations fit half an SM's shared memory
    m->fused = rows_layout(in_dim, width, m->out, dim, true).total <= kRowsMaxSmem;
    if (m->fused)
        e = cudaMalloc((void**)&m->w16, sizeof(__nv_bfloat16) * packed_layout(in_dim, width, m->out).total);
    else
        e = cudaMalloc((void**)&m->p16, sizeof(__nv_bfloat16) * m->nparam);
    if (e != cudaSuccess) {
        messi_mlp_destroy(m);
        return cuda_fail(ctx, e, "mlp weights");
    }
    const int prc = refresh_weights(ctx, m);
    e = cudaStreamSynchronize(ctx->stream);
    if (prc || e != cudaSuccess) {
        messi_mlp_destroy(m);
        return prc ? prc : cuda_fail(ctx, e, "mlp init");
    }
    *out = m;
    return MESSI_OK;
}

int messi_mlp_destroy(messi_mlp* m)
{
    if (!m) return MESSI_EINVAL;
    void* ptrs[] = {m->p32, m->p16, m->grad, m->m1, m->m2, m->x, m->a1, m->a2, m->z1,
                    m->z2,  m->y,   m->dy,   m->d2, m->d1, m->target, m->loss,
                    m->w16, m->xT,  m->a1T,  m->a2T, m->dyT, m->d2T, m->d1T, m->colsum};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (m->stage) cudaFreeHost(m->stage);
    delete m;
    return MESSI_OK;
}

int messi_mlp_nparams(messi_mlp* m, int32_t* n)
{
    if (!m || !n) return MESSI_EINVAL;
    *n = m->nparam;
    return MESSI_OK;
}

int messi_mlp_get_params(messi_ctx* ctx, messi_mlp* m, float* host)
{
    if (!ctx || !m || !host) return MESSI_EINVAL;
    cudaSetDevice(ctx->device);
    cudaError_t e = cudaMemcpy(host, m->p32, sizeof(float) * m->nparam, cudaMemcpyDeviceToHost);
    return (e == cudaSuccess) ? MESSI_OK : cuda_fail(ctx, e, "mlp get params");
}

int messi_mlp_set_params(messi_ctx* ctx, messi_mlp* m, const float* host)
{
    if (!ctx || !m || !host) return MESSI_EINVAL;
    cudaSetDevice(ctx->device);
    cudaError_t e = cudaMemcpyAsync(m->p32, host, sizeof(float) * m->nparam, cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp set params");
    const int rc = refresh_weights(ctx, m);
    e = cudaStreamSynchronize(ctx->stream);
    return rc ? rc : ((e == cudaSuccess) ? MESSI_OK : cuda_fail(ctx, e, "mlp set params"));
}

int messi_mlp_forward(messi_ctx* ctx, messi_mlp* m, int32_t batch, const float* x, float* y)
{
    if (!ctx || !m || batch < 1 || !x || !y) return MESSI_EINVAL;
    ctx->launches = 0;
    cudaSetDevice(ctx->device);
    int rc;
    if (m->fused) {
        if ((rc = mlp_reserve(ctx, m, batch))) return rc;
        std::memcpy(m->stage, x, sizeof(float) * batch * m->in);
        if ((rc = fused_rows(ctx, m, batch, false))) return rc;
        const cudaError_t fe = cudaStreamSynchronize(ctx->stream);
        if (fe != cudaSuccess) return cuda_fail(ctx, fe, "mlp forward");
        std::memcpy(y, stage_y(m), sizeof(float) * batch * m->out);
        return MESSI_OK;
    }
    if ((rc = upload_batch(ctx, m, batch, x, nullptr))) return rc;
    if ((rc = mlp_forward_dev(ctx, m, batch))) return rc;
    cudaError_t e = cudaMemcpyAsync(y, m->y, sizeof(float) * batch * m->out, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    return (e == cudaSuccess) ? MESSI_OK : cuda_fail(ctx, e, "mlp forward");
}

int messi_mlp_gradients(messi_ctx* ctx, messi_mlp* m, int32_t batch, const float* x, const float* target,
                        float* loss, float* grads)
{
    if (!ctx || !m || batch < 1 || !x || !target) return MESSI_EINVAL;
    ctx->launches = 0;
    cudaSetDevice(ctx->device);
    int rc;
    std::vector<float> l(batch);
    cudaError_t e = cudaSuccess;
    if (m->fused) {
        if ((rc = mlp_reserve(ctx, m, batch))) return rc;
        if ((rc = fused_gradients(ctx, m, batch, x, target))) return rc;
    } else {
        if ((rc = upload_batch(ctx, m, batch, x, target))) return rc;
        if ((rc = mlp_forward_dev(ctx, m, batch))) return rc;
        if ((rc = mlp_backward_dev(ctx, m, batch))) return rc;
        e = cudaMemcpyAsync(l.data(), m->loss, sizeof(float) * batch, cudaMemcpyDeviceToHost, ctx->stream);
    }
    if (e == cudaSuccess && grads)
        e = cudaMemcpyAsync(grads, m->grad, sizeof(float) * m->nparam, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp gradients");
    if (m->fused) std::memcpy(l.data(), stage_loss(m), sizeof(float) * batch);
    if (loss) {
        double s = 0.0;
        for (float v : l) s += v;
        *loss = (float)(s / batch);
    }
    return MESSI_OK;
}

int messi_mlp_train_step(messi_ctx* ctx, messi_mlp* m, int32_t batch, const float* x, const float* target, float lr,
                         float max_grad_norm, float* loss)
{
    int rc = messi_mlp_gradients(ctx, m, batch, x, target, loss, nullptr);
    if (rc) return rc;
    float* d_norm = m->grad + m->nparam;  // spare slot
    cudaMemsetAsync(d_norm, 0, sizeof(float), ctx->stream);
    sumsq_kernel<<<64, 256, 0, ctx->stream>>>(m->grad, m->nparam, d_norm);
    LAUNCH_CHECK(ctx, "sumsq_kernel");
    float h = 0.f;
    cudaError_t e = cudaMemcpyAsync(&h, d_norm, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "grad norm");
    const float gn = std::sqrt(h);
    const float clip = (max_grad_norm > 0.f && gn > max_grad_norm) ? max_grad_norm / gn : 1.f;
    m->steps++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)m->steps), c2 = 1.f - std::pow(b2, (float)m->steps);
    adam_kernel<<<blocks(m->nparam), 256, 0, ctx->stream>>>(m->p32, m->grad, m->m1, m->m2, m->p16, m->nparam, lr, b1,
                                                            b2, c1, c2, 1e-8f, clip);
    LAUNCH_CHECK(ctx, "adam_kernel");
    if (m->fused && (rc = fused_pack(ctx, m))) return rc;
    e = cudaStreamSynchronize(ctx->stream);
    return (e == cudaSuccess) ? MESSI_OK : cuda_fail(ctx, e, "adam");
}

}  // extern "C"
