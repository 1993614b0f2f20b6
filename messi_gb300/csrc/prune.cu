// prune.cu -- site-pair pruning (HP1) and unpaired column likelihoods on the GPU.
//
// Replaces the kernels of src/cuda/felsenstein.cu used by
// src/FelsensteinCUDA.jl:214-516 (felsensteinleaves16 :117-133,
// felsensteinhelper16 :153-200, sumfinal :428-442, storearr/logsumexparr
// :135-151) with:
//   * build_P16_kernel: P = exp(Qt) per (category, branch) in FP64 from the
//     host eigensystem, stored as FP32 rows (row = parent state);
//   * message rows: what a node passes to its parent is its partial
//     likelihood vector already multiplied by its own branch's matrix,
//     m_v = P_v x_v, so every node update is x_v = m_left * m_right
//     (elementwise) followed by ONE mat-vec, P_v x_v, done once per unique
//     row at v instead of once per parent pair that reads the row (the
//     reference applies both child matrices inside every parent update,
//     felsenstein.cu:170-190); the root needs no mat-vec, only pi . x;
//   * leaf_msg_kernel: the messages of the leaves (P_leaf x indicator rows)
//     per category pass;
//   * prune_path_kernel: one launch per level of tree segments and category
//     pass; a warp owns 32 unique pairs and walks them through a segment's
//     nodes with the running message in registers, gathering one child row
//     per node and doing the mat-vec on the tensor cores (3xTF32 mma.sync,
//     operands split into hi/lo).  Messages are rescaled by an exact power of
//     two (exponent kept as an int), which computes the same likelihood as
//     the reference's divide-by-max (felsenstein.cu:193-198); the root folds
//     sumfinal and the category log-sum-exp into the same pass (FP64
//     log-likelihood reduction);
//   * prune_tc_kernel: the interior update of single-node segments as
//     tcgen05.mma (A in tensor memory, P in shared memory, accumulators in
//     tensor memory), the same bits as prune_path_kernel; chosen only on
//     request (launch shape 3).
// unpaired_site_kernel + unpaired_mix_kernel restate
// computeunpairedlikelihoodscat (src/FARCE.jl:742-773) in FP64 with the CPU
// rescaling rule.
#include <algorithm>
#include <cmath>

#include "internal.h"

namespace messi {

// P[c][v][a][d] in FP32 (row = parent state), from the FP64 eigensystem:
// P = D^-1/2 U exp(W t) U^T D^1/2.  One CTA per category and run of
// kP16Nodes nodes, a thread per entry: the CTA forms the exponentials of all
// its nodes at once, stages the category's U and the ratios sqrt(pi_d) /
// sqrt(pi_a) once per model group and, per node, W[a][k] = U[a][k] exp(w_k t),
// so an entry is 16 FP64 multiply-adds; U exp(W t) U^T is symmetric, so a thread
// forms one of its 136 entries and scales it both ways.  Bound by the FP64 pipe.
// 36 categories of 127 nodes, of 31 nodes: with 32 nodes per CTA and a node's
// exponentials on its critical path 73 and 69 us (36 CTAs), with all 256 entries
// 53 and 17 us, now 41 and 15; 1,584 nodes 577 -> 448 us.
constexpr int kP16Nodes = 8;
constexpr int kP16Entries = 136;  // i <= j

// x as TF32 hi + lo: hi = x rounded to TF32 (half a TF32 ulp added to the
// magnitude bits, then truncated: round to nearest, ties away), lo = x - hi,
// exact in FP32.
__device__ __forceinline__ float tf32_hi(float x)
{
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
}

// Float offset of entry (a, d) in a stored matrix: the B fragments of the
// pruning kernel, whose lane 4g + t loads P[4(g/2) + 2nt + g%2][4t..4t+3] for
// N tile nt as one of 32 consecutive 16-byte words; the lo part 256 floats on.
__host__ __device__ constexpr int p16_at(int a, int d)
{
    return ((a >> 1) & 1) * 128 + ((((a >> 2) << 1) | (a & 1)) * 4 + (d >> 2)) * 4 + (d & 3);
}

__global__ void __launch_bounds__(256) build_P16_kernel(const double* __restrict__ eig, const double* __restrict__ bl,
                                                       const int* __restrict__ nodegrp, int numnodes, int C,
                                                       float* __restrict__ P)
{
    // one grid dimension: a batch may have more runs of nodes than the second one takes
    const int c = (int)(blockIdx.x % (unsigned)C), t = threadIdx.x;
    const int a = t >> 4, d = t & 15;
    const int v0 = (int)(blockIdx.x / (unsigned)C) * kP16Nodes, v1 = min(numnodes, v0 + kP16Nodes);
    __shared__ double U[256], W[2][256], R[256], ex[kP16Nodes][16];
    auto group = [&](int v) { return nodegrp ? nodegrp[v] : (v == 0 ? -1 : 0); };  // the same in every thread
    if (t < 16 * kP16Nodes && v0 + a < v1) {
        const int grp = group(v0 + a);
        if (grp >= 0) ex[a][d] = exp(eig[((size_t)grp * C + c) * kEigStride + d] * bl[v0 + a]);
    }
    // this thread's entry (i, j), i <= j, of a node: the t-th, row by row
    int i = 0, j = t;
    while (i < 16 && j >= 16 - i) j -= 16 - i++;
    j += i;
    int cur = -1;
    for (int v = v0; v < v1; v++) {
        const int grp = group(v), buf = v & 1;
        const double tl = bl[v];
        if (grp >= 0 && grp != cur) {
            const double* e = eig + ((size_t)grp * C + c) * kEigStride;
            __syncthreads();  // the previous group's U is no longer read
            U[t] = e[16 + t];
            R[t] = e[16 + 256 + d] / e[16 + 256 + a];
            cur = grp;
            __syncthreads();
        }
        // W[a][k], k = d; the other buffer may still be read for the node before
        if (grp >= 0) W[buf][t] = U[t] * ex[v - v0][d];
        __syncthreads();
        if (t >= kP16Entries) continue;
        float up, low;  // (i, j) and (j, i)
        if (grp < 0) {
            up = low = 0.f;  // a root has no branch (gettransitionmatriceslist, src/FARCE.jl:416)
        } else if (tl == 0.0) {
            up = low = (i == j) ? 1.f : 0.f;
        } else {
            double acc = 0.0;
#pragma unroll
            for (int k = 0; k < 16; k++) acc += W[buf][i * 16 + k] * U[j * 16 + k];
            auto entry = [&](double x) { return (x <= 0.0) ? 0.f : (float)x; };  // absmat clamp (1e-50 rounds to 0 in FP32)
            up = entry(acc * R[i * 16 + j]);
            low = entry(acc * R[j * 16 + i]);
        }
        float* p = P + ((size_t)c * numnodes + v) * kP16Floats;
        auto put = [&](int at, float x) {
            const float hi = tf32_hi(x);
            p[at] = hi;
            p[at + 256] = x - hi;
        };
        put(p16_at(i, j), up);
        if (i != j) put(p16_at(j, i), low);
    }
}

__global__ void build_P4_kernel(const double* __restrict__ eig4, const double* __restrict__ bl,
                                const int* __restrict__ nodegrp, int numnodes, int nsite, double* __restrict__ P4)
{
    const int v = blockIdx.x, s = blockIdx.y, t = threadIdx.x;  // 16 threads
    const int grp = nodegrp ? nodegrp[v] : (v == 0 ? -1 : 0);
    const double* e = eig4 + ((size_t)max(grp, 0) * nsite + s) * kEig4Stride;
    const double tl = bl[v];
    const int a = t >> 2, d = t & 3;
    double out;
    if (grp < 0) {
        out = 0.0;
    } else if (tl == 0.0) {
        out = (a == d) ? 1.0 : 0.0;
    } else {
        double acc = 0.0;
        for (int k = 0; k < 4; k++) acc += e[4 + a * 4 + k] * exp(e[k] * tl) * e[4 + d * 4 + k];
        acc *= e[20 + d] / e[20 + a];
        out = (acc <= 0.0) ? 1e-50 : acc;
    }
    P4[((size_t)s * numnodes + v) * 16 + t] = out;
}

int launch_build_P16(messi_ctx* ctx, const double* d_eig, const double* d_bl, const int* d_nodegrp, int numnodes,
                     int C, float* d_P)
{
    const unsigned runs = (unsigned)(numnodes + kP16Nodes - 1) / kP16Nodes;
    build_P16_kernel<<<(unsigned)C * runs, 256, 0, ctx->stream>>>(d_eig, d_bl, d_nodegrp, numnodes, C, d_P);
    LAUNCH_CHECK(ctx, "build_P16_kernel");
    return MESSI_OK;
}

int launch_build_P4(messi_ctx* ctx, const double* d_eig4, const double* d_bl, const int* d_nodegrp, int numnodes,
                    int nsite, double* d_P4)
{
    build_P4_kernel<<<dim3(numnodes, nsite), 16, 0, ctx->stream>>>(d_eig4, d_bl, d_nodegrp, numnodes, nsite, d_P4);
    LAUNCH_CHECK(ctx, "build_P4_kernel");
    return MESSI_OK;
}

__device__ __forceinline__ double lse_d(double a, double b)
{
    if (b == -INFINITY) return a;
    if (a == -INFINITY) return b;
    return (a < b) ? b + log1p(exp(a - b)) : a + log1p(exp(b - a));
}

// lse_d with the correction log(1 + e^-|a-b|) (in [0, log 2]) formed in FP32
// from the FP64 difference: absolute error ~1e-7 on a sum of log-likelihoods
// of magnitude 10-1000, against an FP64 exp and log1p per call (the band
// preparation of a 256-alignment batch calls it for 9.3e7 cells).
__device__ __forceinline__ double lse_d_fast(double a, double b)
{
    if (b == -INFINITY) return a;
    if (a == -INFINITY) return b;
    const double mx = fmax(a, b);
    return mx + (double)log1pf(expf((float)(fmin(a, b) - mx)));
}

// ---------------------------------------------------------------------------
// Leaf messages: out[cc][r][a] = sum_d P[c0+cc][node(r)][a][d] over the states
// d of row r's mask (16 threads per row, FP64 accumulation, one FP32 rounding).
// An observed base pair is one state and needs no FP64 at all; those units
// issue a warp only every 64 cycles per SM quarter, and the 0/1 rows' full
// products kept them busy for 86 us (1,600 rows of 36 categories), now 16.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) leaf_msg_kernel(const int2* __restrict__ rows, long long R,
                                                       const float* __restrict__ P, int numnodes, int c0,
                                                       float* __restrict__ out)
{
    const long long r = (long long)blockIdx.x * 16 + (threadIdx.x >> 4);
    const int a = threadIdx.x & 15, cc = blockIdx.y;
    if (r >= R) return;
    const int2 row = __ldg(rows + r);  // leaf node, mask of its states
    const float* p = P + ((size_t)(c0 + cc) * numnodes + row.x) * kP16Floats;
    auto entry = [&](int d) { return __ldg(p + p16_at(a, d)) + __ldg(p + p16_at(a, d) + 256); };
    const int first = __ffs(row.y) - 1;
    float v = entry(first);
    if (row.y & (row.y - 1)) {  // ambiguous: ascending, as the full product adds them
        double s = (double)v;
        for (int m = row.y & (row.y - 1); m; m &= m - 1) s += (double)entry(__ffs(m) - 1);
        v = (float)s;
    }
    out[((size_t)cc * R + r) * 16 + a] = v;
}

int launch_leaf_messages(messi_ctx* ctx, const int2* d_rows, int64_t R, const float* d_P, int numnodes, int c0, int nc,
                         float* d_out)
{
    if (R <= 0 || nc <= 0) return MESSI_OK;
    leaf_msg_kernel<<<dim3((unsigned)((R + 15) / 16), nc), 256, 0, ctx->stream>>>(d_rows, R, d_P, numnodes, c0, d_out);
    LAUNCH_CHECK(ctx, "leaf_msg_kernel");
    return MESSI_OK;
}

// ---------------------------------------------------------------------------
// Tensor-core node update (3xTF32 mma.sync): for 32 pairs of one node and one
// category x = m_left * m_right and, below the root, the product
// [32 pairs x 16] x [16 x 16]^T with P of the node's own branch, as m16n8k8
// TF32 MMAs with both operands split hi + lo (hi*hi + hi*lo + lo*hi:
// FP32-level accuracy; all operands are non-negative, so there is no
// cancellation).
// Rounding.  The tensor core rounds each MMA's FP32 result toward zero
// (measured on GB300: 99.9% of outputs equal the truncation of the exact
// sum, mean error -0.44 ulp), so a chain of MMAs loses about half an ulp per
// result, always downwards; over the 62 mat-vecs of a 64-leaf tree that
// shifted every pair log-likelihood by about -1.2e-6.  Each of the two
// k-steps therefore accumulates into its own registers (small cross terms
// first, so their truncation is negligible), the two halves are added in
// FP32 (round to nearest), and half an ulp of the sum is added back, again
// rounded to nearest: a tie, which rounds up or down on the last mantissa
// bit, so the truncation bias of the two halves is returned on average.
// The contraction index d is permuted so that lane (g, t) owns
// d = 4t..4t+3: its A fragment for pair row r is one 16-byte piece of each
// message, its B fragment 16 bytes of a row of P (p16_at).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float comp4(const float4& v, int k)
{
    return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w));
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The first MMA of a chain: the accumulator starts from zero (no registers to clear).
__device__ __forceinline__ void mma_tf32_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// A operand split: hi, and lo fed without conversion (the tensor core reads
// the top 19 bits of lo, an error below 2^-21 |x| of either sign, as lo is
// centred on zero).
__device__ __forceinline__ void split_a(float x, uint32_t& hi, uint32_t& lo)
{
    hi = __float_as_uint(tf32_hi(x));
    lo = __float_as_uint(x - __uint_as_float(hi));
}

// v + half an ulp of v, rounded to nearest (ties to even): v or v + ulp,
// each for half of the mantissas.  v >= 0.  The exponent bits alone are the
// power of two 2^e of v, so half an ulp is 2^e * 2^-24 (exact) and one FMA adds it.
__device__ __forceinline__ float add_half_ulp(float v)
{
    return fmaf(__uint_as_float(__float_as_uint(v) & 0x7f800000u), 5.9604644775390625e-8f, v);
}

// D0[mt][nt] = X x P^T over states k-step 0 (d = 4t, 4t+1), D1 over k-step 1
// (d = 4t+2, 4t+3), each as lo*hi + hi*lo + hi*hi, for rows g + 8k (k = 0..3).
__device__ __forceinline__ void msg_mma(const float4 (&X)[4], const float4 (&Bh)[2], const float4 (&Bl)[2],
                                        float (&D0)[2][2][4], float (&D1)[2][2][4])
{
    // The three products of an accumulator depend on one another: the four
    // accumulators of a row half take turns, so that a product does not wait
    // for the one before it.
#pragma unroll
    for (int mt = 0; mt < 2; mt++) {
        uint32_t ah[2][4], al[2][4];
#pragma unroll
        for (int ks = 0; ks < 2; ks++) {
            const float av[4] = {comp4(X[2 * mt], 2 * ks), comp4(X[2 * mt + 1], 2 * ks), comp4(X[2 * mt], 2 * ks + 1),
                                 comp4(X[2 * mt + 1], 2 * ks + 1)};
#pragma unroll
            for (int i = 0; i < 4; i++) split_a(av[i], ah[ks][i], al[ks][i]);
        }
#pragma unroll
        for (int term = 0; term < 3; term++)
#pragma unroll
            for (int ks = 0; ks < 2; ks++)
#pragma unroll
                for (int nt = 0; nt < 2; nt++) {
                    float (&D)[4] = ks ? D1[mt][nt] : D0[mt][nt];
                    const float4& B = (term == 1) ? Bl[nt] : Bh[nt];
                    const uint32_t b0 = __float_as_uint(comp4(B, 2 * ks)), b1 = __float_as_uint(comp4(B, 2 * ks + 1));
                    if (term == 0) mma_tf32_zero(D, al[ks], b0, b1);
                    else mma_tf32(D, ah[ks], b0, b1);
                }
    }
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }

template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Exact power-of-two rescale of a row max m > 0: m * 2^-ex in [0.5, 1), as two
// factors: a denormal m needs more than the largest power of two.
__device__ __forceinline__ void pow2_scale(float m, int& ex, float& pre, float& sc)
{
    const bool denormal = m > 0.f && m < 0x1p-126f;
    pre = denormal ? 0x1p126f : 1.f;
    m *= pre;
    const unsigned bits = __float_as_uint(m);
    const int E = (int)((bits >> 23) & 0xffu);
    if (E >= 1 && E <= 252) {  // normal, and 2^-ex representable
        ex = E - 126;
        sc = __uint_as_float((unsigned)(127 - ex) << 23);
    } else if (m > 0.f) {
        frexpf(m, &ex);
        sc = ldexpf(1.f, -ex);
    } else {
        ex = 0;
        sc = 1.f;
    }
    if (denormal) ex -= 126;
}

// ---------------------------------------------------------------------------
// Segment programs.  A warp owns 32 unique pairs (NP = 1, or 64: NP = 2) of a
// segment's top node and, category by category, runs the segment's program on
// them: the running message M stays in registers from node to node, so of a
// node's two child rows only the one that comes from a table below is read
// and nothing is written but the segment's last message.  (One launch per tree
// level, every node's rows written and gathered again, moved 212 bytes per
// update and was bound by the L1 data pipe, 71% of its wavefronts.)
// Each step gathers one row per pair: the four lanes (g, t) of a pair read
// 16 bytes each, straight to registers.  The gathers are a stream of their
// own: a row is asked for as soon as the one before it is consumed, so that it
// arrives under the mat-vec (without that, 24 warps per SM instead of 20: 15%
// slower), and so is the next matrix, as soon as the MMAs have read this
// one's, both across the end of a category (matrices asked for where they are
// used: lower levels 15-20% slower).  The columns of P are assigned to the MMA's N index so that lane (g, t) ends with
// states 4t..4t+3 of its pairs, which is the A layout of the next product:
// column g of tile nt is state 4(g/2) + 2nt + g%2.
// Measured (GB300, 64 x 1,000 columns, span 500, 36 categories): 2.96e8
// distinct updates in 7.5 ms before; 3.6e8 (some recomputed) in 4.9 ms now,
// DRAM traffic 35 GB -> ~7 GB.  What bounds it: about 245 instructions per 32
// updates at half of the issue slots, the tensor pipe 41% busy (24 MMAs of 8.5
// cycles a step), with the 20 warps per SM the registers allow: 16 took 13%
// more per warp and step, a third of the MMAs 20% less, constant rows or
// matrices 3% less each.
// The CTA's warps are pg pair groups x cs category splits: with few pairs the
// warps of one pair group take every cs-th category each (a level of 50
// tiles of 128 pairs with all 36 categories in turn took 45 us).
// Where a pair group's twelve splits still leave the chip idle, gridDim.y CTAs
// share its categories (the 150 pairs of a structure over 64 sequences, 5 pair
// groups: root level 156 -> 35 us with three CTAs each, and 13 us for the mixtures).
// ROOT: 0 = interior segment, 1 = the tree's root with the category mixture
// kept in registers (cs = 1), 2 = the root with the categories' values
// collected in shared memory (in `shared_values` where CTAs share a group) and
// mixed afterwards in category order by one warp, so that the sum has the same
// bits.
// ---------------------------------------------------------------------------
struct Mixture {
    double m = -INFINITY;
    float s = 0.f;
    __device__ __forceinline__ void add(double tt)
    {
        if (tt > m) {
            s = s * __expf((float)(m - tt)) + 1.f;
            m = tt;
        } else if (tt != -INFINITY) {
            s += __expf((float)(tt - m));
        }
    }
    __device__ __forceinline__ double value() const { return (m == -INFINITY) ? -INFINITY : m + log((double)s); }
};

// Mixes the categories' values v[32 cc] of pair u in category order.
__device__ __forceinline__ void mix_values(const SegDev& sg, const double* v, int u, int c0, int nc,
                                           const int* __restrict__ lam, int per_lambda)
{
    Mixture mix;
    for (int c1 = 0; c1 < nc; c1 += 12) {
        double x[12];  // twelve loads in flight (one after another: 18 us for 36 categories)
#pragma unroll
        for (int k = 0; k < 12; k++) x[k] = v[(size_t)min(c1 + k, nc - 1) * 32];
#pragma unroll
        for (int k = 0; k < 12; k++)
            if (c1 + k < nc) mix.add(x[k]);
    }
    const double res = mix.value();
    sg.mix[u] = (c0 == 0) ? res : lse_d(sg.mix[u], res);
    if (!per_lambda) return;
    for (int q = 0; q < kMaxLambda; q++) {
        Mixture ml;
        for (int cc = 0; cc < nc; cc++)
            if (__ldg(lam + c0 + cc) == q) ml.add(v[(size_t)cc * 32]);
        const double rq = ml.value();
        double* dst = sg.mixlam + (size_t)q * sg.n + u;
        *dst = (c0 == 0) ? rq : lse_d(*dst, rq);
    }
}

// Lane t's own one of four values (pair g + 8t).
__device__ __forceinline__ int own4(const int4& v, int t) { return t == 0 ? v.x : (t == 1 ? v.y : (t == 2 ? v.z : v.w)); }

// A read-only integer load where `pred`, else 0, as one predicated instruction.
__device__ __forceinline__ int ldg_int_if(const int* p, bool pred)
{
    int v;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.b32 %0, 0;\n\t@q ld.global.nc.b32 %0, [%1];\n\t}"
        : "=r"(v)
        : "l"(__cvta_generic_to_global(p)), "r"((int)pred));
    return v;
}

// Reduces v[k] over the four lanes t of a pair; lane t keeps pair k = t: two
// exchanges of halves instead of a butterfly per pair (three shuffles, not eight).
template <typename Op>
__device__ __forceinline__ float quad_reduce(const float (&v)[4], int t, Op op)
{
    const bool o1 = t & 1, o2 = t & 2;
    const float a = op(o1 ? v[1] : v[0], __shfl_xor_sync(0xffffffffu, o1 ? v[0] : v[1], 1));
    const float b = op(o1 ? v[3] : v[2], __shfl_xor_sync(0xffffffffu, o1 ? v[2] : v[3], 1));
    return op(o2 ? b : a, __shfl_xor_sync(0xffffffffu, o2 ? a : b, 2));
}

__device__ __forceinline__ float4 mul4(const float4& a, const float4& b)
{
    return make_float4(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z), __fmul_rn(a.w, b.w));
}
__device__ __forceinline__ float max4(const float4& v) { return fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)); }

template <int ROOT, int NP, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) prune_path_kernel(
    const SegDev* __restrict__ segs, const int2* __restrict__ tiles, const float* __restrict__ P, int numnodes,
    int c0, int nc, int C, const float* __restrict__ pi16, const double* __restrict__ logw,
    const int* __restrict__ lam, int per_lambda, int cs, int max_steps, int max_nb, int max_depth,
    double* __restrict__ shared_values)
{
    extern __shared__ float4 smem_raw[];
    const int2 tile = tiles[blockIdx.x];
    const SegDev& sg = segs[tile.x];
    const int n = sg.n, ns = sg.nsteps, nb = sg.nb;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int pgs = (int)(blockDim.x >> 5) / cs, pg = warp % pgs;
    const int split = warp / pgs + cs * (int)blockIdx.y, stride = cs * (int)gridDim.y;  // this warp's categories
    const int base = tile.y + 32 * NP * pg;  // first pair of this warp
    const bool active = base < n;
    // shared memory: gathers (slot nb repeats slot 0: the stream's last look
    // ahead), mat-vec steps, gather indices per pair group, set-aside messages
    // per warp, collected values
    int4* gathers = reinterpret_cast<int4*>(smem_raw);
    int2* ops = reinterpret_cast<int2*>(gathers + max_nb + 1);
    float4* rest = smem_raw + (max_nb + 1) + (max_steps + 1) / 2;
    int4* sidx = reinterpret_cast<int4*>(rest) + pg * (max_nb + 1) * 8 * NP;
    rest += pgs * (max_nb + 1) * 8 * NP;
    float4* stack = rest + warp * max_depth * 128 * NP + lane;
    double* collected = (ROOT == 2 && gridDim.y > 1)
                            ? shared_values + (size_t)blockIdx.x * pgs * NP * nc * 32
                            : reinterpret_cast<double*>(rest + (int)(blockDim.x >> 5) * max_depth * 128 * NP);
    const int nmul = ROOT ? ns - 1 : ns;  // the root's step has no mat-vec
    for (int i = threadIdx.x; i < ns; i += blockDim.x) {
        const int4* steps = reinterpret_cast<const int4*>(sg.steps);
        const int4 st = __ldg(steps + i);
        // the next mat-vec's matrix; after the last, the next category's first
        unsigned ahead;
        if (i + 1 < nmul) {
            int4 nx = __ldg(steps + i + 1);
            if (nx.w & kStepInit) nx = __ldg(steps + i + 2);
            ahead = (unsigned)nx.z;
        } else {
            ahead = (unsigned)__ldg(steps + 1).z + (unsigned)(stride * numnodes);
        }
        ops[i] = make_int2((int)ahead, st.w);
        if (st.w & kStepGather) {
            const int slot = st.w >> kStepSlotShift;
            gathers[slot] = make_int4(st.x, st.y, st.w & kStepLeaf, -1);
            if (slot == 0) gathers[nb] = make_int4(st.x + stride * st.y, st.y, st.w & kStepLeaf, st.x + (nc - 1) * st.y);
        }
    }
    if (active) {
#pragma unroll
        for (int h = 0; h < NP; h++) {  // (past the last pair the last tile again)
            const int4* src = reinterpret_cast<const int4*>(sg.idx) + (size_t)min((base >> 5) + h, (n - 1) >> 5) * nb * 8;
            int4* dst = sidx + h * (max_nb + 1) * 8;
            for (int i = warp / pgs * 32 + lane; i < (nb + 1) * 8; i += 32 * cs) dst[i] = __ldg(src + (i < nb * 8 ? i : i - nb * 8));
        }
    }
    __syncthreads();
    const int myu = base + g + 8 * t;  // pair whose scalars this lane keeps (and myu + 32)
    Mixture mix[NP];
    if (active && split < nc) {
        float4 M[NP][4], R[NP][4];
        int e[NP], er[NP];
        const float4* rows = reinterpret_cast<const float4*>(sg.rows) + t;
        const int* exps = sg.exps;
        const int4* gp = gathers;
        const int* si = reinterpret_cast<const int*>(sidx);
        int cc = split;
        // The next gather of the stream: states 4t..4t+3 of pairs g + 8k, and
        // the exponent of the lane's own pair.
        auto next = [&]() {
            const int4 gd = *gp++;
            const unsigned row = min((unsigned)gd.x + (unsigned)cc * (unsigned)gd.y, (unsigned)gd.w);
            const float4* f = rows + (size_t)row * 4;
#pragma unroll
            for (int h = 0; h < NP; h++) {
                const int* sh = si + h * (max_nb + 1) * 32;
                const int4 id = *reinterpret_cast<const int4*>(sh + 4 * g);
                R[h][0] = __ldg(f + (size_t)(unsigned)id.x * 4);
                R[h][1] = __ldg(f + (size_t)(unsigned)id.y * 4);
                R[h][2] = __ldg(f + (size_t)(unsigned)id.z * 4);
                R[h][3] = __ldg(f + (size_t)(unsigned)id.w * 4);
                er[h] = ldg_int_if(exps + row + (unsigned)sh[lane], gd.z == 0);
            }
            si += 32;
        };
        auto pop = [&](float4*& top) {
            top -= 128 * NP;
#pragma unroll
            for (int h = 0; h < NP; h++)
#pragma unroll
                for (int k = 0; k < 4; k++) M[h][k] = mul4(M[h][k], top[128 * h + 32 * k]);
        };
        auto product = [&]() {  // x = M * R, then the next rows are asked for
#pragma unroll
            for (int h = 0; h < NP; h++) {
#pragma unroll
                for (int k = 0; k < 4; k++) M[h][k] = mul4(M[h][k], R[h][k]);
                e[h] += er[h];
            }
            next();
        };
        float4 Bh[2], Bl[2];
        const float4* Pc = reinterpret_cast<const float4*>(P + (size_t)(c0 + split) * numnodes * kP16Floats) + lane;
        auto matrix = [&](unsigned node) {
            const float4* pv = Pc + (size_t)node * (kP16Floats / 4);
            Bh[0] = __ldg(pv);
            Bh[1] = __ldg(pv + 32);
            Bl[0] = __ldg(pv + 64);
            Bl[1] = __ldg(pv + 96);
        };
        next();
        matrix((unsigned)__ldg(&sg.steps[1].self));
        for (; cc < nc; cc += stride, Pc += (size_t)stride * numnodes * (kP16Floats / 4)) {
            const unsigned last = (unsigned)((nc - cc) * numnodes - 1);
            gp = gathers + 1;
            si = reinterpret_cast<const int*>(sidx) + 32;
#pragma unroll
            for (int h = 0; h < NP; h++) e[h] = 0;
            float4* top = stack;
            for (int s = 0; s < nmul; s++) {
                const int2 op = ops[s];
                if (op.y & (kStepInit | kStepPop)) {
                    if (op.y & kStepInit) {
#pragma unroll
                        for (int h = 0; h < NP; h++) {
#pragma unroll
                            for (int k = 0; k < 4; k++) M[h][k] = R[h][k];
                            e[h] += er[h];
                        }
                        next();
                        continue;
                    }
                    pop(top);
                } else {
                    product();
                }
                // m_v = P_v x (the node's own branch)
#pragma unroll
                for (int h = 0; h < NP; h++) {
                    float D0[2][2][4], D1[2][2][4];
                    msg_mma(M[h], Bh, Bl, D0, D1);
                    if (h == NP - 1) matrix(min((unsigned)op.x, last));
                    // pair g + 8k, states 4t..4t+3; the two k-step halves
                    // added, then their truncation returned on average
                    float mx[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int mt = k >> 1, o = 2 * (k & 1);
                        M[h][k].x = add_half_ulp(D0[mt][0][o] + D1[mt][0][o]);
                        M[h][k].y = add_half_ulp(D0[mt][0][o + 1] + D1[mt][0][o + 1]);
                        M[h][k].z = add_half_ulp(D0[mt][1][o] + D1[mt][1][o]);
                        M[h][k].w = add_half_ulp(D0[mt][1][o + 1] + D1[mt][1][o + 1]);
                        mx[k] = max4(M[h][k]);
                    }
                    // Exact power-of-two rescale by the pair's largest state m to
                    // [0.5, 1): 2^(126 - E), E the exponent field of m; E = 0, a
                    // zero or denormal m, scales by 2^126 first.
                    const unsigned mb = __float_as_uint(quad_reduce(mx, t, [](float a, float b) { return fmaxf(a, b); }));
                    e[h] += (int)(mb >> 23) - 126;
                    const float sc = __uint_as_float((253u << 23) - (mb & 0x7f800000u));
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float sk = __shfl_sync(0xffffffffu, sc, (lane & 28) + k);
                        M[h][k] = mul4(M[h][k], make_float4(sk, sk, sk, sk));
                    }
                    // a denormal m: the rest of its way, or the next product would
                    // lose digits that a full row keeps (next to never: the vote costs
                    // less than the runs of one side differ)
                    const bool rest = mb - 1u < 0x007fffffu;
                    if (__any_sync(0xffffffffu, rest)) {
                        const unsigned rb = rest ? __float_as_uint(__uint_as_float(mb) * 0x1p126f) : (126u << 23);
                        e[h] += (int)(rb >> 23) - 126;
                        const float s2 = __uint_as_float((253u << 23) - (rb & 0x7f800000u));
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const float sk = __shfl_sync(0xffffffffu, s2, (lane & 28) + k);
                            M[h][k] = mul4(M[h][k], make_float4(sk, sk, sk, sk));
                        }
                    }
                }
                if (op.y & kStepPush) {
#pragma unroll
                    for (int h = 0; h < NP; h++)
#pragma unroll
                        for (int k = 0; k < 4; k++) top[128 * h + 32 * k] = M[h][k];
                    top += 128 * NP;
                }
            }
            if (ROOT) {
                if (ops[nmul].y & kStepPop) pop(top);
                else product();
                const float4 pc = __ldg(reinterpret_cast<const float4*>(pi16 + ((size_t)sg.grp * C + c0 + cc) * 16) + t);
#pragma unroll
                for (int h = 0; h < NP; h++) {
                    float d[4];
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        d[k] = pc.x * M[h][k].x + pc.y * M[h][k].y + pc.z * M[h][k].z + pc.w * M[h][k].w;
                    const float dot = quad_reduce(d, t, [](float a, float b) { return a + b; });
                    const double ll = (dot > 0.f) ? (double)logf(dot) + (double)e[h] * 0.69314718055994530942 : -INFINITY;
                    if (sg.catll && myu + 32 * h < n) sg.catll[(size_t)(c0 + cc) * n + myu + 32 * h] = ll;
                    const double tt = __ldg(logw + (size_t)sg.grp * C + c0 + cc) + ll;
                    if (ROOT == 1) mix[h].add(tt);
                    else collected[((pg * NP + h) * nc + cc) * 32 + lane] = tt;
                }
            } else {
#pragma unroll
                for (int h = 0; h < NP; h++) {
                    const int u0 = base + 32 * h + g;
                    const unsigned ob = sg.out + (unsigned)cc * sg.ocs;
                    float4* o = reinterpret_cast<float4*>(sg.rows) + ((size_t)ob + u0) * 4 + t;
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (u0 + 8 * k < n) o[32 * k] = M[h][k];
                    if (myu + 32 * h < n) sg.exps[(size_t)ob + myu + 32 * h] = e[h];
                }
            }
        }
    }
    if (ROOT == 2) {
        if (gridDim.y > 1) return;  // mix_values_kernel follows
        __syncthreads();
        if (split != 0 || !active) return;
#pragma unroll
        for (int h = 0; h < NP; h++)
            if (myu + 32 * h < n)
                mix_values(sg, collected + (size_t)(pg * NP + h) * nc * 32 + lane, myu + 32 * h, c0, nc, lam, per_lambda);
    }
    if (ROOT == 1 && active) {
#pragma unroll
        for (int h = 0; h < NP; h++) {
            const int u = myu + 32 * h;
            if (u >= n) continue;
            const double res = mix[h].value();
            sg.mix[u] = (c0 == 0) ? res : lse_d(sg.mix[u], res);
        }
    }
}

// The mixtures of the root's pairs whose categories several CTAs have shared: a
// warp per tile of 32 pairs.
__global__ void __launch_bounds__(128) mix_values_kernel(const SegDev* __restrict__ segs, const int2* __restrict__ tiles,
                                                         int ntiles, const double* __restrict__ values, int c0, int nc,
                                                         const int* __restrict__ lam, int per_lambda)
{
    const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (w >= ntiles) return;
    const int2 tile = tiles[w];
    const SegDev& sg = segs[tile.x];
    const int u = tile.y + (lane >> 2) + 8 * (lane & 3);
    if (u < sg.n) mix_values(sg, values + (size_t)w * nc * 32 + lane, u, c0, nc, lam, per_lambda);
}

// Gather indices of a segment from the per-node child lists: position p of a
// 32-pair tile holds pair g + 8k at p = 4g + k (the last pair repeated past
// the end).  One thread per position follows the lists from the top node down.
__global__ void __launch_bounds__(256) segment_idx_kernel(const IdxSeg* __restrict__ segs, const IdxOp* __restrict__ ops,
                                                          int seg0, const int* __restrict__ lr, int* __restrict__ idx)
{
    const IdxSeg sg = segs[seg0 + blockIdx.y];
    const long long pos = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long tile = pos >> 5;
    if (tile * 32 >= sg.n) return;
    const int p = (int)(pos & 31);
    const int u = min((int)tile * 32 + (p >> 2) + 8 * (p & 3), sg.n - 1);
    int row[kSegMaxNodes];
    row[0] = u;
    int* out = idx + sg.out + tile * sg.nb * 32 + p;
    for (int o = sg.op0; o < sg.op1; o++) {
        const IdxOp op = ops[o];
        const int r = __ldg(lr + op.list + row[op.src]);
        if (op.dst >= 0) row[op.dst] = r;
        else out[(size_t)(~op.dst) * 32] = r;
    }
}

int launch_segment_indices(const IdxSeg* d_segs, const IdxOp* d_ops, int nseg, int64_t maxn, const int* d_lr, int* d_idx,
                           cudaStream_t stream)
{
    if (maxn <= 0) return MESSI_OK;
    const unsigned gx = (unsigned)(((maxn + 31) / 32 * 32 + 255) / 256);
    for (int s = 0; s < nseg; s += 65535)
        segment_idx_kernel<<<dim3(gx, std::min(nseg - s, 65535)), 256, 0, stream>>>(d_segs, d_ops, s, d_lr, d_idx);
    return cudaPeekAtLastError() == cudaSuccess ? MESSI_OK : MESSI_ECUDA;
}

// ---------------------------------------------------------------------------
// tcgen05 form of the interior node update (launch shape 3, chosen only on
// request: MESSI_PRUNE_SHAPE=3).  The CTA's 128 unique pairs of one node are
// the M = 128 rows of one tcgen05.mma (kind::tf32, N = 16 states, K = 8):
//   * the child rows are gathered with cp.async into
//     a stage of whole rows with XOR-ordered quads (Stage), so that both the
//     gathers and thread p's reads of pair p's rows are free of bank
//     conflicts;
//   * thread p forms x = m_left * m_right, splits it into TF32 hi and lo and
//     writes both to its own TMEM lane (tcgen05.st): the A operand comes from
//     tensor memory, not through shared memory;
//   * the node's branch matrix P (B operand, N x K, K-major) is split into hi
//     and lo by the CTA and written to shared memory in the canonical
//     no-swizzle layout: core matrices of 8 rows x 16 bytes, the two 8-row
//     groups of N 128 bytes apart (SBO), the two 4-wide K groups of one MMA
//     256 bytes apart (LBO);
//   * one thread issues, per K half, lo*hi, hi*lo, hi*hi into that half's
//     own accumulator (TMEM columns 32..47 and 48..63), the same split and
//     order as prune_path_kernel (K half 0 = states {0,1,4,5,8,9,12,13}), and
//     commits them to an mbarrier;
//   * thread p reads its pair's 2 x 16 accumulators back (tcgen05.ld), adds
//     the halves and half an ulp as prune_path_kernel does, rescales by a power
//     of two and stores the row -- one category late: the MMAs of category c
//     run while the CTA waits for and multiplies the rows of category c + 1,
//     and P is loaded one category ahead.
// TMEM: 64 columns per CTA (A hi 0..15, A lo 16..31, D 32..63); at most 6
// CTAs of this kernel fit on an SM by shared memory (36 KB each), 384 columns.  A wait on
// the mbarrier that gives up (bounded) writes NaN rows, so the likelihood
// that uses them is NaN, and the CTA still frees its TMEM before it returns.
// ---------------------------------------------------------------------------
namespace tc {
constexpr int kStages = 2;
constexpr unsigned kCols = 64;
constexpr unsigned kColAhi = 0, kColAlo = 16, kColD = 32;

// A stage holds each pair's two child rows whole (64 bytes each: the four
// 16-byte copies of one row land side by side, as the gather delivers them),
// with the quads of row p in XOR order q ^ ((p / 2) % 4), so that thread p's
// load of quad q from 32 consecutive rows touches every bank once per
// 128 bytes.
struct Stage {
    float4 x[2][kTile][4];  // [side][pair][quad position]
    int e[2][kTile];
};
__device__ __forceinline__ int qpos(int p, int q) { return q ^ ((p >> 1) & 3); }

struct Smem {
    Stage st[kStages];
    float bhi[256];  // P hi, canonical K-major layout (boff below)
    float blo[256];
    unsigned long long mbar;
    unsigned tmem_base;
    int fail;
};

// Contraction index of column c (0..7) of K half ks: d = 4(c/2) + 2ks + c%2.
__host__ __device__ constexpr int kidx(int ks, int c) { return 4 * (c >> 1) + 2 * ks + (c & 1); }

// Float offset of P[i][d] in the B buffer: K half ks = (d/2)%2 at 128 floats,
// column c = 2(d/4) + d%2 of that half; core matrix (row group i/8, K group
// c/4) at (c/4)*64 + (i/8)*32 floats, row i%8 at 4 floats, element c%4.
__host__ __device__ constexpr int boff(int i, int d)
{
    return ((d >> 1) & 1) * 128 + (((2 * (d >> 2) + (d & 1)) >> 2) * 64) + (i >> 3) * 32 + (i & 7) * 4 +
           ((2 * (d >> 2) + (d & 1)) & 3);
}

// Row and state of P held at float o (even) of the B buffer: the inverse of
// boff, so that a thread storing floats o and o + 1 reads P[row][d..d+1].
__host__ __device__ constexpr int brow(int o) { return (((o & 127) >> 5 & 1) << 3) | (((o & 127) >> 2) & 7); }
__host__ __device__ constexpr int bstate(int o) { return kidx(o >> 7, (((o & 127) >> 6) << 2) | (o & 3)); }

constexpr bool b_layout_ok()
{
    bool seen[256] = {};
    for (int i = 0; i < 16; i++)
        for (int d = 0; d < 16; d++) {
            const int o = boff(i, d);
            if (o < 0 || o >= 256 || seen[o]) return false;
            seen[o] = true;
        }
    for (int o = 0; o < 256; o += 2)
        if ((bstate(o) & 1) || boff(brow(o), bstate(o)) != o || boff(brow(o), bstate(o) + 1) != o + 1) return false;
    return true;
}
static_assert(b_layout_ok(), "B operand layout: boff must be a bijection and brow/bstate its inverse");

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, no swizzle: start, LBO, SBO in 16-byte
// units; bit 46 = descriptor version 1.
__device__ __forceinline__ unsigned long long bdesc(unsigned addr)
{
    return (unsigned long long)((addr & 0x3FFFFu) >> 4) | ((unsigned long long)(256u >> 4) << 16) |
           ((unsigned long long)(128u >> 4) << 32) | (1ull << 46);
}

// Instruction descriptor, kind::tf32: D F32 (bits 4-5 = 1), A and B TF32
// (bits 7-9, 10-12 = 2), both K-major, N >> 3 at bits 17-22, M >> 4 at 24-28.
constexpr unsigned kIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void mma_ts(unsigned d, unsigned a, unsigned long long b, unsigned acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(kIdesc), "r"(acc));
}

__device__ __forceinline__ void st16(unsigned taddr, const uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(
            taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]));
}

__device__ __forceinline__ void ld32(unsigned taddr, uint32_t (&v)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// Bounded wait for phase `parity` of the mbarrier; false if it gave up.
__device__ __forceinline__ bool mbar_wait(unsigned addr, unsigned parity)
{
    for (int it = 0; it < (1 << 16); it++) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
}  // namespace tc

__global__ void __launch_bounds__(kTile, 6) prune_tc_kernel(const SegDev* __restrict__ segs,
                                                           const int2* __restrict__ tiles,
                                                           const float* __restrict__ P, int numnodes, int c0, int nc)
{
    extern __shared__ float4 smem_raw[];
    tc::Smem& S = *reinterpret_cast<tc::Smem*>(smem_raw);
    const int2 tile = tiles[blockIdx.x];
    const SegDev& nd = segs[tile.x];  // one node: its program is the two gathered children
    const StepDev sl = nd.steps[0], sr = nd.steps[1];
    const int self = sr.self;
    const int n = nd.n;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const unsigned mbar = tc::smem_u32(&S.mbar);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         tc::smem_u32(&S.tmem_base)),
                     "r"(tc::kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(mbar));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        S.fail = 0;
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const unsigned tbase = S.tmem_base;
    const unsigned tlane = tbase + ((unsigned)(32 * warp) << 16);  // this warp's 32 TMEM lanes

    // gathers: lane (g, t) copies state quad t of pairs g + 8k of its warp
    const int wbase = 32 * warp;
    const int4* src = reinterpret_cast<const int4*>(nd.idx) + (size_t)min((tile.y >> 5) + warp, (n - 1) >> 5) * 16 + g;
    const int4 l4 = __ldg(src), r4 = __ldg(src + 8);
    const int li[4] = {l4.x, l4.y, l4.z, l4.w}, ri[4] = {r4.x, r4.y, r4.z, r4.w};
    const int myl = own4(l4, t), myr = own4(r4, t);
    const float* lf = nd.rows + (size_t)sl.row * 16;
    const float* rf = nd.rows + (size_t)sr.row * 16;
    const int* le = (sl.flags & kStepLeaf) ? nullptr : nd.exps + sl.row;
    const int* re = (sr.flags & kStepLeaf) ? nullptr : nd.exps + sr.row;
    const long long lcs = sl.cs, rcs = sr.cs;
    auto issue = [&](int cc) {
        tc::Stage& st = S.st[cc % tc::kStages];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int pl = wbase + g + 8 * k;
            cp_async16(&st.x[0][pl][tc::qpos(pl, t)], lf + ((size_t)cc * lcs + li[k]) * 16 + 4 * t);
            cp_async16(&st.x[1][pl][tc::qpos(pl, t)], rf + ((size_t)cc * rcs + ri[k]) * 16 + 4 * t);
        }
        if (le) cp_async4(&st.e[0][wbase + g + 8 * t], le + (size_t)cc * lcs + myl);
        if (re) cp_async4(&st.e[1][wbase + g + 8 * t], re + (size_t)cc * rcs + myr);
    };
#pragma unroll
    for (int s0 = 0; s0 < tc::kStages - 1; s0++) {
        if (s0 < nc) issue(s0);
        cp_async_commit();
    }
    const int myu = tile.y + tid;  // the pair this thread finishes
    const bool myvalid = myu < n;
    // this thread's two B entries, in layout order (floats 2 tid and 2 tid + 1
    // of the buffer, the inverse of boff, so the stores are conflict-free): row
    // pi_ of P, states pd and pd + 1
    const int bo = 2 * tid;
    const int pi_ = tc::brow(bo), pd = tc::bstate(bo);
    auto pload = [&](int cc) {
        const float* p = P + ((size_t)(c0 + cc) * numnodes + self) * kP16Floats + p16_at(pi_, pd);
        const float2 h = __ldg(reinterpret_cast<const float2*>(p)), l = __ldg(reinterpret_cast<const float2*>(p + 256));
        return make_float2(h.x + l.x, h.y + l.y);
    };
    // category cf's accumulators back from TMEM (its MMAs ran while the next
    // category's rows were read), rescaled and stored with exponent ef
    auto finish = [&](int cf, int ef) {
        const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(mbar, (unsigned)(cf & 1)));
        tc::fence_after();
        float V[16];
        if (ok) {
            uint32_t D[32];
            tc::ld32(tlane + tc::kColD, D);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            // D[c] / D[16 + c]: K halves 0 and 1 of state c
#pragma unroll
            for (int c = 0; c < 16; c++) V[c] = add_half_ulp(__uint_as_float(D[c]) + __uint_as_float(D[16 + c]));
        } else {
#pragma unroll
            for (int c = 0; c < 16; c++) V[c] = __int_as_float(0x7fc00000);
            if (lane == 0) *(volatile int*)&S.fail = 1;
        }
        tc::fence_before();
        float m = V[0];
#pragma unroll
        for (int c = 1; c < 16; c++) m = fmaxf(m, V[c]);
        int ex;
        float pre, sc;
        pow2_scale(m, ex, pre, sc);
#pragma unroll
        for (int c = 0; c < 16; c++) V[c] *= pre;
        if (myvalid) {
            // the row as two 32-byte stores: whole sectors
            float* o = nd.rows + ((size_t)nd.out + (size_t)cf * nd.ocs + myu) * 16;
#pragma unroll
            for (int h = 0; h < 2; h++)
                asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(o + 8 * h),
                             "f"(V[8 * h] * sc), "f"(V[8 * h + 1] * sc), "f"(V[8 * h + 2] * sc),
                             "f"(V[8 * h + 3] * sc), "f"(V[8 * h + 4] * sc), "f"(V[8 * h + 5] * sc),
                             "f"(V[8 * h + 6] * sc), "f"(V[8 * h + 7] * sc)
                             : "memory");
            nd.exps[(size_t)nd.out + (size_t)cf * nd.ocs + myu] = ef + ex;
        }
    };
    float2 ppn = (nc > 0) ? pload(0) : make_float2(0.f, 0.f);
    int eprev = 0;
    for (int cc = 0; cc < nc; cc++) {
        if (cc + tc::kStages - 1 < nc) issue(cc + tc::kStages - 1);
        cp_async_commit();
        cp_async_wait<tc::kStages - 1>();
        __syncwarp();
        const float2 pp = ppn;
        if (cc + 1 < nc) ppn = pload(cc + 1);
        const tc::Stage& st = S.st[cc % tc::kStages];
        float x[16];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float4 a = st.x[0][tid][tc::qpos(tid, q)], b = st.x[1][tid][tc::qpos(tid, q)];
            x[4 * q] = a.x * b.x;
            x[4 * q + 1] = a.y * b.y;
            x[4 * q + 2] = a.z * b.z;
            x[4 * q + 3] = a.w * b.w;
        }
        const int e = (le ? st.e[0][tid] : 0) + (re ? st.e[1][tid] : 0);
        // the previous category's MMAs are done with A, B and D after this
        if (cc > 0) finish(cc - 1, eprev);
        {
            uint32_t hi[16], lo[16];
#pragma unroll
            for (int ks = 0; ks < 2; ks++)
#pragma unroll
                for (int c = 0; c < 8; c++) split_a(x[tc::kidx(ks, c)], hi[8 * ks + c], lo[8 * ks + c]);
            tc::st16(tlane + tc::kColAhi, hi);
            tc::st16(tlane + tc::kColAlo, lo);
        }
        {
            uint32_t h0, l0, h1, l1;
            split_a(pp.x, h0, l0);
            split_a(pp.y, h1, l1);
            *reinterpret_cast<float2*>(S.bhi + bo) = make_float2(__uint_as_float(h0), __uint_as_float(h1));
            *reinterpret_cast<float2*>(S.blo + bo) = make_float2(__uint_as_float(l0), __uint_as_float(l1));
        }
        asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        tc::fence_before();
        __syncthreads();
        if (*(volatile int*)&S.fail) break;  // a wait gave up (uniform: read after the barrier)
        if (tid == 0) {
            tc::fence_after();
            const unsigned bh = tc::smem_u32(S.bhi), bl = tc::smem_u32(S.blo);
#pragma unroll
            for (int ks = 0; ks < 2; ks++) {
                const unsigned d = tbase + tc::kColD + 16 * ks;
                const unsigned long long dh = tc::bdesc(bh + 512 * ks), dl = tc::bdesc(bl + 512 * ks);
                tc::mma_ts(d, tbase + tc::kColAlo + 8 * ks, dh, 0u);
                tc::mma_ts(d, tbase + tc::kColAhi + 8 * ks, dl, 1u);
                tc::mma_ts(d, tbase + tc::kColAhi + 8 * ks, dh, 1u);
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar)
                         : "memory");
        }
        eprev = e;
    }
    // S.fail is uniform here: last written before the final loop barrier
    if (nc > 0 && !*(volatile int*)&S.fail) finish(nc - 1, eprev);
    cp_async_wait<0>();
    tc::fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tbase), "r"(tc::kCols));
    }
}

static int launch_prune_tc(messi_ctx* ctx, const SegDev* d_segs, const int2* d_tiles, int nt, const float* d_P,
                           int numnodes, int c0, int nc)
{
    prune_tc_kernel<<<nt, kTile, sizeof(tc::Smem), ctx->stream>>>(d_segs, d_tiles, d_P, numnodes, c0, nc);
    LAUNCH_CHECK(ctx, "prune_tc_kernel");
    return MESSI_OK;
}

// pgs: pair groups of 32 * NP pairs per CTA (the level's tiles hold 32 * lv.pg pairs)
template <int ROOT, int NP, int MAXT, int MINB>
static int launch_path(messi_ctx* ctx, const SegDev* d_segs, const int2* d_tiles, const SegLevel& lv, int cs,
                       const float* d_P, int numnodes, int c0, int nc, int C, const float* d_pi16,
                       const double* d_logw, const int* d_lam, bool per_lambda, int ctas = 1,
                       double* shared_values = nullptr)
{
    const int pgs = lv.pg / NP, warps = pgs * cs;
    const size_t smem = sizeof(float4) * ((size_t)(lv.max_nb + 1) * (1 + 8 * lv.pg) + (lv.max_steps + 1) / 2 +
                                          (size_t)warps * NP * lv.max_depth * 128) +
                        (ROOT == 2 && ctas == 1 ? sizeof(double) * 32 * (size_t)lv.pg * nc : 0);
    const cudaError_t e = allow_smem(ctx->device, (const void*)prune_path_kernel<ROOT, NP, MAXT, MINB>, smem);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "prune_path_kernel attributes");
    prune_path_kernel<ROOT, NP, MAXT, MINB><<<dim3(lv.tile_cnt, ctas), 32 * warps, smem, ctx->stream>>>(
        d_segs, d_tiles + lv.tile_off, d_P, numnodes, c0, nc, C, d_pi16, d_logw, d_lam, per_lambda ? 1 : 0, cs,
        lv.max_steps, lv.max_nb, lv.max_depth, shared_values);
    LAUNCH_CHECK(ctx, ROOT ? "prune_path_kernel<root>" : "prune_path_kernel");
    return MESSI_OK;
}

constexpr int kMaxSplits = 12;  // category splits of a pair group: CTAs of up to 384 threads

int launch_prune_level(messi_ctx* ctx, const SegDev* d_segs, const int2* d_tiles, const SegLevel& lv, bool root,
                       const float* d_P, int numnodes, int c0, int nc, int C, const float* d_pi16,
                       const double* d_logw, const int* d_lam, bool per_lambda)
{
    if (lv.tile_cnt <= 0) return MESSI_OK;
    if (ctx->prune_shape == 3 && !root && lv.max_nb == 2 && lv.pg == 4)
        return launch_prune_tc(ctx, d_segs, d_tiles + lv.tile_off, lv.tile_cnt, d_P, numnodes, c0, nc);
#define MESSI_PATH(ROOT, NP, MAXT, MINB, CS)                                                                         \
    launch_path<ROOT, NP, MAXT, MINB>(ctx, d_segs, d_tiles, lv, CS, d_P, numnodes, c0, nc, C, d_pi16, d_logw, d_lam, \
                                      per_lambda)
    if (lv.pg == 4 && !per_lambda) {
        switch (ctx->prune_shape) {
            case 1: return root ? MESSI_PATH(1, 1, 128, 4, 1) : MESSI_PATH(0, 1, 128, 4, 1);
            case 2: return root ? MESSI_PATH(1, 2, 64, 6, 1) : MESSI_PATH(0, 2, 64, 6, 1);
            default: return root ? MESSI_PATH(1, 1, 128, 5, 1) : MESSI_PATH(0, 1, 128, 5, 1);
        }
    }
    // few pairs (or per-lambda mixtures): the warps of a pair group share the
    // categories until the GPU's 16 warps per SM are filled
    const int sms = ctx->num_sms > 0 ? ctx->num_sms : 152;
    const int64_t want = (lv.pg == 1) ? (16 * (int64_t)sms + lv.warps - 1) / std::max<int64_t>(lv.warps, 1) : 1;
    const int splits = (int)std::max<int64_t>(1, std::min<int64_t>(want, nc));
    const int ctas = (splits + kMaxSplits - 1) / kMaxSplits, cs = (splits + ctas - 1) / ctas;
    if (!root)
        return launch_path<0, 1, 32 * kMaxSplits, 1>(ctx, d_segs, d_tiles, lv, cs, d_P, numnodes, c0, nc, C, d_pi16, d_logw,
                                                     d_lam, per_lambda, ctas);
    void* values = nullptr;
    if (ctas > 1) {
        const int rc = ensure(ctx, kSlotCatMix, (size_t)lv.tile_cnt * nc * 32 * sizeof(double), &values);
        if (rc) return rc;
    }
    const int rc = launch_path<2, 1, 32 * kMaxSplits, 1>(ctx, d_segs, d_tiles, lv, cs, d_P, numnodes, c0, nc, C, d_pi16,
                                                         d_logw, d_lam, per_lambda, ctas, (double*)values);
    if (rc || ctas == 1) return rc;
    mix_values_kernel<<<(lv.tile_cnt + 3) / 4, 128, 0, ctx->stream>>>(d_segs, d_tiles + lv.tile_off, lv.tile_cnt,
                                                                     (const double*)values, c0, nc, d_lam,
                                                                     per_lambda ? 1 : 0);
    LAUNCH_CHECK(ctx, "mix_values_kernel");
    return MESSI_OK;
#undef MESSI_PATH
}

int run_pairs(messi_ctx* ctx, messi_dataset* ds, const float* d_P, const float* d_pi16, const double* d_logw,
              const int* d_lam, int C, int nlam, bool per_lambda)
{
    (void)nlam;
    const int chunk = std::min(ds->chunk, kCollectCategories);
    for (int c0 = 0; c0 < C; c0 += chunk) {
        const int nc = std::min(chunk, C - c0);
        int rc = launch_leaf_messages(ctx, ds->d_leaf, ds->leaf_rows, d_P, ds->numnodes, c0, nc, ds->d_leafmsg);
        if (rc) return rc;
        for (int lv = 1; lv <= ds->SH; lv++) {
            const SegLevel& sl = ds->seg_levels[lv];
            if (sl.tile_cnt == 0) continue;
            prof_begin(ctx, 0, sl.units * nc);
            rc = launch_prune_level(ctx, ds->d_segs, ds->d_tiles, sl, lv == ds->SH, d_P, ds->numnodes, c0, nc, C,
                                    d_pi16, d_logw, d_lam, per_lambda);
            if (rc) return rc;
            prof_end(ctx);
        }
    }
    return MESSI_OK;
}

// ---------------------------------------------------------------------------
// Unpaired columns (FP64), a warp per eight columns and site-rate category,
// lane 4 col + a for state a, then the mixture over site rates in the
// reference's order.  The FP64 units issue a warp only every 64 cycles per SM
// quarter, so the work is spread over four times the warps a thread per column
// would give, a leaf's 0/1 vector costs additions only for its second to
// fourth state, and the maximum is taken on the bits.  The nodes come as a
// program (plan.cpp): the last result stays in registers, one that waits for
// its sibling goes to a stack in shared memory, the deeper subtree first, so
// that the stack holds at most log2(sequences) results.  64 sequences x 1,000
// columns: 198 us with every node's partials in global memory and a thread per
// column, 160 with the program alone, 62 now; 100 x 733: 310 -> 96 us.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double shfl_d(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }

// staged: the tile's masks fit shared memory
__global__ void __launch_bounds__(32) unpaired_site_kernel(const uint8_t* __restrict__ masks, int N,
                                                           const int4* __restrict__ ops, int nops, int depth,
                                                           int staged, int L, const double* __restrict__ P4,
                                                           int pstride, const double* __restrict__ pi4,
                                                           double* __restrict__ ll)
{
    extern __shared__ double unpaired_smem[];
    double* stack = unpaired_smem + threadIdx.x;  // [depth][state, log scale][32]
    uint8_t* sm = reinterpret_cast<uint8_t*>(unpaired_smem + (size_t)depth * 64);
    const int col = threadIdx.x >> 2, a = threadIdx.x & 3, quad = threadIdx.x & 28;
    const int x = blockIdx.x * 8 + col, xc = min(x, L - 1);
    const int s = blockIdx.y;
    const double* Ps = P4 + (size_t)s * pstride * 16 + 4 * a;  // this lane's row of every matrix
    if (staged) {
        for (int k = threadIdx.x; k < 8 * N; k += 32)
            sm[k] = masks[(size_t)(k >> 3) * L + min((int)blockIdx.x * 8 + (k & 7), L - 1)];
        __syncwarp();
    }
    // sum over the leaf's states of P[a][.], ascending as the full product would add them
    auto leaf = [&](int seq, const double2& p01, const double2& p23) {
        const int m = staged ? sm[seq * 8 + col] : masks[(size_t)seq * L + xc];
        const double p[4] = {p01.x, p01.y, p23.x, p23.y};
        const int first = __ffs(m) - 1;
        double v = p[3];
#pragma unroll
        for (int d = 0; d < 3; d++)
            if (first == d) v = p[d];
#pragma unroll
        for (int d = 1; d < 4; d++)
            if (__any_sync(0xffffffffu, d > first && (m >> d & 1)) && d > first && (m >> d & 1)) v += p[d];
        return v;
    };
    auto inner = [&](double own, const double2& p01, const double2& p23) {
        double v = 0.0;
        v += p01.x * shfl_d(own, quad);
        v += p01.y * shfl_d(own, quad + 1);
        v += p23.x * shfl_d(own, quad + 2);
        v += p23.y * shfl_d(own, quad + 3);
        return v;
    };
    double top = 0.0, lm = 0.0;
    for (int t = 0; t < nops; t++) {
        const int4 op = __ldg(ops + t);  // children A, B; sequence of A, B (-1: A = the last result, B = the stack's)
        const double2* PA = reinterpret_cast<const double2*>(Ps + (size_t)op.x * 16);
        const double2* PB = reinterpret_cast<const double2*>(Ps + (size_t)op.y * 16);
        const double2 a01 = __ldg(PA), a23 = __ldg(PA + 1), b01 = __ldg(PB), b23 = __ldg(PB + 1);
        double l, r;
        if (op.z >= 0) {
            if (t > 0) {  // a new path: the last result waits for its sibling
                stack[0] = top;
                stack[32] = lm;
                stack += 64;
            }
            l = leaf(op.z, a01, a23);
            lm = 0.0;
        } else {
            l = inner(top, a01, a23);
        }
        if (op.w >= 0) {
            r = leaf(op.w, b01, b23);
        } else {
            stack -= 64;
            r = inner(stack[0], b01, b23);
            lm += stack[32];
        }
        top = l * r;
        // the largest state: non-negative doubles compare as their bits
        long long m = __double_as_longlong(top);
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
        if (__longlong_as_double(m) < 1e-20) {  // src/FARCE.jl:2226-2238
            top /= __longlong_as_double(m);
            lm += log(__longlong_as_double(m));
        }
    }
    double tot = 0.0;
#pragma unroll
    for (int d = 0; d < 4; d++) tot += pi4[d] * shfl_d(top, quad + d);
    if (x < L && a == 0) ll[(size_t)s * L + x] = log(tot) + lm;
}

__global__ void unpaired_mix_kernel(const double* __restrict__ ll, const double* __restrict__ logw_site, int nsite,
                                    int L, double* __restrict__ u)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= L) return;
    double acc = -INFINITY;
    for (int s = 0; s < nsite; s++) {
        const double v = ll[(size_t)s * L + x] + logw_site[s];
        acc = (s == 0) ? v : lse_d(acc, v);
    }
    u[x] = acc;
}

int launch_unpaired(messi_ctx* ctx, messi_dataset* ds, const double* d_P4, int pstride, const double* d_pi4,
                    const double* d_logw_site, int nsite, double* d_u, double* d_ll)
{
    // d_ll: nsite * L doubles, or nullptr for the context's buffer
    if (!d_ll) {
        void* scratch;
        int rc = ensure(ctx, kSlotUnpaired, (size_t)nsite * ds->L * sizeof(double), &scratch);
        if (rc) return rc;
        d_ll = (double*)scratch;
    }
    const size_t stack = (size_t)ds->unpaired_depth * 64 * sizeof(double), tile = (size_t)ds->N * 8;
    const int staged = stack + tile <= 48 * 1024 ? 1 : 0;
    unpaired_site_kernel<<<dim3((ds->L + 7) / 8, nsite), 32, stack + (staged ? tile : 0), ctx->stream>>>(
        ds->d_masks, ds->N, ds->d_uops, ds->N - 1, ds->unpaired_depth, staged, ds->L, d_P4, pstride, d_pi4, d_ll);
    LAUNCH_CHECK(ctx, "unpaired_site_kernel");
    unpaired_mix_kernel<<<(ds->L + 127) / 128, 128, 0, ctx->stream>>>(d_ll, d_logw_site, nsite, ds->L, d_u);
    LAUNCH_CHECK(ctx, "unpaired_mix_kernel");
    return MESSI_OK;
}

// ---------------------------------------------------------------------------
// Output layouts
// ---------------------------------------------------------------------------
// The symmetric L x L matrix from the band's unique root pairs.  A CTA takes 8
// rows by 32 columns that reach above the diagonal, a cell per thread along the
// band index's rows; a value is formed once and written to both triangles, the
// lower one through shared memory.  The factorised term is FP64 (an exp and a
// log1p a cell, 64 cycles a warp instruction and SM quarter): formed for both
// triangles a 733 x 733 matrix took 136 us, now 77.
constexpr int kScatterRows = 8;

__global__ void __launch_bounds__(32 * kScatterRows) scatter_dense_kernel(const int* __restrict__ bandidx,
                                                                          const double* __restrict__ vals,
                                                                          const double* __restrict__ u, double addw,
                                                                          int L, int W, double* __restrict__ out)
{
    __shared__ double tile[32][kScatterRows + 1];
    const int i0 = blockIdx.x * kScatterRows, j0 = blockIdx.y * 32;
    if (j0 + 31 < i0) return;
    const int c = threadIdx.x & 31, r = threadIdx.x >> 5, i = i0 + r, j = j0 + c;
    double val = -INFINITY;
    if (j < L && i < j && j - i <= W) {
        const int b = bandidx[(size_t)i * (W + 1) + (j - i)];
        if (b >= 0) {
            if (vals) val = vals[b];
            if (addw != -INFINITY) val = lse_d(val, addw + u[i] + u[j]);
        }
    }
    tile[c][r] = val;
    if (j < L && i <= j) out[(size_t)i * L + j] = val;
    __syncthreads();
    const int c2 = threadIdx.x / kScatterRows, r2 = threadIdx.x % kScatterRows;  // eight rows of a column side by side
    if (j0 + c2 < L && i0 + r2 < j0 + c2) out[(size_t)(j0 + c2) * L + i0 + r2] = tile[c2][r2];
}

int launch_scatter_dense(messi_ctx* ctx, messi_dataset* ds, const double* d_vals, const double* d_u, double addw,
                         double* d_out)
{
    const dim3 tiles((unsigned)((ds->L + kScatterRows - 1) / kScatterRows), (unsigned)((ds->L + 31) / 32));
    if (tiles.y > 65535u) return fail(ctx, MESSI_EINVAL, "scatter: more than 2,097,120 columns");
    if (addw != -INFINITY && !d_u) return fail(ctx, MESSI_EINVAL, "scatter: factorised term without unpaired values");
    scatter_dense_kernel<<<tiles, 32 * kScatterRows, 0, ctx->stream>>>(ds->d_bandidx, d_vals, d_u, addw, ds->L, ds->W,
                                                                     d_out);
    LAUNCH_CHECK(ctx, "scatter_dense_kernel");
    return MESSI_OK;
}

// Banded log-odds pair scores from the root mixtures (device-resident path),
// with maskgapped! (src/RNATools.jl:441-451) folded in.
// The factorised lambda categories add logwF + u[i] + u[j] to the mixture
// (logwF read from d_logwF when given: a replayed graph then sees each call's
// value).
__global__ void bandprep_from_mix_kernel(const int* __restrict__ bandidx, const double* __restrict__ mix, int L, int W,
                                         int Wb, int RS, const uint8_t* __restrict__ gapmask,
                                         const double* __restrict__ u, double logwF_value,
                                         const double* __restrict__ d_logwF, const double* __restrict__ b, double B,
                                         float* __restrict__ pb)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)L * RS) return;
    const double logwF = d_logwF ? *d_logwF : logwF_value;
    const int i = (int)(idx / RS), k = (int)(idx % RS);
    float out = -INFINITY;
    if (k >= 1 && k <= Wb && i + k < L && k <= W) {
        const int bi = bandidx[(size_t)i * (W + 1) + k];
        if (bi >= 0 && !(gapmask && (gapmask[i] || gapmask[i + k]))) {
            double p = mix[bi];
            if (logwF != -INFINITY) p = lse_d_fast(p, logwF + u[i] + u[i + k]);
            if (p != -INFINITY) out = (float)(B * p - b[i] - b[i + k]);
        }
    }
    pb[idx] = out;
}

int launch_bandprep_from_mix(messi_ctx* ctx, messi_dataset* ds, const Band& t, const uint8_t* d_gapmask, double B,
                             double logwF, const double* d_logwF)
{
    const long long n = (long long)t.L * t.RS;
    const int bs = 256;
    bandprep_from_mix_kernel<<<(unsigned)((n + bs - 1) / bs), bs, 0, ctx->stream>>>(
        ds->d_bandidx, ds->d_mix, ds->L, ds->W, t.Wb, t.RS, d_gapmask, t.u, logwF, d_logwF, t.b, B, t.pb);
    LAUNCH_CHECK(ctx, "bandprep_from_mix_kernel");
    return MESSI_OK;
}

// ---------------------------------------------------------------------------
// Site-rate conditionals (felsensteinposteriorsiterateconditionalscuda,
// src/FelsensteinCUDA.jl:518-717): for column x and site-rate category s,
//   LSE( log w_s + log single[x] + u_s[x],
//        over band partners y > x, categories with s1 = s:
//            log pair[x,y] + log w_c + ll_c(x, y),
//        over band partners y < x, categories with s2 = s:
//            log pair[y,x] + log w_c + ll_c(y, x) )
// Categories in the order s1, s2, lambda.  Two kernels:
//   * siterate_pairs_kernel, a thread per (unique root pair, site-rate
//     category, side): the log-sum-exp over the ns * nl categories that have
//     the rate s at the pair's first (side 0) or second column (side 1), so
//     that a column adds one term per partner, not ns * nl;
//   * siterate_cols_kernel, a warp per (column, category): its partners over
//     the lanes, each lane a running log-sum-exp, merged at the end.
// FP64 throughout; bound by the FP64 pipe (one exp per pair and category).  A
// term more than 45 nats below its maximum is below 2^-64 of the sum and its
// exp is not formed.  A NaN term, or infinities that meet, make the sum NaN (the
// comparisons with the limit are written so that a NaN takes the exp); an
// infinite pair posterior enters all ns * nl categories of its pair.  (One thread per (column, category) walking every partner
// and category with a log1p(exp) each took 16.6 ms at 64 x 600, span 300.)
// ---------------------------------------------------------------------------
constexpr double kNegligible = -45.0;

__global__ void __launch_bounds__(256) siterate_pairs_kernel(const double* __restrict__ catll, long long nroot,
                                                             const double* __restrict__ logw, int ns, int nl,
                                                             double* __restrict__ out)
{
    const long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int s = blockIdx.y % ns, side = blockIdx.y / ns;
    if (b >= nroot) return;
    double m = -INFINITY;
    for (int o = 0; o < ns; o++)
        for (int l = 0; l < nl; l++) {
            const int c = (side ? o * ns + s : s * ns + o) * nl + l;
            m = fmax(m, logw[c] + catll[(size_t)c * nroot + b]);
        }
    double acc = 0.0;
    if (m != -INFINITY)
        for (int o = 0; o < ns; o++)
            for (int l = 0; l < nl; l++) {
                const int c = (side ? o * ns + s : s * ns + o) * nl + l;
                const double d = logw[c] + catll[(size_t)c * nroot + b] - m;
                if (!(d < kNegligible)) acc += exp(d);
            }
    out[(size_t)blockIdx.y * nroot + b] = (m == -INFINITY) ? -INFINITY : m + log(acc);
}

// Running log-sum-exp in FP64.
struct LogSum {
    double m = -INFINITY, s = 0.0;
    __device__ __forceinline__ void add(double v, double w = 1.0)  // w e^v
    {
        if (v == -INFINITY) {
            s += 0.0 * w;  // (another sum's NaN)
        } else if (v > m) {
            s = s * ((m - v >= kNegligible) ? exp(m - v) : 0.0) + w;
            m = v;
        } else {
            s += w * ((v - m < kNegligible) ? 0.0 : exp(v - m));  // (a negligible sum's NaN, too)
        }
    }
    __device__ __forceinline__ double value() const { return (m == -INFINITY && s == 0.0) ? -INFINITY : m + log(s); }
};

__global__ void __launch_bounds__(128) siterate_cols_kernel(const int* __restrict__ bandidx, int L, int W,
                                                            const double* __restrict__ pairll, long long nroot, int ns,
                                                            int nl,
                                                            const double* __restrict__ single,
                                                            const double* __restrict__ pair,
                                                            const double* __restrict__ ull,
                                                            const double* __restrict__ logw_site,
                                                            double* __restrict__ out)
{
    const int x = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    const int s = blockIdx.y;
    if (x >= L) return;  // warp-uniform
    const double* first = pairll + (size_t)s * nroot;
    const double* second = pairll + (size_t)(ns + s) * nroot;
    LogSum acc;
    auto partner = [&](double pp, double ll) {
        if (pp > 0.0) acc.add((pp == INFINITY && ns * nl > 1) ? (double)NAN : log(pp) + ll);
    };
    if (lane == 0) {
        const double us = ull[(size_t)s * L + x];
        if (us != -INFINITY) acc.add(logw_site[s] + log(single[x]) + us);
    }
    for (int k = 1 + lane; k <= W && x + k < L; k += 32) {
        const int b = bandidx[(size_t)x * (W + 1) + k];
        if (b < 0) continue;
        partner(pair[(size_t)x + (size_t)(x + k) * L], first[b]);
    }
    for (int k = 1 + lane; k <= W && k <= x; k += 32) {
        const int b = bandidx[(size_t)(x - k) * (W + 1) + k];
        if (b < 0) continue;
        partner(pair[(size_t)(x - k) + (size_t)x * L], second[b]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double m2 = __shfl_down_sync(0xffffffffu, acc.m, off), s2 = __shfl_down_sync(0xffffffffu, acc.s, off);
        acc.add(m2, s2);
    }
    if (lane == 0) out[(size_t)s + (size_t)x * ns] = acc.value();
}

// d_pairll: 2 * nsite * nroot doubles of scratch
int launch_siterate_conditionals(messi_ctx* ctx, messi_dataset* ds, const double* d_catll, const double* d_logw,
                                 int nsite, int nlam, const double* d_single, const double* d_pair,
                                 const double* d_ull, const double* d_logw_site, double* d_pairll, double* d_out)
{
    if (ds->nroot > 0) {
        siterate_pairs_kernel<<<dim3((unsigned)((ds->nroot + 255) / 256), 2 * nsite), 256, 0, ctx->stream>>>(
            d_catll, ds->nroot, d_logw, nsite, nlam, d_pairll);
        LAUNCH_CHECK(ctx, "siterate_pairs_kernel");
    }
    siterate_cols_kernel<<<dim3((ds->L + 3) / 4, nsite), 128, 0, ctx->stream>>>(
        ds->d_bandidx, ds->L, ds->W, d_pairll, ds->nroot, nsite, nlam, d_single, d_pair, d_ull, d_logw_site, d_out);
    LAUNCH_CHECK(ctx, "siterate_cols_kernel");
    return MESSI_OK;
}

// ---------------------------------------------------------------------------
// Fixed-structure likelihood: sum of the unpaired columns and of the pairs
// (one block, FP64, fixed reduction order).  On return u holds the unpaired
// log-likelihood of unpaired columns and 0 on paired ones (the reference's
// computeunpairedlikelihoods(..., paired), src/FARCE.jl:1222-1250), pairll
// the pair log-likelihood at the first column of each pair and 0 elsewhere.
// colu[c]: unique root pair of the pair opened at column c (>= 0), -2 on the
// closing column of a pair, -1 on an unpaired column; partner[c] the other
// column of the pair opened at c.  The factorised lambda categories add
// logwF + u[c] + u[partner] to each pair, so the unpaired values of paired
// columns are read before they are cleared.
// ---------------------------------------------------------------------------
// A pair's value by a thread each, a warp per CTA: the FP64 units take 64 cycles
// a warp instruction, and one CTA's 1,000 columns kept its SM busy for 21 us.
__global__ void __launch_bounds__(32) structure_pairs_kernel(const double* __restrict__ u, const int* __restrict__ colu,
                                                             const int* __restrict__ partner, int L,
                                                             const double* __restrict__ mix, double logwF,
                                                             double* __restrict__ pairll)
{
    const int c = blockIdx.x * 32 + threadIdx.x;
    if (c >= L) return;
    const int k = colu[c];
    double pv = 0.0;
    if (k >= 0) {
        pv = mix[k];
        if (logwF != -INFINITY) pv = lse_d(pv, logwF + u[c] + u[partner[c]]);
    }
    pairll[c] = pv;
}

__global__ void __launch_bounds__(1024) structure_sum_kernel(double* __restrict__ u, const int* __restrict__ colu, int L,
                                                             double* __restrict__ total,
                                                             const double* __restrict__ pairll)
{
    __shared__ double part[1024];
    double acc = 0.0;
    for (int c = threadIdx.x; c < L; c += blockDim.x) {
        if (colu[c] == -1) acc += u[c];
        else u[c] = 0.0;
        acc += pairll[c];
    }
    part[threadIdx.x] = acc;
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) part[threadIdx.x] += part[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) total[0] = part[0];
}

int launch_structure_sum(messi_ctx* ctx, int L, double* d_u, const int* d_colu, const int* d_partner,
                         const double* d_mix, double logwF, double* d_total, double* d_pairll)
{
    structure_pairs_kernel<<<(L + 31) / 32, 32, 0, ctx->stream>>>(d_u, d_colu, d_partner, L, d_mix, logwF, d_pairll);
    LAUNCH_CHECK(ctx, "structure_pairs_kernel");
    structure_sum_kernel<<<1, 1024, 0, ctx->stream>>>(d_u, d_colu, L, d_total, d_pairll);
    LAUNCH_CHECK(ctx, "structure_sum_kernel");
    return MESSI_OK;
}

}  // namespace messi
