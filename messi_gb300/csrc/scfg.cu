// scfg.cu -- KH99 SCFG inside/outside passes and base-pairing posteriors (HP2).
//
// Replaces initialiseinside / insidealgorithm / insidez / outsidealgorithm of
// src/cuda/inside.cu (driven by src/InsideCUDA.jl:87-181, 301-389) and the
// CPU computebasepairprobs (src/InsideOutsideAlgorithm.jl:486-533).
//
// Representation.  Cells are stored as FP32 log-odds against a per-column
// baseline b_k = B*(u_k + log r1 + log r6) (u_k: unpaired log-likelihood):
//     Xbar(i,j) = X(i,j) - sum_{k=i..j} b_k.
// The baseline is additive over the split point, so the recurrences keep
// their form with pair scores pbar_ij = B*p_ij - b_i - b_j; an all-unpaired
// span keeps Sbar constant, which keeps FP32 magnitudes small.  The prefix
// sums of b and Z = Sbar(0, L-1) + sum_k b_k are FP64.
//
// Banding.  With every pair of span > Wb forbidden, only cells of span <= Wb
// and the S cells of the last column (the "suffix") reach Z
// (S->LS chains end at j = L-1; F and L need an enclosing or own pair), so
// the pass keeps a band of Wb+1 diagonals plus one suffix column.
//
// Layouts (row stride RS floats, RS >= Wb+1, multiple of 32):
//   Lrow[i][k] = Lbar(i, i+k)     Lcol[j][k] = Lbar(j-k, j)
//   Srow[i][k] = Sbar(i, i+k)     Scol[j][k] = Sbar(j-k, j)
//   Frow[i][k] = Fbar(i, i+k)     pb[i][k]   = pbar(i, i+k)
//   Ssuf[i]    = Sbar(i, L-1)
// so the split sum of cell (i, j) reads row i of L and column j of S with
// unit stride.  Outside tables mirror them (OSrow/OScol/OFrow/OFcol/OLrow/Osuf).
//
// Schedule.  One persistent cooperative launch walks the band diagonals (a
// wavefront): all cells of a span are independent, so each diagonal is spread
// over the whole grid, two diagonals at a time (the rows of a pair are dealt to
// the CTAs, and the second diagonal reads the first only at the CTA's own rows).
// The CTAs wait for one another's cells; the waits have a bounded
// iteration count: on timeout an error flag is raised, every CTA leaves, Z
// becomes NaN and the host returns MESSI_ETIMEOUT.  A cell's split sum is
// reduced by a group of G lanes (G grows with the number of split points) with
// shuffle log-sum-exp; its middle split points, which do not read the diagonals
// just finished, are summed one pair ahead.  The suffix recurrences run in one
// CTA of 16 warps in blocks of 32 cells: the terms that reach outside the
// block are summed by its warps in parallel, the in-block triangle by one warp.
#include <algorithm>
#include <cmath>

#include "internal.h"
#include "wave.cuh"

namespace messi {

namespace {

__device__ __forceinline__ void lse_add(float& m, float& s, float x)
{
    if (x > m) {
        s = s * __expf(m - x) + 1.f;
        m = x;
    } else if (x != -INFINITY) {
        s += __expf(x - m);
    }
}

// Four terms at once: the loads feeding them are independent, so a lane keeps
// four L2 requests in flight instead of one.
__device__ __forceinline__ void lse_add4(float& m, float& s, float x0, float x1, float x2, float x3)
{
    const float mx = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3));
    if (mx == -INFINITY) return;
    if (mx > m) {
        s *= __expf(m - mx);
        m = mx;
    }
    s += (__expf(x0 - m) + __expf(x1 - m)) + (__expf(x2 - m) + __expf(x3 - m));
}

// Eight terms at once (sixteen independent loads in flight per lane).
// Without branches: the rescale of (m, s) always runs (exp(0) = 1 leaves s
// exactly as it is when the block brings no larger term, and a block of
// -inf terms adds exact zeros), so lanes of a warp never diverge here.
__device__ __forceinline__ void lse_add8(float& m, float& s, const float (&x)[8])
{
    // the maximum as a tree (three dependent steps instead of seven; exact)
    const float mx = fmaxf(fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3])), fmaxf(fmaxf(x[4], x[5]), fmaxf(x[6], x[7])));
    const float nm = fmaxf(m, mx);
    const float base = (nm == -INFINITY) ? 0.f : nm;
    s *= __expf(m - base);
    m = nm;
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q += 2) {
        a += __expf(x[q] - base);
        b += __expf(x[q + 1] - base);
    }
    s += a + b;
}

__device__ __forceinline__ void lse_merge(float& m, float& s, float m2, float s2)
{
    if (m2 > m) {
        s = s * __expf(m - m2) + s2;
        m = m2;
    } else if (m2 != -INFINITY) {
        s += s2 * __expf(m2 - m);
    }
}

__device__ __forceinline__ float lse_val(float m, float s) { return (m == -INFINITY) ? -INFINITY : m + __logf(s); }

__device__ __forceinline__ float lse2f(float a, float b)
{
    const float m = fmaxf(a, b);
    if (m == -INFINITY) return -INFINITY;
    return m + __logf(__expf(a - m) + __expf(b - m));
}

// Adds sl * exp(x0) to the log-sum-exp (m, s) without branches (x0, m may
// be -inf): the serial triangle of the suffix recurrences, where a branch
// would split the warp on every step.
__device__ __forceinline__ void lse_add_scaled(float& m, float& s, float x0, float sl)
{
    const float mx = fmaxf(m, x0);
    const float base = (mx == -INFINITY) ? 0.f : mx;
    s = s * __expf(m - base) + sl * __expf(x0 - base);
    m = mx;
}

template <int G>
__device__ __forceinline__ void group_reduce(float& m, float& s)
{
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, off);
        const float s2 = __shfl_xor_sync(0xffffffffu, s, off);
        lse_merge(m, s, m2, s2);
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// workspace
// ---------------------------------------------------------------------------
int band_alloc(messi_ctx* ctx, int L, int Wb, bool outside, Band* t)
{
    t->L = L;
    t->Wb = Wb;
    t->RS = ((Wb + 1 + 31) / 32) * 32;
    const size_t tab = (size_t)L * t->RS * sizeof(float);
    void* p;
    int rc;
    float** in_tabs[6] = {&t->Lrow, &t->Lcol, &t->Srow, &t->Scol, &t->Frow, &t->pb};
    for (int k = 0; k < 6; k++) {
        if ((rc = ensure(ctx, k, tab, &p))) return rc;
        *in_tabs[k] = (float*)p;
    }
    if ((rc = ensure(ctx, 6, (size_t)(L + 1) * sizeof(float) * 2, &p))) return rc;
    t->Ssuf = (float*)p;
    t->Osuf = t->Ssuf + (L + 1);
    if ((rc = ensure(ctx, 7, (size_t)(3 * L + 8 + kSyncWords / 2) * sizeof(double), &p))) return rc;
    t->b = (double*)p;
    t->cb = t->b + L;
    t->u = t->cb + (L + 1);
    t->Zd = t->u + L;
    t->maxspan = (int*)(t->Zd + 2);
    t->sync = (unsigned int*)(t->Zd + 4);
    if (outside) {
        float** out_tabs[6] = {&t->OSrow, &t->OScol, &t->OFrow, &t->OFcol, &t->OLrow, &t->PP};
        for (int k = 0; k < 6; k++) {
            if ((rc = ensure(ctx, 8 + k, tab, &p))) return rc;
            *out_tabs[k] = (float*)p;
        }
        if ((rc = ensure(ctx, 14, (size_t)3 * L * sizeof(float), &p))) return rc;
        t->SL = (float*)p;
        t->nrm = t->SL + L;
        t->OSlast = t->nrm + L;
    } else {
        t->OSrow = t->OScol = t->OFrow = t->OFcol = t->OLrow = t->PP = t->SL = t->nrm = t->OSlast = nullptr;
    }
    return MESSI_OK;
}

Rules make_rules(double B)
{
    Rules r;
    for (int k = 0; k < 7; k++) r.r[k] = (float)(B * std::log(kKH99Prob[k]));
    return r;
}

static double baseline_c() { return std::log(0.868534) + std::log(0.894603); }

// ---------------------------------------------------------------------------
// baseline b_k and prefix sums cb (one block, deterministic FP64 scan)
// ---------------------------------------------------------------------------
__device__ void baseline_body(const double* __restrict__ u, int L, double B, double c, double* __restrict__ b,
                              double* __restrict__ cb)
{
    __shared__ double part[1024];
    const int t = threadIdx.x, nt = blockDim.x;
    const int per = (L + nt - 1) / nt;
    const int lo = min(L, t * per), hi = min(L, lo + per);
    double s = 0.0;
    for (int k = lo; k < hi; k++) {
        const double uk = u[k];
        const double bk = B * ((isfinite(uk) ? uk : 0.0) + c);
        b[k] = bk;
        s += bk;
    }
    part[t] = s;
    __syncthreads();
    for (int off = 1; off < nt; off <<= 1) {
        const double v = (t >= off) ? part[t - off] : 0.0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    double run = (t == 0) ? 0.0 : part[t - 1];
    for (int k = lo; k < hi; k++) {
        cb[k] = run;
        run += b[k];
    }
    if (t == nt - 1) cb[L] = part[nt - 1];
}

__global__ void baseline_kernel(const double* __restrict__ u, int L, double B, double c, double* __restrict__ b,
                                double* __restrict__ cb)
{
    baseline_body(u, L, B, c, b, cb);
}

// one block per alignment of a batch
__global__ void baseline_batch_kernel(const Band* __restrict__ bands, double B, double c)
{
    const Band t = bands[blockIdx.x];
    baseline_body(t.u, t.L, B, c, t.b, t.cb);
}

int launch_baseline(messi_ctx* ctx, const Band& t, double B)
{
    baseline_kernel<<<1, 1024, 0, ctx->stream>>>(t.u, t.L, B, baseline_c(), t.b, t.cb);
    LAUNCH_CHECK(ctx, "baseline_kernel");
    return MESSI_OK;
}

// ---------------------------------------------------------------------------
// pair-score preparation from a dense host matrix
// ---------------------------------------------------------------------------
__global__ void maxspan_kernel(const double* __restrict__ p, int L, int* __restrict__ out)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int best = 0;
    if (idx < (long long)L * L) {
        const int i = (int)(idx % L), j = (int)(idx / L);
        if (i < j && isfinite(p[idx])) best = j - i;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, off));
    if ((threadIdx.x & 31) == 0 && best > 0) atomicMax(out, best);
}

int launch_maxspan(messi_ctx* ctx, int L, const double* d_dense, int* d_out)
{
    cudaError_t e = cudaMemsetAsync(d_out, 0, sizeof(int), ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "memset maxspan");
    const long long n = (long long)L * L;
    maxspan_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(d_dense, L, d_out);
    LAUNCH_CHECK(ctx, "maxspan_kernel");
    return MESSI_OK;
}

// pb[i][k] from the upper triangle p(i, i+k) of a dense column-major matrix.
// Threads walk i fastest for a fixed column j so the dense reads coalesce.
__global__ void bandprep_from_dense_kernel(const double* __restrict__ p, int L, int Wb, int RS,
                                           const double* __restrict__ b, double B, float* __restrict__ pb)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)L * RS) return;
    const int j = (int)(idx / RS), r = (int)(idx % RS);
    // r enumerates rows i = j - RS + 1 + r .. j; k = j - i
    const int k = RS - 1 - r;
    const int i = j - k;
    if (i < 0) return;
    float out = -INFINITY;
    if (k >= 1 && k <= Wb) {
        const double v = p[(size_t)i + (size_t)j * L];
        if (v != -INFINITY && !isnan(v)) out = (float)(B * v - b[i] - b[j]);
    }
    pb[(size_t)i * RS + k] = out;
}

__global__ void fill_kernel(float* __restrict__ a, long long n, float v)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < n) a[idx] = v;
}

static int fill(messi_ctx* ctx, float* a, long long n, float v)
{
    fill_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(a, n, v);
    LAUNCH_CHECK(ctx, "fill_kernel");
    return MESSI_OK;
}

int launch_bandprep_from_dense(messi_ctx* ctx, const Band& t, const double* d_dense, double B)
{
    int rc = fill(ctx, t.pb, (long long)t.L * t.RS, -INFINITY);
    if (rc) return rc;
    const long long n = (long long)t.L * t.RS;
    bandprep_from_dense_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(d_dense, t.L, t.Wb, t.RS, t.b,
                                                                                      B, t.pb);
    LAUNCH_CHECK(ctx, "bandprep_from_dense_kernel");
    return MESSI_OK;
}

// ---------------------------------------------------------------------------
// inside
// ---------------------------------------------------------------------------
// Ssuf[i] for spans beyond the band (i < T = L-1-Wb), descending i:
// Ssuf[i] = r1 + LSE_{k=0..Wb} (Lrow[i][k] + Ssuf[i+k+1]), a recurrence
// whose every cell waits for the Wb+1 cells after it.  One CTA, blocks of 32
// cells from the top.  Every cell keeps a running log-sum-exp (m, s) of the
// terms whose S cell is already final, in shared memory over a window of
// cells (slot c % win): first the terms into the band's last column (j >= T),
// then, each time a block is final, its 32 values are pushed into the cells
// that reference them.  A push of S cell j into cell c adds L(c, j-1) +
// Ssuf[j]; for fixed j, L(c, j-1) = Lcol[j-1][j-1-c] is contiguous in c, so
// threads that own consecutive cells load consecutive words.  Warp 0 pushes
// into the next block's cells and solves that block's in-block triangle by
// column-oriented substitution; meanwhile the other warps push into the
// farther cells; one CTA barrier per block.  (The former form pulled each
// block's Wb+1 terms per cell from global memory after the block above was
// final: 2.7 ms for the 8,199 suffix cells of a 9,000-column alignment with
// span 800.)
// threads of a suffix CTA (16 warps: 128 registers each, so warp 0 keeps its
// 32 prefetched terms in registers across the triangle)
constexpr int kSuffixThreads = 512;

__host__ __device__ inline int suffix_window(int Wb) { return Wb + 64; }

// Asks L2 to fetch rows [r0, r1] of a band table (RS floats per row) from
// DRAM, `nlines` 128-byte lines from the start of each row, by threads tid
// of nthr; rows outside [0, L) are skipped.  The suffix recurrences walk the
// band tables one 32-row block at a time, and when the inside wavefront's
// tables exceed L2 each block's rows would otherwise arrive at DRAM latency
// on the single CTA's critical path.
__device__ __forceinline__ void prefetch_rows_l2(const float* tab, int RS, int L, int r0, int r1, int nlines, int tid,
                                                 int nthr)
{
    r0 = max(r0, 0);
    r1 = min(r1, L - 1);
    if (r1 < r0) return;
    const int n = (r1 - r0 + 1) * nlines;
    for (int x = tid; x < n; x += nthr) {
        const float* p = tab + (size_t)(r0 + x / nlines) * RS + (size_t)(x % nlines) * 32;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(p)));
    }
}

// A read-only global load under a predicate (`dflt` where it is false),
// written as one predicated instruction so that a run of them stays a run of
// independent loads in flight (a conditional expression may become a branch
// around each load, and the loads one after another).  `p` is never read
// when `pred` is false.
__device__ __forceinline__ float ldg_if(const float* p, bool pred, float dflt)
{
    float v;
    asm("{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %2, 0;\n\t"
        "mov.f32 %0, %3;\n\t"
        "@q ld.global.nc.f32 %0, [%1];\n\t}"
        : "=f"(v)
        : "l"(__cvta_generic_to_global(p)), "r"((int)pred), "f"(dflt));
    return v;
}

// ldg_if through L2 only (ld.global.cg): for the wavefronts' tables, which
// other CTAs write during the launch.
__device__ __forceinline__ float ldcg_if(const float* p, bool pred, float dflt)
{
    float v;
    asm("{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %2, 0;\n\t"
        "mov.f32 %0, %3;\n\t"
        "@q ld.global.cg.f32 %0, [%1];\n\t}"
        : "=f"(v)
        : "l"(__cvta_generic_to_global(p)), "r"((int)pred), "f"(dflt));
    return v;
}

// Adds to (m, s) the terms col[u] + vals[u] for the block's values u < nb,
// where col[u] = tab[(jbase + dj*u) * RS + kbase - u] (the L cell that joins
// this thread's cell to value u; skipped when its band offset kbase - u is
// outside 0..Wb): the valid u are one range, computed once, and the
// addresses one base plus u times a stride, so a load costs two compares and
// an address step; the 32 loads are issued together, then summed in blocks
// of eight.
__device__ __forceinline__ void suffix_push_terms(float& m, float& s, const float* __restrict__ tab, int RS,
                                                  int jbase, int dj, int kbase, const float* vals, int nb, int Wb)
{
    const int ulo = max(0, kbase - Wb), uhi = min(nb - 1, kbase);
    const long long step = (long long)dj * RS - 1;
    const float* base = tab + ((ulo <= uhi) ? (long long)jbase * RS + kbase : 0);
    float x[32];
#pragma unroll
    for (int u = 0; u < 32; u++) {
        const bool on = u >= ulo && u <= uhi;
        x[u] = ldg_if(base + (on ? u * step : 0), on, -INFINITY);
    }
#pragma unroll
    for (int u = 0; u < 32; u++) x[u] += vals[u];
#pragma unroll
    for (int u = 0; u < 32; u += 8) {
        const float y[8] = {x[u], x[u + 1], x[u + 2], x[u + 3], x[u + 4], x[u + 5], x[u + 6], x[u + 7]};
        lse_add8(m, s, y);
    }
}

// In-block triangle of a suffix recurrence, by one warp: lane q owns cell q
// of the block (nb cells) and enters with the log-sum-exp (m, s) of its
// terms from outside the block; once cell l is final it adds
// tri[q][q-l-1] + r1 + value_l to every later lane q (recv: the lane takes
// in-block terms).  Returns every lane's final (m, s).
// Linear form first: values relative to the block's largest accumulator in
// FP32, the factors E = exp(tri + r1) staged beside tri by the staging warp,
// so a step of the serial chain is one broadcast and one multiply-add (the
// log form's step, two exponentials and their max, took ~290 cycles).  Where
// a value leaves [1e-30, 1e30] of the reference (FP32 would lose digits or
// overflow) the block is redone in the log-sum-exp form.
__device__ __forceinline__ void suffix_triangle(float& m, float& s, const float (&tri)[32][33],
                                                const float (&etri)[32][33], int nb, bool recv, int Wb, float r1,
                                                int lane)
{
    float mx = m;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    const float ref = (mx == -INFINITY) ? 0.f : mx;
    float A = (m == -INFINITY) ? 0.f : s * __expf(m - ref);
    // the factors exp(tri + r1), staged with tri (unconditional shared
    // loads at a clamped index, then the selects)
    float E[32];
#pragma unroll
    for (int l = 0; l < 32; l++) E[l] = etri[lane][max(lane - l - 1, 0)];
#pragma unroll
    for (int l = 0; l < 32; l++) {
        const int k = lane - l - 1;
        E[l] = (recv && l < lane && k <= Wb) ? E[l] : 0.f;
    }
    // the serial chain: lane l's A is final at step l (full blocks without
    // the per-step bound check)
    if (nb == 32) {
#pragma unroll
        for (int l = 0; l < 32; l++) A = fmaf(E[l], __shfl_sync(0xffffffffu, A, l), A);
    } else {
#pragma unroll
        for (int l = 0; l < 32; l++)
            if (l < nb) A = fmaf(E[l], __shfl_sync(0xffffffffu, A, l), A);
    }
    // whether the lane has any term (a zero A is then an underflow), off the chain
    bool any = (m != -INFINITY);
#pragma unroll
    for (int l = 0; l < 32; l++) {
        const float V = __shfl_sync(0xffffffffu, A, l);
        any = any || (l < nb && E[l] > 0.f && V > 0.f);
    }
    const bool bad = (lane < nb) && (!(A <= 1e30f) || (any && A < 1e-30f));
    if (!__any_sync(0xffffffffu, bad)) {
        if (A > 0.f) {
            m = ref;
            s = A;
        } else {
            m = -INFINITY;
            s = 0.f;
        }
        return;
    }
#pragma unroll
    for (int l = 0; l < 32; l++) {
        if (l < nb) {
            const float ml = __shfl_sync(0xffffffffu, m, l), sl = __shfl_sync(0xffffffffu, s, l);
            const int k = lane - l - 1;
            if (recv && lane > l && k <= Wb) lse_add_scaled(m, s, tri[lane][k] + r1 + ml, sl);
        }
    }
}

__device__ void inside_suffix_body(const Band& t, const Rules& R, float* am, float* as, int win)
{
    const int L = t.L, Wb = t.Wb, RS = t.RS;
    const int T = L - 1 - Wb;
    if (T <= 0) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    // tri[q][k] = Lrow[i0 - q][k]: the in-block terms of the block's cells,
    // double-buffered (warp 1 stages the next block's while warp 0 solves)
    __shared__ float tri2[2][32][33];
    __shared__ float etri2[2][32][33];  // exp(tri + r1), staged with tri
    // finished block values, double-buffered: the far pushes of one block may
    // still read them while warp 0 solves the next block
    __shared__ float vals2[2][32];
    // xs[u][q]: the L value joining next-block cell lo-1-q to this block's
    // cell i0-u (warp 0's push after the triangle), staged a block ahead by
    // warp 1 and read into registers at the top of the block
    __shared__ float xs2[2][32][33];
    int parity = 0, tb = 0;
    for (int c = threadIdx.x; c < win; c += blockDim.x) {
        am[c] = -INFINITY;
        as[c] = 0.f;
    }
    __syncthreads();
    // terms into the band's last column: cells T-1 down to T-1-Wb, a warp per cell
    const int c_first = max(0, T - 1 - Wb);
    for (int c = T - 1 - w; c >= c_first; c -= nw) {
        float m = -INFINITY, s = 0.f;
        const float* lrow = t.Lrow + (size_t)c * RS;
        const int k1 = min(L - 1, c + Wb + 1) - c - 1;
        for (int k = (T - c - 1) + lane; k <= k1; k += 512) {
            float x[16];
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const int kq = k + 32 * q;
                x[q] = (kq <= k1) ? __ldg(lrow + kq) + t.Ssuf[c + kq + 1] : -INFINITY;
            }
            const float y0[8] = {x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7]};
            const float y1[8] = {x[8], x[9], x[10], x[11], x[12], x[13], x[14], x[15]};
            lse_add8(m, s, y0);
            lse_add8(m, s, y1);
        }
        group_reduce<32>(m, s);
        if (lane == 0) {
            am[c % win] = m;
            as[c % win] = s;
        }
    }
    int i0 = T - 1, lo = max(0, i0 - 31);
    // the first two blocks' pushes (Lcol rows lo-33 .. i0-1) and the second
    // block's in-block terms (first line of Lrow rows lo-32 .. lo-1)
    prefetch_rows_l2(t.Lcol, RS, L, lo - 33, i0 - 1, RS / 32, threadIdx.x, blockDim.x);
    prefetch_rows_l2(t.Lrow, RS, L, lo - 32, lo - 1, 1, threadIdx.x, blockDim.x);
    if (w == 1) {
        for (int q = 0; q < 32; q++) {
            const float v = (i0 - q >= lo && lane <= Wb) ? __ldg(t.Lrow + (size_t)(i0 - q) * RS + lane) : -INFINITY;
            tri2[0][q][lane] = v;
            etri2[0][q][lane] = __expf(v + R.r[0]);
        }
        const int nb0 = i0 - lo + 1, nlo0 = max(0, lo - 32), c = lo - 1 - lane;
        for (int u = 0; u < 32; u++) {
            const int k = i0 - 1 - c - u;
            xs2[0][u][lane] = (lo > 0 && c >= nlo0 && u < nb0 && k <= Wb) ? __ldg(t.Lcol + (size_t)(i0 - 1 - u) * RS + k)
                                                                          : -INFINITY;
        }
    }
    __syncthreads();
    float cm = -INFINITY, cs = 0.f;  // warp 0: accumulator of cell i0 - lane
    if (w == 0 && i0 - lane >= lo) {
        cm = am[(i0 - lane) % win];
        cs = as[(i0 - lane) % win];
    }
    for (;;) {
        const int nb = i0 - lo + 1;
        const int nlo = max(0, lo - 32);
        float* vals = vals2[parity];
        parity ^= 1;
        float x[32];  // warp 0: L values joining its next-block cell to this block's cells
        if (w == 0) {
            // column-oriented substitution: lane q owns cell i0 - q
            float m = (lane < nb) ? cm : -INFINITY, s = (lane < nb) ? cs : 0.f;
            suffix_triangle(m, s, tri2[tb], etri2[tb], nb, lane < nb, Wb, R.r[0], lane);
            // the block's values, formed and stored by all lanes at once
            if (lane < nb) {
                const float sv = R.r[0] + lse_val(m, s);
                t.Ssuf[i0 - lane] = sv;
                vals[lane] = sv;
            }
            // the push operands, before the barrier: warp 1 refills this
            // buffer in the next block
#pragma unroll
            for (int u = 0; u < 32; u++) x[u] = xs2[tb][u][lane];
        } else if (w == 1 && lo > 0) {
            // the next block's in-block terms and push operands: all 64 loads
            // first, then the stores (one memory round trip)
            const int i0n = lo - 1, nbn = lo - nlo, nlon = max(0, nlo - 32), c = nlo - 1 - lane;
            float v[32], y[32];
#pragma unroll
            for (int q = 0; q < 32; q++) {
                const bool onv = lo - 1 - q >= nlo && lane <= Wb;
                v[q] = ldg_if(t.Lrow + (onv ? (size_t)(lo - 1 - q) * RS + lane : 0), onv, -INFINITY);
                const int k = i0n - 1 - c - q;
                const bool ony = nlo > 0 && c >= nlon && q < nbn && k <= Wb;
                y[q] = ldg_if(t.Lcol + (ony ? (size_t)(i0n - 1 - q) * RS + k : 0), ony, -INFINITY);
            }
#pragma unroll
            for (int q = 0; q < 32; q++) {
                tri2[tb ^ 1][q][lane] = v[q];
                etri2[tb ^ 1][q][lane] = __expf(v[q] + R.r[0]);
                xs2[tb ^ 1][q][lane] = y[q];
            }
        } else if (w >= 2) {
            // the block after the next one: its pushes read Lcol rows
            // lo-65 .. lo-34, its in-block terms Lrow rows lo-64 .. lo-33
            prefetch_rows_l2(t.Lcol, RS, L, lo - 65, lo - 34, RS / 32, threadIdx.x - 64, blockDim.x - 64);
            prefetch_rows_l2(t.Lrow, RS, L, lo - 64, lo - 33, 1, threadIdx.x - 64, blockDim.x - 64);
        }
        __syncthreads();
        if (lo == 0) break;
        // push the block [lo, i0] (value u = S cell i0 - u) into the cells
        // lo-1 .. lo-1-Wb; a cell's first push starts it afresh unless the
        // band already gave it terms
        if (w == 0) {
            const int c = lo - 1 - lane;
            cm = -INFINITY;
            cs = 0.f;
            if (c >= nlo) {
                const bool fresh = (c < c_first) && (c + Wb + 1 <= i0);
                if (!fresh) {
                    cm = am[c % win];
                    cs = as[c % win];
                }
#pragma unroll
                for (int u = 0; u < 32; u += 8) {
                    const float y[8] = {x[u] + vals[u], x[u + 1] + vals[u + 1], x[u + 2] + vals[u + 2],
                                        x[u + 3] + vals[u + 3], x[u + 4] + vals[u + 4], x[u + 5] + vals[u + 5],
                                        x[u + 6] + vals[u + 6], x[u + 7] + vals[u + 7]};
                    lse_add8(cm, cs, y);
                }
            }
        } else if (w >= 2) {
            for (int c = nlo - 1 - (threadIdx.x - 64); c >= max(0, lo - 1 - Wb); c -= (int)blockDim.x - 64) {
                const bool fresh = (c < c_first) && (c + Wb + 1 <= i0);
                float m = fresh ? -INFINITY : am[c % win], s = fresh ? 0.f : as[c % win];
                suffix_push_terms(m, s, t.Lcol, RS, i0 - 1, -1, i0 - 1 - c, vals, nb, Wb);
                am[c % win] = m;
                as[c % win] = s;
            }
        }
        tb ^= 1;
        i0 = lo - 1;
        lo = nlo;
    }
}

// Blocks of 32 cells pulled from global memory (bands wider than the
// shared-memory window of the pushing form).
__device__ void inside_suffix_body_pull(const Band& t, const Rules& R)
{
    const int T = t.L - 1 - t.Wb;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    __shared__ float known[32];
    __shared__ float tri[32][33];  // Lrow[i0 - l][k], k < 32: the in-block terms, read by the serial warp
    for (int i0 = T - 1; i0 >= 0; i0 -= 32) {
        const int lo = max(0, i0 - 31);
        for (int q = w; q < 32; q += nw) {  // a warp per cell i0 - q
            const int i = i0 - q;
            tri[q][lane] = (i >= lo && lane <= t.Wb) ? t.Lrow[(size_t)i * t.RS + lane] : -INFINITY;
            if (i < lo) continue;
            float m = -INFINITY, s = 0.f;
            const float* lrow = t.Lrow + (size_t)i * t.RS;
            int k = (i0 - i) + lane;
            for (; k + 96 <= t.Wb; k += 128)
                lse_add4(m, s, lrow[k] + t.Ssuf[i + k + 1], lrow[k + 32] + t.Ssuf[i + k + 33],
                         lrow[k + 64] + t.Ssuf[i + k + 65], lrow[k + 96] + t.Ssuf[i + k + 97]);
            for (; k <= t.Wb; k += 32) lse_add(m, s, lrow[k] + t.Ssuf[i + k + 1]);
            group_reduce<32>(m, s);
            if (lane == 0) known[q] = lse_val(m, s);
        }
        __syncthreads();
        if (w == 0) {
            // column-oriented substitution: lane q owns cell i0 - q; once cell l
            // is final it is broadcast and every later cell adds its term
            const int nb = i0 - lo + 1;
            float am = (lane < nb) ? known[lane] : -INFINITY, as = (am == -INFINITY) ? 0.f : 1.f;
            for (int l = 0; l < nb; l++) {
                const float sv = __shfl_sync(0xffffffffu, R.r[0] + lse_val(am, as), l);
                if (lane == 0) t.Ssuf[i0 - l] = sv;
                const int k = lane - l - 1;
                if (lane > l && lane < nb && k <= t.Wb) lse_add(am, as, tri[lane][k] + sv);
            }
        }
        __syncthreads();
    }
}

__device__ void inside_suffix_any(const Band& t, const Rules& R, float* smem, int win)
{
    if (suffix_window(t.Wb) <= win) inside_suffix_body(t, R, smem, smem + win, win);
    else inside_suffix_body_pull(t, R);
}

// win: cells of the dynamic shared-memory window (2 * win floats)
__global__ void __launch_bounds__(kSuffixThreads) inside_suffix_kernel(Band t, Rules R, int win)
{
    extern __shared__ float suffix_smem[];
    inside_suffix_any(t, R, suffix_smem, win);
}

// one block per alignment of a batch (alignments whose band reaches the last column skip)
__global__ void __launch_bounds__(kSuffixThreads) inside_suffix_batch_kernel(const Band* __restrict__ bands, Rules R,
                                                                           int win)
{
    extern __shared__ float suffix_smem[];
    const Band t = bands[blockIdx.x];
    if (t.L - 1 > t.Wb) inside_suffix_any(t, R, suffix_smem, win);
}

// Window for the largest band that needs a suffix (0: none fits, the pull form runs).
static int suffix_launch_window(const messi_ctx* ctx, int maxWb)
{
    const int win = suffix_window(maxWb);
    return (win <= ctx->suffix_window) ? win : 0;
}

// The window for a batch: the widest band among those that take the pushing
// form (a band too wide for any window takes the pull form in a single call
// too, so both paths give the same bits).
static int suffix_batch_window(const messi_ctx* ctx, const BandBatch& bb)
{
    int win = 0;
    for (const Band& t : bb.host)
        if (t.L - 1 > t.Wb && suffix_window(t.Wb) <= ctx->suffix_window) win = std::max(win, suffix_window(t.Wb));
    return win;
}

__global__ void finish_Z_kernel(Band t)
{
    if (threadIdx.x == 0 && blockIdx.x == 0)
        t.Zd[0] = (t.sync[2] != 0u) ? (double)NAN : (double)t.Ssuf[0] + t.cb[t.L];
}

__global__ void finish_Z_batch_kernel(const Band* __restrict__ bands, int n, const unsigned int* __restrict__ sync,
                                      double* __restrict__ Z)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    const Band& t = bands[b];
    Z[b] = (sync[2] != 0u) ? (double)NAN : (double)t.Ssuf[0] + t.cb[t.L];
}

int launch_finish_Z(messi_ctx* ctx, const Band& t)
{
    finish_Z_kernel<<<1, 32, 0, ctx->stream>>>(t);
    LAUNCH_CHECK(ctx, "finish_Z_kernel");
    return queue_status(ctx, t.sync + 2);
}


// Log-sum-exp over a group of G lanes: the group's maximum by a butterfly,
// one rescale per lane, then a butterfly sum (max and sum are commutative,
// so every lane of the group ends with the same bits) -- about a third of the
// instructions of a pairwise merge per round.
__device__ __forceinline__ void group_reduce_rt(float& m, float& s, int G)
{
    float mx = m;
    for (int off = G >> 1; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    const float base = (mx == -INFINITY) ? 0.f : mx;
    float v = s * __expf(m - base);
    for (int off = G >> 1; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    m = mx;
    s = v;
}

// Span-0 cells of row i.
__device__ __forceinline__ void inside_init_cell(const Band& t, int i, const Rules& R, double B)
{
    const double ui = t.u[i];
    const float S = (ui == -INFINITY) ? -INFINITY : (float)(B * ui + (double)R.r[1] - t.b[i]);
    const float Lv = (ui == -INFINITY) ? -INFINITY : (float)(B * ui + (double)R.r[5] - t.b[i]);
    const size_t o = (size_t)i * t.RS;
    t.Srow[o] = S;
    st_cell(t.Scol + o, S);
    st_cell(t.Lrow + o, Lv);
    t.Lcol[o] = Lv;
    st_cell(t.Frow + o, -INFINITY);
    if (i == t.L - 1) t.Ssuf[i] = S;
}

// Cell (i, i+d) in two parts, by a group of G lanes (every lane of the warp
// calls both, `valid` false for padding groups: the shuffles need the whole
// warp).  The split sum runs over k = 0 .. d-1 of L(i, i+k) + S(i+k+1, j),
// spans k and d-1-k.  The partial part sums the middle split points k =
// NLO .. d-NHI-1 (both spans <= d-1-min(NLO, NHI)), reduces them over the
// group and loads the pair score; the finishing part (lane 0) adds the
// outer split points k < NLO and k >= d-NHI in ascending order, the enclosed
// F (span d-2) and writes the cell.  Odd spans use NLO = NHI = 2, even spans
// 3: the partial sums of a diagonal pair (2p-1, 2p) then read spans <= 2p-4
// only, which the paired wavefront has before its wait, and every kernel
// splits a cell the same way, so all of them give the same bits.
// Sixteen split points of a lane that are all in range (two blocks of eight,
// summed in order): no predicates, and with the group width a constant the
// 32 loads take immediate offsets from two base addresses.  Long spans spend
// most of their points here; the integer pipe (addresses, range checks,
// selects) was the busiest one in the predicated form.
template <int GS>
__device__ __forceinline__ void split_full16(float& m, float& s, const float* lrow, const float* scol, int k)
{
    const float* pa = lrow + k;
    const float* pb = scol - k;
    float a[16], b[16];
#pragma unroll
    for (int q = 0; q < 16; q++) {
        a[q] = __ldcg(pa + q * GS);
        b[q] = __ldcg(pb - q * GS);
    }
    float x0[8], x1[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        x0[q] = a[q] + b[q];
        x1[q] = a[8 + q] + b[8 + q];
    }
    lse_add8(m, s, x0);
    lse_add8(m, s, x1);
}

// The last rem points (1..16) of a lane at G = 32, in one or two blocks of
// eight (TWO), summed in order: predicated loads at constant offsets from two
// base addresses, the absent points -inf.  Most of a lane's points on bands
// up to 800 wide fall here (at most 25 per lane).
template <bool TWO>
__device__ __forceinline__ void split_tail32(float& m, float& s, const float* lrow, const float* scol, int k,
                                             int rem)
{
    constexpr int NQ = TWO ? 16 : 8;
    const float* pa = lrow + k;
    const float* pb = scol - k;
    float a[NQ], b[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) {
        const bool on = q < rem;
        a[q] = ldcg_if(pa + q * 32, on, -INFINITY);
        b[q] = ldcg_if(pb - q * 32, on, -INFINITY);
    }
    float x0[8];
#pragma unroll
    for (int q = 0; q < 8; q++) x0[q] = a[q] + b[q];
    lse_add8(m, s, x0);
    if (TWO) {
        float x1[8];
#pragma unroll
        for (int q = 0; q < 8; q++) x1[q] = a[(8 + q) % NQ] + b[(8 + q) % NQ];
        lse_add8(m, s, x1);
    }
}

// Split points k = e .. d-e-1 of cell (i, i+d), its L row and S column given
// (scol at span d-1), reduced over the group; lane 0 of the group has the sum.
__device__ __forceinline__ void cell_partial(const float* lrow, const float* scol, int d, int e, bool valid, int lane,
                                             int G, float& m, float& s)
{
    m = -INFINITY;
    s = 0.f;
    const int kend = d - e;
    if (valid && kend > e) {
        // blocks of eight split points per lane, summed in order; while a lane
        // has more than eight points left, two blocks' 32 loads are issued
        // together (one L2 round trip for sixteen points: long spans have up
        // to 63 points per lane).  Points past the end are -inf, which
        // lse_add8 skips exactly.
        int k = e + lane;
        if (G == 32) {  // warp-uniform: one cell per warp, constant strides
            for (; k + 15 * 32 < kend; k += 16 * 32) split_full16<32>(m, s, lrow, scol, k);
            const int rem = (kend - k + 31) / 32;  // points left (<= 0: none)
            if (rem > 8) split_tail32<true>(m, s, lrow, scol, k, rem);
            else if (rem > 0) split_tail32<false>(m, s, lrow, scol, k, rem);
        } else {
            for (; k < kend; k += 8 * G) {
                float x[8];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const int kq = k + q * G;
                    const bool on = kq < kend;
                    x[q] = ldcg_if(lrow + kq, on, -INFINITY) + ldcg_if(scol - kq, on, -INFINITY);
                }
                lse_add8(m, s, x);
            }
        }
    }
    // the shuffles only where some lane group of the warp has a cell
    if (__any_sync(0xffffffffu, valid)) group_reduce_rt(m, s, G);
}

// Operands of a cell's outer split points, k < N and k >= hb = max(N, d-N) in
// ascending k: L(i, i+k) and S(i+k+1, j), both -inf where the split point is
// absent (an absent term is then -inf, which lse_add8 skips exactly), and the
// enclosed F(i+1, j-1).  With N = 3 (even spans) L(i, i+d-1) and S(i+1, j), the
// two operands on diagonal d-1, are left to outer_patch.
template <int N>
struct Outer {
    float l[2 * N], s[2 * N], fin;
    __device__ __forceinline__ bool complete() const
    {
        bool ok = !unwritten(fin);
#pragma unroll
        for (int q = 0; q < 2 * N; q++) ok = ok && !unwritten(l[q]) && !unwritten(s[q]);
        return ok;
    }
};

template <int N>
__device__ __forceinline__ void outer_load(const Band& t, int i, int d, Outer<N>& o)
{
    const float* lrow = t.Lrow + (size_t)i * t.RS;
    const float* scol = t.Scol + (size_t)(i + d) * t.RS + (d - 1);
    const int hb = max(N, d - N);
#pragma unroll
    for (int q = 0; q < 2 * N; q++) {
        const int k = (q < N) ? q : hb + (q - N);
        o.l[q] = o.s[q] = -INFINITY;
        if (k < d && !(N == 3 && k == d - 1)) o.l[q] = ld_cell(lrow + k);
        if (k < d && !(N == 3 && q == 0)) o.s[q] = ld_cell(scol - k);
    }
    o.fin = -INFINITY;
    if (d >= 2) o.fin = ld_cell(t.Frow + (size_t)(i + 1) * t.RS + (d - 2));
}

// The same once every operand is there, for the whole warp; false if that took too long.
template <int N>
__device__ __forceinline__ bool outer_wait(const Band& t, int i, int d, bool mine, Outer<N>& o, unsigned int* sync)
{
    unsigned int spins = 0;
    for (;;) {
        if (mine) outer_load<N>(t, i, d, o);
        mine = mine && !o.complete();
        if (!__any_sync(0xffffffffu, mine)) return true;
        if (!warp_keep_waiting(spins, sync)) return false;
    }
}

__device__ __forceinline__ void outer_patch(Outer<3>& o, int d, float l_last, float s_first)
{
    const int hb = max(3, d - 3);
#pragma unroll
    for (int q = 0; q < 6; q++)
        if (((q < 3) ? q : hb + (q - 3)) == d - 1) o.l[q] = l_last;
    o.s[0] = s_first;
}

// Adds the outer split points to the partial sum (m, s) and writes cell
// (i, i+d); returns its L and S.  pbv: the pair's score.
template <int N>
__device__ __forceinline__ float2 cell_write(const Band& t, int i, int d, float m, float s, float pbv,
                                             const Outer<N>& o, const Rules& R)
{
    const int RS = t.RS;
    const int j = i + d;
    // the outer split points as one block (one max, independent exponentials:
    // this is the serial part of a cell after the wait)
    float x[8];
#pragma unroll
    for (int q = 0; q < 8; q++) x[q] = (q < 2 * N) ? o.l[q % (2 * N)] + o.s[q % (2 * N)] : -INFINITY;
    lse_add8(m, s, x);
    const float tmp = lse_val(m, s);
    const float v = pbv + o.fin;
    const float S = lse2f(R.r[0] + tmp, R.r[2] + v);
    const float F = lse2f(R.r[4] + tmp, R.r[3] + v);
    const float Lv = R.r[6] + v;
    st_cell(t.Lrow + (size_t)i * RS + d, Lv);
    st_cell(t.Scol + (size_t)j * RS + d, S);
    st_cell(t.Frow + (size_t)i * RS + d, F);
    t.Lcol[(size_t)j * RS + d] = Lv;
    t.Srow[(size_t)i * RS + d] = S;
    if (j == t.L - 1) t.Ssuf[i] = S;
    return make_float2(Lv, S);
}

// Band of the batch with span d or more: bands are sorted by width, descending.
__device__ __forceinline__ int batch_active(const int* __restrict__ wbs, int n, int d)
{
    int lo = 0, hi = n;  // first band with Wb < d
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(wbs + mid) >= d) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ int batch_band(const long long* __restrict__ cumL, int nact, int d, long long item)
{
    int lo = 0, hi = nact - 1;  // last band b with cumL[b] - d*b <= item
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(cumL + mid) - (long long)d * mid <= item) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

constexpr int kInsideThreads = 512;       // 128 registers a thread
constexpr int kInsideManyThreads = 768;   // 80
constexpr int kInsideManyRows = 16;       // cells of a diagonal per CTA from which on there are so many threads
constexpr int kInsideFinish = 64;  // threads that finish each diagonal of a pair
constexpr int kInsideCells = 512;  // cells of a diagonal that a CTA takes at a time

// The bands of an inside launch: one (t) or a batch of n, whose cells of
// diagonal d, flattened in band order, start at cumL[b] - d*b for band b.
template <bool BATCH>
struct InsideBands {
    Band t;
    const Band* bands;
    const long long* cumL;
    const int* wbs;
    int n;
    __device__ __forceinline__ const Band& at(int b) const { return BATCH ? bands[b] : t; }
};

// The cells of diagonal d (the pair's odd one) that this CTA owns: [f0, f0 +
// nb) of the flattened list; of the odd diagonal also the one after them
// (na = nb + 1, unless the list ends there).
struct PairRows {
    long long f0;
    int nact, na, nb;
};

template <bool BATCH>
__device__ __forceinline__ PairRows pair_rows(const InsideBands<BATCH>& ib, int d)
{
    PairRows p;
    p.nact = BATCH ? batch_active(ib.wbs, ib.n, d) : 1;
    const long long ncell = BATCH ? __ldg(ib.cumL + p.nact) - (long long)d * p.nact : ib.t.L - d;
    const int rows = (int)(((unsigned)ncell + gridDim.x - 1) / gridDim.x);
    p.f0 = (long long)blockIdx.x * rows;
    const long long left = ncell - p.f0;
    p.nb = (int)max(0ll, min((long long)rows, left));
    p.na = (int)max(0ll, min((long long)rows + 1, left));
    return p;
}

template <bool BATCH>
__device__ __forceinline__ int2 pair_cell(const InsideBands<BATCH>& ib, const PairRows& p, int d, int r)
{
    if (!BATCH) return make_int2(0, (int)p.f0 + r);
    const int b = batch_band(ib.cumL, p.nact, d, p.f0 + r);
    return make_int2(b, (int)(p.f0 + r - (__ldg(ib.cumL + b) - (long long)d * b)));
}

// All band diagonals of the inside pass (of one alignment, or of a batch: one
// diagonal of every alignment at a time), in pairs (d = 2p-1, d+1).  The cells
// of a pair are dealt evenly over the CTAs, pair by pair.  A CTA finishes
// diagonal d for its cells and the next CTA's first one (which that CTA also
// computes, to the same bits) and then diagonal d+1, whose cells read diagonal
// d only at rows i and i+1, its own.
// Four warps finish the cells, a thread per cell and two warps per diagonal:
// they add the outer split points and write the cells.  The other warps
// meanwhile form the partial sums of the next pair, which read spans <= d-1, and
// leave them in shared memory: the sums are off the critical path, and a
// finishing lane does not idle the rest of its warp.
// The CTAs wait for one another's cells, not at a barrier: the tables are
// filled with kUnwritten before the launch and a cell is its own flag (a grid
// barrier's release alone took 2,100 cycles of a pair's 4,900: every store has
// to be acknowledged before the arrival).  The finishing threads look at their
// operands until all are there.  Those are spans d-1 and d-2, and what the other
// warps read for the pair p+1 was written before them by the same chain of
// CTAs, so a partial sum hardly ever meets an unwritten cell; it would be NaN,
// and is then formed again once its cells are there.
// Bound by the chain write -> look from L2 -> cells of d -> cells of d+1, about
// 1.7 us a pair, and on long bands by the latency of the partial sums' loads.
// Against one grid barrier per pair with every warp summing and then finishing
// its own cell: span 500 of 1,000 columns 0.74 -> 0.49 ms, every span of 120
// 154 -> 93 us and of 2,001 5.18 -> 3.39 ms, span 800 of 9,000 4.82 -> 4.70 ms;
// 24 alignments of 80-600 columns, with a barrier per diagonal before, 3.23 ->
// 1.23 ms.
template <bool BATCH, int MAXT>
__global__ void __launch_bounds__(MAXT) inside_pair_kernel(InsideBands<BATCH> ib, Rules R, double B,
                                                                      unsigned int* sync)
{
    __shared__ float2 part[2][2][kInsideCells + 1];  // [pair parity][diagonal][cell]: partial (max, sum)
    __shared__ float score[2][2][kInsideCells + 1];  // and the pair's score
    __shared__ float2 last[kInsideCells + 1];        // L and S of diagonal d
    __shared__ int2 cells[2][BATCH ? kInsideCells + 1 : 1];
    __shared__ PairRows rows[2];
    const int tid = threadIdx.x, nwork = (int)blockDim.x - 2 * kInsideFinish;
    const bool fin = tid < 2 * kInsideFinish;
    const int maxW = BATCH ? (ib.n > 0 ? ib.wbs[0] : 0) : ib.t.Wb;
    bool bad = false;      // a wait of this thread took too long
    bool own_nan = false;  // this warp has met a NaN that was no unwritten cell
    for (long long it = blockIdx.x * (long long)blockDim.x + tid; it < (BATCH ? ib.cumL[ib.n] : ib.t.L);
         it += (long long)gridDim.x * blockDim.x) {
        const int b = BATCH ? batch_band(ib.cumL, ib.n, 0, it) : 0;
        inside_init_cell(ib.at(b), (int)(BATCH ? it - ib.cumL[b] : it), R, B);
    }

    // A partial sum came out NaN: again, until the cells are there.  After 64
    // times (or once that has been the case) the cells are looked at one by one;
    // a NaN of written cells is the scores' own.
    auto again = [&](const float* lrow, const float* scol, int dd, int e, bool valid, int lane, int G, float& m,
                     float& s) {
        unsigned int spins = 0;
        for (bool there = false; !there;) {
            bad = !warp_keep_waiting(spins, sync) || bad;
            if (bad) break;
            if (own_nan || (spins & 63u) == 0u) {
                bool missing = false;
                if (valid)
                    for (int k = e + lane; k < dd - e; k += G)
                        missing = missing || unwritten(ld_cell(lrow + k)) || unwritten(ld_cell(scol - k));
                there = !__any_sync(0xffffffffu, missing);
                own_nan = own_nan || there;
            }
            asm volatile("" : "+l"(lrow), "+l"(scol)::"memory");  // not the cells read before
            cell_partial(lrow, scol, dd, e, valid, lane, G, m, s);
            if (!__any_sync(0xffffffffu, valid && s != s)) break;
        }
    };

    // partial sums of cells [c0, c0 + kInsideCells) of the pair (d, d+1), by the other warps
    auto partials = [&](const PairRows& p, int d, int c0, int buf) {
        const int na = min(kInsideCells + 1, p.na - c0), nb = min(kInsideCells, p.nb - c0);
        const int wt = tid - 2 * kInsideFinish;
        if (BATCH) {
            for (int r = wt; r < na; r += nwork) cells[buf][r] = pair_cell(ib, p, d, c0 + r);
            asm volatile("bar.sync 2, %0;" ::"r"(nwork) : "memory");
        }
        if (c0 == 0) {
            if (wt == 0) rows[buf] = p;
            asm volatile("bar.arrive 3, %0;" ::"r"(nwork + 2 * kInsideFinish) : "memory");
        }
        const int G = group_width(d);  // of both diagonals: the limits are even, d is odd
        const int gpb = nwork / G, lane = wt & (G - 1);
        // Sum w of the pair: of cell r of diagonal dd, its L row and S column.
        struct Item {
            const float *lrow, *scol;
            int r, dd;
            float pbv;
            bool valid;
        };
        auto item = [&](int w) {
            Item q;
            const int x = w >= na ? 1 : 0;
            q.r = x ? w - na : w;
            q.dd = d + x;
            q.valid = w < na + nb;
            const int2 c = BATCH ? cells[buf][q.valid ? q.r : 0] : make_int2(0, (int)p.f0 + c0 + q.r);
            const Band& t = ib.at(c.x);
            q.valid = q.valid && c.y + q.dd < t.L && q.dd <= t.Wb;
            q.lrow = t.Lrow + (size_t)c.y * t.RS;
            q.scol = t.Scol + (size_t)(c.y + q.dd) * t.RS + (q.dd - 1);
            q.pbv = (q.valid && lane == 0 && q.dd >= 2) ? __ldg(t.pb + (size_t)c.y * t.RS + q.dd) : -INFINITY;
            return q;
        };
        // A cell's sum is formed (m, s): kept, unless it is NaN for cells that
        // were not there yet.
        auto keep = [&](const Item& q, float m, float s) {
            if (__any_sync(0xffffffffu, q.valid && s != s)) again(q.lrow, q.scol, q.dd, 2 + (q.dd - d), q.valid, lane, G, m, s);
            if (q.valid && lane == 0) {
                part[buf][q.dd - d][q.r] = make_float2(m, s);
                score[buf][q.dd - d][q.r] = q.pbv;
            }
        };
        if (G < 32 || MAXT > kInsideThreads) {
            for (int base = 0; base < na + nb; base += gpb) {
                const Item q = item(base + wt / G);
                float m, s;
                cell_partial(q.lrow, q.scol, q.dd, 2 + (q.dd - d), q.valid, lane, G, m, s);
                keep(q, m, s);
            }
            return;
        }
        // A warp per cell: sixteen split points of a lane at a time, the loads
        // of the next sixteen (of this cell or the warp's next one) in flight
        // meanwhile (span 500 of 1,000 columns: 537 -> 511 us, the batch of 24
        // 1.37 -> 1.23 ms).
        auto load = [&](const Item& q, int k, float (&a)[16], float (&b)[16]) {
            // (sixteen that all 32 lanes have go without predicates: span 500 of
            // 1,000 columns 520 -> 489 us, L = 2,001 3.81 -> 3.39 ms)
            const int left = q.valid ? q.dd - 2 - (q.dd - d) - (k - lane) : 0;  // split points from here on
            const float* pa = q.lrow + k;
            const float* pb = q.scol - k;
            if (left >= 512) {
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    a[j] = __ldcg(pa + j * 32);
                    b[j] = __ldcg(pb - j * 32);
                }
                return;
            }
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const bool on = j * 32 + lane < left;
                a[j] = ldcg_if(pa + j * 32, on, -INFINITY);
                b[j] = ldcg_if(pb - j * 32, on, -INFINITY);
            }
        };
        int w = wt >> 5;
        if (w >= na + nb) return;
        Item q = item(w);
        int k = 2 + (q.dd - d) + lane;
        float a[16], b[16], m = -INFINITY, s = 0.f;
        load(q, k, a, b);
        for (bool next = true; next;) {
            float x0[8], x1[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                x0[j] = a[j] + b[j];
                x1[j] = a[8 + j] + b[8 + j];
            }
            const Item now = q;
            const int left = now.valid ? now.dd - 2 - (now.dd - d) - (k - lane) : 0;  // split points from here on
            const bool more = left > 512;                                               // of this cell, after these
            next = more || w + gpb < na + nb;
            if (more) {
                k += 512;
            } else if (next) {
                q = item(w += gpb);
                k = 2 + (q.dd - d) + lane;
            }
            if (next) load(q, k, a, b);
            lse_add8(m, s, x0);
            if (left > 256) lse_add8(m, s, x1);
            if (!more) {
                group_reduce_rt(m, s, 32);
                keep(now, m, s);
                m = -INFINITY;
                s = 0.f;
            }
        }
    };

    // The cells [c0, c0 + kInsideCells) of diagonal dd = d + N - 2, by a thread
    // each of 64; `ready`: what to do between the first cells' operands and the rest.
    auto finish = [&](auto width, const PairRows& p, int d, int c0, int buf, auto ready) {
        constexpr int N = decltype(width)::value;
        const int x = N - 2, dd = d + x, n = x ? min(kInsideCells, p.nb - c0) : min(kInsideCells + 1, p.na - c0);
        const int first = tid & (kInsideFinish - 1);
        for (int r = first; r - (first & 31) < n || r == first; r += kInsideFinish) {
            bool mine = r < n;
            int2 c = make_int2(0, 0);
            if (mine) c = (BATCH && c0 == 0) ? cells[buf][r] : pair_cell(ib, p, d, c0 + r);
            const Band& t = ib.at(c.x);
            mine = mine && c.y + dd < t.L && dd <= t.Wb;
            Outer<N> o;
            bad = !outer_wait<N>(t, c.y, dd, mine, o, sync) || bad;
            if (r == first) ready();
            if (!mine) continue;
            if constexpr (N == 3) outer_patch(o, dd, last[r].x, last[r + 1].y);
            const float2 ms = part[buf][x][r];
            const float2 ls = cell_write<N>(t, c.y, dd, ms.x, ms.y, score[buf][x][r], o, R);
            if constexpr (N == 2) last[r] = ls;
        }
    };
    auto inside_barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(2 * kInsideFinish) : "memory"); };

    int buf = 0;
    if (!fin && maxW > 0) partials(pair_rows(ib, 1), 1, 0, 0);
    for (int d = 1; d <= maxW; d += 2, buf ^= 1) {
        PairRows p;
        bool stop = false;
        // every thread: the pair's partial sums are there, and its operands
        auto together = [&] { stop = __syncthreads_or(bad) != 0; };
        if (fin) {
            asm volatile("bar.sync 3, %0;" ::"r"(nwork + 2 * kInsideFinish) : "memory");
            p = rows[buf];
            if (tid < kInsideFinish) {
                finish(std::integral_constant<int, 2>{}, p, d, 0, buf, together);
                inside_barrier();
            } else {
                finish(std::integral_constant<int, 3>{}, p, d, 0, buf, [&] {
                    together();
                    inside_barrier();  // diagonal d of this CTA's cells is in `last`
                });
            }
        } else {
            together();
            p = rows[buf];
            if (!stop && d + 2 <= maxW) partials(pair_rows(ib, d + 2), d + 2, 0, buf ^ 1);
        }
        // more cells than a CTA holds: the rest apart
        for (int c0 = kInsideCells; c0 < p.nb; c0 += kInsideCells) {
            __syncthreads();
            if (!fin) partials(p, d, c0, buf);
            __syncthreads();
            if (tid < kInsideFinish) {
                finish(std::integral_constant<int, 2>{}, p, d, c0, buf, [] {});
                inside_barrier();
            } else if (fin) {
                finish(std::integral_constant<int, 3>{}, p, d, c0, buf, inside_barrier);
            }
        }
        if (stop) return;
    }
}

// Outside cell (i, j = i+d): the parent sums run over q of OS/OF(i, j+1+q) *
// S(j+1, j+1+q) (side 0, "L") and of OS/OF(i-1-q, j) * L(i-1-q, i-1) (side
// 1, "S"), spans d+1+q.  Each sum is computed apart: q >= Q and the
// suffix-column terms by a lane group (outside_sum, reduced over the group),
// then q = 0 .. Q-1 in ascending order by one thread (near_finish); the F value
// comes from the enclosing pair (i-1, j+1) (span d+2).  Diagonals go in pairs
// (e, e-1), with Q = 2 for e and Q = 3 for e-1: the sums then read spans >= e+3
// only, which are complete when the finishing threads have the operands of the
// pair before, (e+2, e+1).  A cell's bits depend only on its span (the group
// width), not on which CTA, warp or thread computes it.

// Parents q < n of one sum: OS and OF at o1[q], o2[q], the inside factor at
// in[q]; extra: the suffix column's part.
struct SumArgs {
    const float *o1, *o2, *in;
    int n;
    float extra;
};

__device__ __forceinline__ SumArgs sum_args(const Band& t, int i, int d, int side, bool first, const Rules& R)
{
    const int L = t.L, Wb = t.Wb, RS = t.RS, j = i + d;
    SumArgs a;
    a.extra = -INFINITY;
    if (side == 0) {
        const bool has = j + 1 <= L - 1;
        a.n = has ? min(i + Wb, L - 1) - j : 0;
        a.o1 = t.OSrow + (size_t)i * RS + d + 1;
        a.o2 = t.OFrow + (size_t)i * RS + d + 1;
        a.in = t.Srow + (size_t)min(j + 1, L - 1) * RS;
        if (first && has && L - 1 > i + Wb) a.extra = R.r[0] + __ldcg(t.Osuf + i) + t.Ssuf[j + 1];
    } else {
        const bool has = i >= 1;
        a.n = has ? i - max(0, j - Wb) : 0;
        a.o1 = t.OScol + (size_t)j * RS + d + 1;
        a.o2 = t.OFcol + (size_t)j * RS + d + 1;
        a.in = t.Lcol + (size_t)max(i - 1, 0) * RS;
        // the last column's parents beyond the band, summed before the launch
        if (first && has && j == L - 1) a.extra = t.OSlast[i];
    }
    return a;
}

// Eight points of one sum that are all in range (two blocks of four points,
// eight terms each, summed in order): no range checks, and with the group
// width a constant the 24 loads take immediate offsets.
template <int GS>
__device__ __forceinline__ void outside_full8(float& m, float& s, const float* o1, const float* o2, const float* in,
                                              int q, const Rules& R)
{
    const float* p1 = o1 + q;
    const float* p2 = o2 + q;
    const float* p3 = in + q;
    float a[8], b[8], v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
        a[u] = __ldcg(p1 + u * GS);
        b[u] = __ldcg(p2 + u * GS);
        v[u] = p3[u * GS];
    }
    float x0[8], x1[8];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        x0[2 * u] = R.r[0] + a[u] + v[u];
        x0[2 * u + 1] = R.r[4] + b[u] + v[u];
        x1[2 * u] = R.r[0] + a[4 + u] + v[4 + u];
        x1[2 * u + 1] = R.r[4] + b[4 + u] + v[4 + u];
    }
    lse_add8(m, s, x0);
    lse_add8(m, s, x1);
}

__device__ __forceinline__ float2 outside_sum(const SumArgs& g, int Q, bool valid, int lane, int G, const Rules& R)
{
    float m = -INFINITY, s = 0.f;
    if (!__any_sync(0xffffffffu, valid)) return make_float2(m, s);  // no cell in this warp (warp-uniform)
    if (valid) {
        const int n = g.n;
        int q = Q + lane;
        if (G == 32) {  // warp-uniform: one sum per warp, constant strides
            for (; q + 7 * 32 < n; q += 8 * 32) outside_full8<32>(m, s, g.o1, g.o2, g.in, q, R);
            const int rem = (n - q + 31) / 32;  // points left (0..7)
            if (rem > 0) {
                const float* p1 = g.o1 + q;
                const float* p2 = g.o2 + q;
                const float* p3 = g.in + q;
                float x0[8], x1[8];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const bool on = u < rem;
                    const float v = ldg_if(p3 + u * 32, on, 0.f);
                    const float a = ldcg_if(p1 + u * 32, on, -INFINITY);
                    const float b = ldcg_if(p2 + u * 32, on, -INFINITY);
                    float* x = (u < 4) ? x0 : x1;
                    x[2 * (u & 3)] = R.r[0] + a + v;
                    x[2 * (u & 3) + 1] = R.r[4] + b + v;
                }
                lse_add8(m, s, x0);
                lse_add8(m, s, x1);
            }
            q = n;
        }
        for (; q < n; q += 8 * G) {
            float x0[8], x1[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int qq = q + u * G;
                const bool on = qq < n;
                const float v = ldg_if(g.in + qq, on, 0.f);
                const float a = ldcg_if(g.o1 + qq, on, -INFINITY);
                const float b = ldcg_if(g.o2 + qq, on, -INFINITY);
                float* x = (u < 4) ? x0 : x1;
                x[2 * (u & 3)] = R.r[0] + a + v;
                x[2 * (u & 3) + 1] = R.r[4] + b + v;
            }
            lse_add8(m, s, x0);
            lse_add8(m, s, x1);
        }
        lse_add(m, s, g.extra);
    }
    group_reduce_rt(m, s, G);
    return make_float2(m, s);
}

// Parents 0 .. Q-1 of one sum.
template <int Q>
struct NearSum {
    float a[Q], b[Q], v[Q];
    __device__ __forceinline__ bool complete() const
    {
        bool ok = true;
#pragma unroll
        for (int q = 0; q < Q; q++) ok = ok && !unwritten(a[q]) && !unwritten(b[q]);
        return ok;
    }
};

// Q = 3 (diagonal e-1): parent 0, on diagonal e, comes from shared memory.
template <int Q>
__device__ __forceinline__ void near_load(const SumArgs& g, NearSum<Q>& s)
{
#pragma unroll
    for (int q = 0; q < Q; q++) {
        s.v[q] = 0.f;
        s.a[q] = s.b[q] = -INFINITY;
        if (q < g.n) {
            s.v[q] = __ldg(g.in + q);
            if (Q == 2 || q > 0) {
                s.a[q] = ld_cell(g.o1 + q);
                s.b[q] = ld_cell(g.o2 + q);
            }
        }
    }
}

template <int Q>
__device__ __forceinline__ float near_finish(const NearSum<Q>& s, float2 c, const Rules& R)
{
    float x[8];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const bool on = q < Q;
        const int qq = on ? q : 0;
        x[2 * q] = on ? R.r[0] + s.a[qq] + s.v[qq] : -INFINITY;
        x[2 * q + 1] = on ? R.r[4] + s.b[qq] + s.v[qq] : -INFINITY;
    }
    lse_add8(c.x, c.y, x);
    return lse_val(c.x, c.y);
}

struct FOperands {
    float pp, a, b, c;
    __device__ __forceinline__ bool complete() const { return !unwritten(a) && !unwritten(b) && !unwritten(c); }
};

__device__ __forceinline__ void f_load(const Band& t, int i, int d, FOperands& f)
{
    f = FOperands{-INFINITY, -INFINITY, -INFINITY, -INFINITY};
    if (i < 1 || i + d > t.L - 2 || d + 2 > t.Wb) return;
    const size_t pr = (size_t)(i - 1) * t.RS + d + 2;
    f = FOperands{__ldg(t.pb + pr), ld_cell(t.OSrow + pr), ld_cell(t.OFrow + pr), ld_cell(t.OLrow + pr)};
}

__device__ __forceinline__ float f_finish(const FOperands& f, const Rules& R)
{
    if (f.pp == -INFINITY) return -INFINITY;
    float m = -INFINITY, s = 0.f;
    lse_add4(m, s, R.r[2] + f.pp + f.a, R.r[3] + f.pp + f.b, R.r[6] + f.pp + f.c, -INFINITY);
    return lse_val(m, s);
}

// Writes the finished value of a sum (side 0: OL, side 1: OS); returns it.
__device__ __forceinline__ float sum_write(const Band& t, int i, int d, int side, float v)
{
    const int j = i + d;
    if (side == 0) {
        st_cell(t.OLrow + (size_t)i * t.RS + d, v);
        return v;
    }
    if (i == 0 && j == t.L - 1) v = 0.f;
    st_cell(t.OSrow + (size_t)i * t.RS + d, v);
    st_cell(t.OScol + (size_t)j * t.RS + d, v);
    if (j == t.L - 1) t.Osuf[i] = v;
    return v;
}

__device__ __forceinline__ void f_write(const Band& t, int i, int d, float v)
{
    st_cell(t.OFrow + (size_t)i * t.RS + d, v);
    st_cell(t.OFcol + (size_t)(i + d) * t.RS + d, v);
}

// Suffix-column terms of the outside S sums of the last column's band cells:
// cell (i, L-1) has the parents (ip, L-1) beyond the band, ip = max(0, i-1-Wb)
// .. L-2-Wb, each adding r1 + OS(ip, L-1) + L(ip, i-1).  They read only the
// suffix column and the inside tables, so one launch before the wavefront
// sums them for every row, a warp per row: inside the wavefront the cell of
// diagonal d has d+1 of them, summed by the single lane group of a long
// diagonal while every other CTA waited.
__global__ void outside_lastcol_kernel(Band t, Rules R)
{
    const int L = t.L, Wb = t.Wb, RS = t.RS;
    const int lane = threadIdx.x & 31;
    const int i = max(1, L - 1 - Wb) + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (i > L - 1) return;  // warp-uniform
    const int a = max(0, i - 1 - Wb), bnd = min(i - 1, L - 2 - Wb);
    const float* lcol = t.Lcol + (size_t)(i - 1) * RS;
    float m = -INFINITY, s = 0.f;
    for (int ip = a + lane; ip <= bnd; ip += 256) {
        float x[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int iq = ip + 32 * q;
            x[q] = (iq <= bnd) ? R.r[0] + t.Osuf[iq] + lcol[i - 1 - iq] : -INFINITY;
        }
        lse_add8(m, s, x);
    }
    group_reduce<32>(m, s);
    if (lane == 0) t.OSlast[i] = lse_val(m, s);
}

constexpr int kOutsideFinish = 128;   // threads that finish a pair: two warps per diagonal
constexpr int kOutsideRows = 256;     // rows of a diagonal that a CTA takes at a time

// All band diagonals of the outside pass, descending spans, in pairs (e, e-1).
// The rows of a pair are dealt evenly over the CTAs, pair by pair: a CTA owns
// rows [r0, r0 + nb) of diagonal e-1 and finishes diagonal e for rows r0 - 1 ..
// r0 + nb - 1 (row r0 - 1 is computed by the previous CTA too, to the same
// bits): a cell of e-1 reads diagonal e only at rows i and i-1.
// As in the inside pass, the CTAs wait for one another's cells (the five tables
// are filled with kUnwritten before the launch) and four warps finish a pair
// while the others form the sums of the next one.  Of the four, warps 0 and 2
// take the two near sums of the rows of e and e-1, two lanes a row, warps 1 and
// 3 their F values; what e-1 needs of e comes through shared memory.
// Against one grid barrier per pair: span 500 over 1,000 columns 1.41 -> 1.07 ms,
// 300 over 600 0.81 -> 0.44, every span of 300 611 -> 308 us, span 500 over
// 3,000 columns 4.51 -> 2.29 ms.  Bound by the sums (24 loads and 16
// exponentials of a lane per L2 round trip); with few rows by the chain write
// -> look -> cells of e -> cells of e-1, as the inside pass.
template <int MAXT>
__global__ void __launch_bounds__(MAXT) outside_pair_kernel(Band t, Rules R, unsigned int* sync)
{
    __shared__ float2 part[2][2][2 * (kOutsideRows + 1)];  // [pair parity][diagonal][2 row + side]
    __shared__ float oS[kOutsideRows + 1], oF[kOutsideRows + 1];
    const int tid = threadIdx.x, nwork = (int)blockDim.x - kOutsideFinish;
    const bool fin = tid < kOutsideFinish;
    const int L = t.L, Wb = t.Wb, grid = (int)gridDim.x;
    bool bad = false;      // a wait of this thread took too long
    bool own_nan = false;  // this warp has met a NaN that was no unwritten cell
    int rows = 1;
    struct Pair {
        int r0, na, nb;  // rows r0 - 1 .. of diagonal e (row -1 is none), r0 .. of diagonal e - 1
    };
    auto pair_at = [&](int e) {  // e descending: the rows grow
        const int most = L - max(e - 1, 0);
        rows = max(rows, (most + grid - 1) / grid);
        Pair p;
        p.r0 = blockIdx.x * rows;
        const int nr = max(min(rows, most - p.r0), 0);
        p.na = nr > 0 ? min(p.r0 + rows, L - e) - (p.r0 - 1) : 0;
        p.nb = e >= 1 ? nr : 0;
        return p;
    };

    // the sums of rows [c0, c0 + kOutsideRows) of the pair (e, e-1), by the other warps
    auto sums = [&](const Pair& p, int e, int c0, int buf) {
        const int na = min(kOutsideRows + 1, p.na - c0), nb = max(min(kOutsideRows, p.nb - c0), 0);
        const int wt = tid - kOutsideFinish;
        const int G = group_width(2 * (Wb - e) + 2);  // of both: the limits are multiples of four
        const int gpb = nwork / G, lane = wt & (G - 1);
        for (int base = 0; base < 2 * (na + nb); base += gpb) {
            const int w = base + wt / G;
            const int x = w >= 2 * na ? 1 : 0, tau = x ? w - 2 * na : w, d = e - x;
            const int i = p.r0 - 1 + x + c0 + (tau >> 1);
            const bool valid = w < 2 * (na + nb) && i >= 0;
            SumArgs g{nullptr, nullptr, nullptr, 0, -INFINITY};
            if (valid) g = sum_args(t, i, d, tau & 1, lane == 0, R);
            unsigned int spins = 0;
            float2 c;
            for (bool there = false;;) {
                c = outside_sum(g, 2 + x, valid, lane, G, R);
                if (there || !__any_sync(0xffffffffu, valid && c.y != c.y)) break;
                // a NaN: again, as in the inside pass
                bad = !warp_keep_waiting(spins, sync) || bad;
                if (bad) break;
                if (own_nan || (spins & 63u) == 0u) {
                    bool missing = false;
                    for (int q = 2 + x + lane; q < g.n; q += G)
                        missing = missing || unwritten(ld_cell(g.o1 + q)) || unwritten(ld_cell(g.o2 + q));
                    there = !__any_sync(0xffffffffu, missing);
                    own_nan = own_nan || there;
                }
                asm volatile("" : "+l"(g.o1), "+l"(g.o2)::"memory");  // not the cells read before
            }
            if (valid && lane == 0) part[buf][x][tau] = c;
        }
    };

    auto fin_barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(kOutsideFinish) : "memory"); };
    // until the warp's operands are there
    auto await = [&](bool mine, auto load, auto complete) {
        for (unsigned int spins = 0;;) {
            if (mine) load();
            mine = mine && !complete();
            if (!__any_sync(0xffffffffu, mine)) return;
            if (!warp_keep_waiting(spins, sync)) {
                bad = true;
                return;
            }
        }
    };
    // The near sums (a lane per side) or F values of diagonal d = e - Q + 2 for
    // its rows [c0, c0 + kOutsideRows); `ready`: what to do between the first
    // rows' operands and the rest.
    auto finish_sums = [&](auto parents, const Pair& p, int e, int c0, int buf, auto ready) {
        constexpr int Q = decltype(parents)::value;
        const int x = Q - 2, d = e - x, n = x ? min(kOutsideRows, p.nb - c0) : min(kOutsideRows + 1, p.na - c0);
        const int side = tid & 1;
        for (int base = 0; base < n || base == 0; base += 16) {
            const int r = base + ((tid & 31) >> 1), i = p.r0 - 1 + x + c0 + r;
            const bool mine = r < n && i >= 0;
            SumArgs g{nullptr, nullptr, nullptr, 0, -INFINITY};
            if (mine) g = sum_args(t, i, d, side, false, R);
            NearSum<Q> s;
            await(mine, [&] { near_load<Q>(g, s); }, [&] { return s.complete(); });
            if (base == 0) ready();
            if (!mine) continue;
            if constexpr (Q == 3) {
                if (g.n > 0) {  // parent 0: (i, j+1) for side 0 and (i-1, j) for side 1
                    s.a[0] = oS[r + 1 - side];
                    s.b[0] = oF[r + 1 - side];
                }
            }
            const float v = sum_write(t, i, d, side, near_finish<Q>(s, part[buf][x][2 * r + side], R));
            if (Q == 2 && side == 1) oS[r] = v;
        }
    };
    auto finish_f = [&](int x, const Pair& p, int e, int c0, auto ready) {
        const int d = e - x, n = x ? min(kOutsideRows, p.nb - c0) : min(kOutsideRows + 1, p.na - c0);
        for (int base = 0; base < n || base == 0; base += 32) {
            const int r = base + (tid & 31), i = p.r0 - 1 + x + c0 + r;
            const bool mine = r < n && i >= 0;
            FOperands f;
            await(mine, [&] { f_load(t, i, d, f); }, [&] { return f.complete(); });
            if (base == 0) ready();
            if (!mine) continue;
            const float v = f_finish(f, R);
            f_write(t, i, d, v);
            if (x == 0) oF[r] = v;
        }
    };
    // Diagonal e by warps 0 and 1, then (behind a barrier of the four) e-1 by 2 and 3.
    auto finish = [&](const Pair& p, int e, int c0, int buf, auto ready) {
        const int warp = tid >> 5;
        const auto both = [&] {
            ready();
            fin_barrier();  // diagonal e of this CTA's rows is in oS / oF
        };
        if (warp == 0) finish_sums(std::integral_constant<int, 2>{}, p, e, c0, buf, ready);
        else if (warp == 1) finish_f(0, p, e, c0, ready);
        else if (warp == 2) finish_sums(std::integral_constant<int, 3>{}, p, e, c0, buf, both);
        else finish_f(1, p, e, c0, both);
        if (warp < 2) fin_barrier();
    };

    int buf = 0;
    Pair p = pair_at(Wb);
    if (!fin) sums(p, Wb, 0, 0);
    for (int e = Wb; e >= 0; e -= 2, buf ^= 1) {
        bool stop = false;
        // every thread: the pair's sums are there, and its operands
        auto together = [&] { stop = __syncthreads_or(bad) != 0; };
        const Pair next = e >= 2 ? pair_at(e - 2) : Pair{0, 0, 0};
        if (fin) {
            finish(p, e, 0, buf, together);
        } else {
            together();
            if (!stop && e >= 2) sums(next, e - 2, 0, buf ^ 1);
        }
        // more rows than a CTA holds: the rest apart
        for (int c0 = kOutsideRows; c0 < max(p.na - 1, p.nb); c0 += kOutsideRows) {
            __syncthreads();
            if (!fin) sums(p, e, c0, buf);
            __syncthreads();
            if (fin) finish(p, e, c0, buf, [] {});
        }
        if (stop) return;
        p = next;
    }
}

// CTAs of a cooperative launch: one per SM at most (more would share the SM's
// loads and lengthen every wait), fewer where the context caps them.
static int wave_grid(messi_ctx* ctx)
{
    int sms = ctx->num_sms;
    if (sms <= 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        ctx->num_sms = sms;
    }
    return ctx->wave_ctas > 0 ? std::min(sms, ctx->wave_ctas) : std::max(sms, 1);
}

// Tables to be filled with kUnwritten before a wavefront launch, and its status
// words cleared, in one launch (a memset each: four or six launches, 6-10 us of
// a small alignment's pass).
struct WaitTables {
    float* cells[5] = {};
    size_t n[5] = {};  // multiples of 4
};

__global__ void __launch_bounds__(256) wait_tables_kernel(WaitTables w, unsigned int* sync)
{
    if (blockIdx.x == 0 && threadIdx.x < kSyncWords) sync[threadIdx.x] = 0u;
    const uint4 v = make_uint4(kUnwritten, kUnwritten, kUnwritten, kUnwritten);
    for (int k = 0; k < 5; k++) {
        uint4* c = reinterpret_cast<uint4*>(w.cells[k]);
        for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < w.n[k] / 4; i += (size_t)gridDim.x * blockDim.x)
            c[i] = v;
    }
}

static int launch_wait_tables(messi_ctx* ctx, const WaitTables& w, unsigned int* sync)
{
    size_t total = 0;
    bool aligned = true;
    for (int k = 0; k < 5; k++) {
        total += w.n[k];
        aligned = aligned && ((uintptr_t)w.cells[k] & 15) == 0 && w.n[k] % 4 == 0;
    }
    if (!aligned) {
        cudaError_t e = cudaMemsetAsync(sync, 0, kSyncWords * sizeof(unsigned int), ctx->stream);
        for (int k = 0; k < 5 && e == cudaSuccess; k++)
            if (w.n[k]) e = cudaMemsetAsync(w.cells[k], 0xff, w.n[k] * sizeof(float), ctx->stream);
        return e == cudaSuccess ? MESSI_OK : cuda_fail(ctx, e, "wavefront table reset");
    }
    const int grid = (int)std::max<size_t>(1, std::min<size_t>(total / 4 / 256, 152 * 8));
    wait_tables_kernel<<<grid, 256, 0, ctx->stream>>>(w, sync);
    LAUNCH_CHECK(ctx, "wait_tables_kernel");
    return MESSI_OK;
}

// The inside kernel (cooperative: every CTA resident), one CTA per SM, after
// the tables it waits on are filled with kUnwritten.
// 512 threads (1,024 leave 64 registers a thread and spill: span 500 of 1,000
// columns 0.67 ms against 0.54); 256 where a CTA has at most two cells of a
// diagonal and four warps form their sums (L = 120: 93 us against 102, L = 300:
// 250 against 266, but L = 600, four cells: 370 against 277).  `many`, null for
// a batch: with 16 cells and more per CTA twenty warps that form the sums are
// worth more than twelve with their next loads in flight (span 800 of 3,000,
// 4,500, 6,000 columns: 1.83, 2.52, 3.22 ms against 1.99, 2.87, 3.75; L = 2,001,
// 13 cells: 3.98 against 3.39; the batch, which needs more registers, 1.34
// against 1.23).
static int launch_inside(messi_ctx* ctx, const void* kernel, const void* many, void** args, unsigned int* sync,
                         long long columns, const WaitTables& tables)
{
    if (const int rc = launch_wait_tables(ctx, tables, sync)) return rc;
    const int most = wave_grid(ctx);  // also sets ctx->num_sms
    const int grid = (int)std::min<long long>(most, columns);
    int threads = columns <= 2 * (long long)ctx->num_sms ? kInsideThreads / 2 : kInsideThreads;
    if (ctx->wave_threads == 256 || ctx->wave_threads >= kInsideThreads)
        threads = std::min(ctx->wave_threads, kInsideThreads);
    if (many && threads == kInsideThreads && columns >= (long long)kInsideManyRows * grid) {
        kernel = many;
        threads = kInsideManyThreads;
    }
    const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(threads), args, 0, ctx->stream);
    ctx->launches++;
    return e == cudaSuccess ? MESSI_OK : cuda_fail(ctx, e, "inside_pair_kernel");
}

// Self-test of the bounded wait: a warp waits for a cell (sync[3]) that nothing
// writes.  First lane 0 alone sees an error flag that is up (its status words are
// the second set): all lanes have to leave at the look that finds it; the looks
// of every lane are left behind the two sets.  Then the wait gives up after
// `limit` looks and raises the flag of the first set.  Nothing faults and nothing
// waits unboundedly; the context stays usable.
__global__ void __launch_bounds__(32) wait_selftest_kernel(unsigned int* sync, unsigned int limit)
{
    const float* cell = reinterpret_cast<const float*>(sync + 3);
    unsigned int spins = 0;
    while (unwritten(ld_cell(cell)))
        if (!warp_keep_waiting(spins, threadIdx.x == 0 ? sync + kSyncWords : sync, limit)) break;
    sync[2 * kSyncWords + threadIdx.x] = spins;
    spins = 0;
    while (unwritten(ld_cell(cell)))
        if (!warp_keep_waiting(spins, sync, limit)) return;
}

int launch_wait_selftest(messi_ctx* ctx, unsigned int* d_sync)
{
    cudaError_t e = cudaMemsetAsync(d_sync, 0, kSelftestWords * sizeof(unsigned int), ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_sync + 3, 0xff, sizeof(unsigned int), ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_sync + kSyncWords + 2, 0xff, sizeof(unsigned int), ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "wait self-test reset");
    wait_selftest_kernel<<<1, 32, 0, ctx->stream>>>(d_sync, 1u << 12);
    LAUNCH_CHECK(ctx, "wait_selftest_kernel");
    return MESSI_OK;
}

// The outside kernel (cooperative), one CTA per SM, after its tables are filled
// with kUnwritten.  More rows per CTA want more warps for their sums, although
// fewer registers a thread then spill: 512, 768, 1,024 threads took 308, 366, 433
// us with 2 rows (every span of 300 columns), 522, 439, 492 with 4 (span 300 of
// 600) and 1,217, 1,175, 1,065 with 7 (span 500 of 1,000).
static int launch_outside(messi_ctx* ctx, const Band& t, void** args, unsigned int* sync)
{
    const size_t tab = (size_t)t.L * t.RS;
    const WaitTables tables{{t.OSrow, t.OScol, t.OFrow, t.OFcol, t.OLrow}, {tab, tab, tab, tab, tab}};
    if (const int rc = launch_wait_tables(ctx, tables, sync)) return rc;
    const void* kernel = (const void*)outside_pair_kernel<1024>;
    const int grid = std::min(wave_grid(ctx), t.L);
    const int rows = (t.L + grid - 1) / grid;
    int threads = ctx->wave_threads ? ctx->wave_threads : (rows <= 2 ? 512 : (rows <= 5 ? 768 : 1024));
    if (threads <= 512) kernel = (const void*)outside_pair_kernel<512>;
    else if (threads == 768) kernel = (const void*)outside_pair_kernel<768>;
    const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(threads), args, 0, ctx->stream);
    ctx->launches++;
    return e == cudaSuccess ? MESSI_OK : cuda_fail(ctx, e, "outside_pair_kernel");
}

int run_inside(messi_ctx* ctx, const Band& t, double B)
{
    Rules R = make_rules(B);
    const size_t tab = (size_t)t.L * t.RS;
    InsideBands<false> ib{t, nullptr, nullptr, nullptr, 1};
    double Bv = B;
    unsigned int* sync = t.sync;
    void* args[] = {&ib, &R, &Bv, &sync};
    prof_begin(ctx, 1, (double)t.L * (t.Wb + 1) - 0.5 * t.Wb * (t.Wb + 1.0));
    int rc = launch_inside(ctx, (const void*)inside_pair_kernel<false, kInsideThreads>,
                           (const void*)inside_pair_kernel<false, kInsideManyThreads>, args, sync, t.L,
                           WaitTables{{t.Lrow, t.Scol, t.Frow}, {tab, tab, tab}});
    if (rc) return rc;
    prof_end(ctx);
    if (t.L - 1 > t.Wb) {
        prof_begin(ctx, 2, (double)(t.L - 1 - t.Wb));
        const int win = suffix_launch_window(ctx, t.Wb);
        const cudaError_t e = allow_smem(ctx->device, (const void*)inside_suffix_kernel, (size_t)2 * win * sizeof(float));
        if (e != cudaSuccess) return cuda_fail(ctx, e, "inside_suffix_kernel attributes");
        inside_suffix_kernel<<<1, kSuffixThreads, (size_t)2 * win * sizeof(float), ctx->stream>>>(t, R, win);
        LAUNCH_CHECK(ctx, "inside_suffix_kernel");
        prof_end(ctx);
    }
    return launch_finish_Z(ctx, t);
}

// ---------------------------------------------------------------------------
// batched inside
// ---------------------------------------------------------------------------
int bandbatch_alloc(const std::vector<int>& L, const std::vector<int>& Wb, BandBatch* bb, std::string* err)
{
    const int n = (int)L.size();
    bb->n = n;
    bb->order.resize(n);
    for (int a = 0; a < n; a++) bb->order[a] = a;
    std::stable_sort(bb->order.begin(), bb->order.end(), [&](int x, int y) { return Wb[x] > Wb[y]; });
    bb->slot.assign(n, 0);
    for (int k = 0; k < n; k++) bb->slot[bb->order[k]] = k;
    // one allocation: per band 6 tables, Ssuf/Osuf, b/cb/u/Zd; then the batch arrays
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    std::vector<size_t> off_polled(n), off_tab(n), off_suf(n), off_dbl(n);
    size_t bytes = 0;
    for (int k = 0; k < n; k++) {  // the tables that the inside kernel waits on, for one fill
        const int a = bb->order[k];
        off_polled[k] = bytes;
        bytes = al(bytes + 3 * (size_t)L[a] * (((size_t)Wb[a] + 1 + 31) / 32 * 32) * sizeof(float));
    }
    bb->polled = bytes / sizeof(float);
    for (int k = 0; k < n; k++) {
        const int a = bb->order[k];
        const size_t RS = ((size_t)Wb[a] + 1 + 31) / 32 * 32;
        off_tab[k] = bytes;
        bytes = al(bytes + 3 * (size_t)L[a] * RS * sizeof(float));
        off_suf[k] = bytes;
        bytes = al(bytes + (size_t)(L[a] + 1) * 2 * sizeof(float));
        off_dbl[k] = bytes;
        bytes = al(bytes + (size_t)(3 * L[a] + 8) * sizeof(double));
    }
    const size_t off_bands = bytes;
    bytes = al(bytes + (size_t)n * sizeof(Band));
    const size_t off_cum = bytes;
    bytes = al(bytes + (size_t)(n + 1) * sizeof(long long));
    const size_t off_wbs = bytes;
    bytes = al(bytes + (size_t)n * sizeof(int));
    const size_t off_sync = bytes;
    bytes = al(bytes + kSyncWords * sizeof(unsigned int));
    const size_t off_Z = bytes;
    bytes = al(bytes + (size_t)n * sizeof(double));
    cudaError_t e = cudaMalloc(&bb->mem, bytes);
    if (e != cudaSuccess) {
        bb->mem = nullptr;
        *err = std::string("batch band tables: ") + cudaGetErrorString(e);
        return MESSI_ENOMEM;
    }
    bb->bytes = bytes;
    char* base = (char*)bb->mem;
    bb->host.assign(n, Band{});
    std::vector<long long> cum(n + 1, 0);
    std::vector<int> wbs(n);
    bb->d_sync = (unsigned int*)(base + off_sync);
    for (int k = 0; k < n; k++) {
        const int a = bb->order[k];
        Band& t = bb->host[k];
        t.L = L[a];
        t.Wb = Wb[a];
        t.RS = ((Wb[a] + 1 + 31) / 32) * 32;
        const size_t tab = (size_t)t.L * t.RS;
        float* f = (float*)(base + off_polled[k]);
        t.Lrow = f;
        t.Scol = f + tab;
        t.Frow = f + 2 * tab;
        f = (float*)(base + off_tab[k]);
        t.Lcol = f;
        t.Srow = f + tab;
        t.pb = f + 2 * tab;
        t.Ssuf = (float*)(base + off_suf[k]);
        t.Osuf = t.Ssuf + (t.L + 1);
        t.b = (double*)(base + off_dbl[k]);
        t.cb = t.b + t.L;
        t.u = t.cb + (t.L + 1);
        t.Zd = t.u + t.L;
        t.maxspan = nullptr;
        t.sync = bb->d_sync;
        t.OSrow = t.OScol = t.OFrow = t.OFcol = t.OLrow = t.PP = t.SL = t.nrm = t.OSlast = nullptr;
        cum[k + 1] = cum[k] + t.L;
        wbs[k] = t.Wb;
    }
    bb->total_cols = cum[n];
    bb->d_bands = (Band*)(base + off_bands);
    bb->d_cumL = (long long*)(base + off_cum);
    bb->d_wbs = (int*)(base + off_wbs);
    bb->d_Z = (double*)(base + off_Z);
    e = cudaMemcpy(bb->d_bands, bb->host.data(), (size_t)n * sizeof(Band), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(bb->d_cumL, cum.data(), (size_t)(n + 1) * sizeof(long long), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(bb->d_wbs, wbs.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);  // the contexts' streams do not wait for the default stream
    if (e != cudaSuccess) {
        *err = std::string("batch band descriptors: ") + cudaGetErrorString(e);
        return MESSI_ECUDA;
    }
    return MESSI_OK;
}

void bandbatch_free(BandBatch* bb)
{
    if (bb->mem) cudaFree(bb->mem);
    bb->mem = nullptr;
    bb->host.clear();
}

int launch_baseline_batch(messi_ctx* ctx, const BandBatch& bb, double B)
{
    if (bb.n == 0) return MESSI_OK;
    baseline_batch_kernel<<<bb.n, 1024, 0, ctx->stream>>>(bb.d_bands, B, baseline_c());
    LAUNCH_CHECK(ctx, "baseline_batch_kernel");
    return MESSI_OK;
}

int run_inside_batch(messi_ctx* ctx, const BandBatch& bb, double B)
{
    if (bb.n == 0) return MESSI_OK;
    Rules R = make_rules(B);
    const Band* bands = bb.d_bands;
    const long long* cum = bb.d_cumL;
    const int* wbs = bb.d_wbs;
    int n = bb.n;
    double Bv = B;
    unsigned int* sync = bb.d_sync;
    InsideBands<true> ib{bb.host[0], bands, cum, wbs, n};
    void* args[] = {&ib, &R, &Bv, &sync};
    double cells = 0.0;
    for (const Band& t : bb.host) cells += (double)t.L * (t.Wb + 1) - 0.5 * t.Wb * (t.Wb + 1.0);
    prof_begin(ctx, 1, cells);
    int rc = launch_inside(ctx, (const void*)inside_pair_kernel<true, kInsideThreads>, nullptr, args, sync, bb.total_cols,
                           WaitTables{{bb.host[0].Lrow}, {bb.polled}});
    if (rc) return rc;
    cudaError_t e;
    prof_end(ctx);
    prof_begin(ctx, 2, 0.0);
    const int win = suffix_batch_window(ctx, bb);
    e = allow_smem(ctx->device, (const void*)inside_suffix_batch_kernel, (size_t)2 * win * sizeof(float));
    if (e != cudaSuccess) return cuda_fail(ctx, e, "inside_suffix_batch_kernel attributes");
    inside_suffix_batch_kernel<<<n, kSuffixThreads, (size_t)2 * win * sizeof(float), ctx->stream>>>(bands, R, win);
    LAUNCH_CHECK(ctx, "inside_suffix_batch_kernel");
    prof_end(ctx);
    finish_Z_batch_kernel<<<(n + 127) / 128, 128, 0, ctx->stream>>>(bands, n, sync, bb.d_Z);
    LAUNCH_CHECK(ctx, "finish_Z_batch_kernel");
    return queue_status(ctx, sync + 2);
}

// ---------------------------------------------------------------------------
// outside
// ---------------------------------------------------------------------------
// Osuf[i] for spans beyond the band on the last column, ascending i:
// Osuf[0] = 0;  Osuf[i] = r1 + LSE_{k=0..Wb, i-k-1>=0} (Osuf[i-k-1] + Lcol[i-1][k]).
// Osuf[i] (outside of S(i, L-1) beyond the band, i < T = L-1-Wb), ascending
// i: Osuf[0] = 0, Osuf[i] = r1 + LSE_{k=0..min(Wb, i-1)} (Osuf[i-k-1] +
// Lcol[i-1][k]).  The mirror of the inside suffix: blocks of 32 cells from
// the bottom, every finished block pushed into the next Wb+1 cells'
// shared-memory accumulators (warp 0 into the next block and its triangle,
// the other warps into the farther cells, one barrier per block).
__device__ void outside_suffix_body(const Band& t, const Rules& R, float* am, float* as, int win)
{
    const int Wb = t.Wb, RS = t.RS;
    const int T = t.L - 1 - Wb;
    if (T <= 0) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // tri[q][k] = Lcol[i0 + q - 1][k] for the block's cells i0 + q, double-buffered
    __shared__ float tri2[2][32][33];
    __shared__ float etri2[2][32][33];  // exp(tri + r1), staged with tri
    __shared__ float vals2[2][32];
    // xs[u][q]: the L value joining next-block cell hi+1+q to this block's
    // cell i0+u (warp 0's push after the triangle), staged a block ahead by warp 1
    __shared__ float xs2[2][32][33];
    int parity = 0, tb = 0;
    for (int c = threadIdx.x; c < win; c += blockDim.x) {
        am[c] = -INFINITY;
        as[c] = 0.f;
    }
    int i0 = 0, hi = min(T - 1, 31);
    // the first two blocks' pushes (Lrow rows i0 .. hi+32) and the second
    // block's in-block terms (first line of Lcol rows hi .. hi+31)
    prefetch_rows_l2(t.Lrow, RS, t.L, i0, hi + 32, RS / 32, threadIdx.x, blockDim.x);
    prefetch_rows_l2(t.Lcol, RS, t.L, hi, hi + 31, 1, threadIdx.x, blockDim.x);
    if (w == 1) {
        for (int q = 0; q < 32; q++) {
            const int c = i0 + q;
            const float v = (c <= hi && c >= 1 && lane <= Wb) ? __ldg(t.Lcol + (size_t)(c - 1) * RS + lane) : -INFINITY;
            tri2[0][q][lane] = v;
            etri2[0][q][lane] = __expf(v + R.r[0]);
        }
        const int nb0 = hi - i0 + 1, nhi0 = min(T - 1, hi + 32), c = hi + 1 + lane;
        for (int u = 0; u < 32; u++) {
            const int k = c - 1 - i0 - u;
            xs2[0][u][lane] = (hi < T - 1 && c <= nhi0 && u < nb0 && k >= 0 && k <= Wb)
                                  ? __ldg(t.Lrow + (size_t)(i0 + u) * RS + k)
                                  : -INFINITY;
        }
    }
    __syncthreads();
    float cm = -INFINITY, cs = 0.f;
    for (;;) {
        const int nb = hi - i0 + 1;
        const int nhi = min(T - 1, hi + 32);
        float* vals = vals2[parity];
        parity ^= 1;
        float x[32];  // warp 0: L values joining its next-block cell to this block's cells
        if (w == 0) {
            // column-oriented substitution (lane q owns cell i0 + q); Osuf[0]
            // = 0 is (m, s) = (-r1, 1), so every value is r1 + m + log s
            float m = (lane < nb) ? cm : -INFINITY, s = (lane < nb) ? cs : 0.f;
            if (i0 + lane == 0) {
                m = -R.r[0];
                s = 1.f;
            }
            suffix_triangle(m, s, tri2[tb], etri2[tb], nb, lane < nb && i0 + lane >= 1, Wb, R.r[0], lane);
            // the block's values, stored by all lanes at once
            if (lane < nb) {
                const float sv = (i0 + lane == 0) ? 0.f : R.r[0] + lse_val(m, s);
                t.Osuf[i0 + lane] = sv;
                vals[lane] = sv;
            }
            // the push operands, before the barrier: warp 1 refills this
            // buffer in the next block
#pragma unroll
            for (int u = 0; u < 32; u++) x[u] = xs2[tb][u][lane];
        } else if (w == 1 && hi < T - 1) {
            // the next block's in-block terms and push operands: all 64 loads
            // first, then the stores (one memory round trip)
            const int i0n = hi + 1, nbn = nhi - hi, nhin = min(T - 1, nhi + 32), c = nhi + 1 + lane;
            float v[32], y[32];
#pragma unroll
            for (int q = 0; q < 32; q++) {
                const int cq = hi + 1 + q;
                const bool onv = cq <= nhi && lane <= Wb;
                v[q] = ldg_if(t.Lcol + (onv ? (size_t)(cq - 1) * RS + lane : 0), onv, -INFINITY);
                const int k = c - 1 - i0n - q;
                const bool ony = nhi < T - 1 && c <= nhin && q < nbn && k >= 0 && k <= Wb;
                y[q] = ldg_if(t.Lrow + (ony ? (size_t)(i0n + q) * RS + k : 0), ony, -INFINITY);
            }
#pragma unroll
            for (int q = 0; q < 32; q++) {
                tri2[tb ^ 1][q][lane] = v[q];
                etri2[tb ^ 1][q][lane] = __expf(v[q] + R.r[0]);
                xs2[tb ^ 1][q][lane] = y[q];
            }
        } else if (w >= 2) {
            // the block after the next one: its pushes read Lrow rows
            // hi+33 .. hi+64, its in-block terms Lcol rows hi+32 .. hi+63
            prefetch_rows_l2(t.Lrow, RS, t.L, hi + 33, hi + 64, RS / 32, threadIdx.x - 64, blockDim.x - 64);
            prefetch_rows_l2(t.Lcol, RS, t.L, hi + 32, hi + 63, 1, threadIdx.x - 64, blockDim.x - 64);
        }
        __syncthreads();
        if (hi == T - 1) break;
        // push the block [i0, hi] (value u = cell i0 + u) into the cells
        // hi+1 .. hi+1+Wb: L(i0 + u, c - 1) = Lrow[i0 + u][c - 1 - i0 - u],
        // contiguous in c; a cell's first push (from the block holding its
        // smallest referenced cell) starts it afresh
        if (w == 0) {
            const int c = hi + 1 + lane;
            cm = -INFINITY;
            cs = 0.f;
            if (c <= nhi) {
                const bool fresh = i0 <= max(0, c - 1 - Wb);
                if (!fresh) {
                    cm = am[c % win];
                    cs = as[c % win];
                }
#pragma unroll
                for (int u = 0; u < 32; u += 8) {
                    const float y[8] = {x[u] + vals[u], x[u + 1] + vals[u + 1], x[u + 2] + vals[u + 2],
                                        x[u + 3] + vals[u + 3], x[u + 4] + vals[u + 4], x[u + 5] + vals[u + 5],
                                        x[u + 6] + vals[u + 6], x[u + 7] + vals[u + 7]};
                    lse_add8(cm, cs, y);
                }
            }
        } else if (w >= 2) {
            for (int c = nhi + 1 + (threadIdx.x - 64); c <= min(T - 1, hi + 1 + Wb); c += (int)blockDim.x - 64) {
                const bool fresh = i0 <= max(0, c - 1 - Wb);
                float m = fresh ? -INFINITY : am[c % win], s = fresh ? 0.f : as[c % win];
                suffix_push_terms(m, s, t.Lrow, RS, i0, 1, c - 1 - i0, vals, nb, Wb);
                am[c % win] = m;
                as[c % win] = s;
            }
        }
        tb ^= 1;
        i0 = hi + 1;
        hi = nhi;
    }
}

// Blocks of 32 cells pulled from global memory (bands wider than the window).
__device__ void outside_suffix_body_pull(const Band& t, const Rules& R)
{
    const int T = t.L - 1 - t.Wb;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    __shared__ float known[32];
    __shared__ float tri[32][33];  // Lcol[i0 + l - 1][k], k < 32: the in-block terms
    for (int i0 = 0; i0 < T; i0 += 32) {
        const int hi = min(T - 1, i0 + 31);
        for (int q = w; q < 32; q += nw) {  // a warp per cell i0 + q
            const int i = i0 + q;
            tri[q][lane] = (i <= hi && i >= 1 && lane <= t.Wb) ? t.Lcol[(size_t)(i - 1) * t.RS + lane] : -INFINITY;
            if (i > hi) continue;
            float m = -INFINITY, s = 0.f;
            if (i >= 1) {
                const float* lcol = t.Lcol + (size_t)(i - 1) * t.RS;
                const int kmax = min(t.Wb, i - 1);
                int k = (i - i0) + lane;
                for (; k + 96 <= kmax; k += 128)
                    lse_add4(m, s, t.Osuf[i - k - 1] + lcol[k], t.Osuf[i - k - 33] + lcol[k + 32],
                             t.Osuf[i - k - 65] + lcol[k + 64], t.Osuf[i - k - 97] + lcol[k + 96]);
                for (; k <= kmax; k += 32) lse_add(m, s, t.Osuf[i - k - 1] + lcol[k]);
            }
            group_reduce<32>(m, s);
            if (lane == 0) known[q] = lse_val(m, s);
        }
        __syncthreads();
        if (w == 0) {
            // column-oriented substitution (lane q owns cell i0 + q); Osuf[0] = 0
            const int nb = hi - i0 + 1;
            float am = (lane < nb) ? known[lane] : -INFINITY, as = (am == -INFINITY) ? 0.f : 1.f;
            for (int l = 0; l < nb; l++) {
                const int ic = i0 + l;
                const float fin = (ic == 0) ? 0.f : R.r[0] + lse_val(am, as);
                const float sv = __shfl_sync(0xffffffffu, fin, l);
                if (lane == 0) t.Osuf[ic] = sv;
                const int k = lane - l - 1;
                if (lane > l && lane < nb && k <= t.Wb && i0 + lane >= 1) lse_add(am, as, tri[lane][k] + sv);
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kSuffixThreads) outside_suffix_kernel(Band t, Rules R, int win)
{
    extern __shared__ float suffix_smem[];
    if (suffix_window(t.Wb) <= win) outside_suffix_body(t, R, suffix_smem, suffix_smem + win, win);
    else outside_suffix_body_pull(t, R);
}

int run_outside(messi_ctx* ctx, const Band& t, double B)
{
    Rules R = make_rules(B);
    if (t.L - 1 > t.Wb) {
        const int win = suffix_launch_window(ctx, t.Wb);
        const cudaError_t e = allow_smem(ctx->device, (const void*)outside_suffix_kernel, (size_t)2 * win * sizeof(float));
        if (e != cudaSuccess) return cuda_fail(ctx, e, "outside_suffix_kernel attributes");
        outside_suffix_kernel<<<1, kSuffixThreads, (size_t)2 * win * sizeof(float), ctx->stream>>>(t, R, win);
        LAUNCH_CHECK(ctx, "outside_suffix_kernel");
    }
    {
        const int rows = t.L - std::max(1, t.L - 1 - t.Wb);  // last-column band cells with i >= 1
        if (rows > 0) {
            outside_lastcol_kernel<<<(rows + 7) / 8, 256, 0, ctx->stream>>>(t, R);
            LAUNCH_CHECK(ctx, "outside_lastcol_kernel");
        }
    }
    Band tt = t;
    unsigned int* sync = t.sync;
    void* args[] = {&tt, &R, &sync};
    prof_begin(ctx, 3, (double)t.L * (t.Wb + 1) - 0.5 * t.Wb * (t.Wb + 1.0));
    int rc = launch_outside(ctx, tt, args, sync);
    if (rc) return rc;
    prof_end(ctx);
    return queue_status(ctx, t.sync + 2);
}

// ---------------------------------------------------------------------------
// posteriors (computebasepairprobs, row-normalised)
// ---------------------------------------------------------------------------
__global__ void post_cells_kernel(Band t, Rules R, double B)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)t.L * t.RS) return;
    const int j = (int)(idx / t.RS), d = (int)(idx % t.RS);
    const float Zbar = t.Ssuf[0];
    if (d == 0) {
        float m = -INFINITY, s = 0.f;
        lse_add(m, s, t.OSrow[(size_t)j * t.RS] + R.r[1]);
        lse_add(m, s, t.OLrow[(size_t)j * t.RS] + R.r[5]);
        const double uj = t.u[j];
        t.SL[j] = (uj == -INFINITY) ? -INFINITY : (float)((double)lse_val(m, s) + B * uj - t.b[j]) - Zbar;
        t.PP[idx] = -INFINITY;
        return;
    }
    float out = -INFINITY;
    if (d <= t.Wb && j + d < t.L) {
        const float pp = t.pb[idx];
        const float fin = (d >= 2) ? t.Frow[(size_t)(j + 1) * t.RS + (d - 2)] : -INFINITY;
        if (pp != -INFINITY && fin != -INFINITY) {
            float m = -INFINITY, s = 0.f;
            lse_add(m, s, t.OSrow[idx] + R.r[2]);
            lse_add(m, s, t.OFrow[idx] + R.r[3]);
            lse_add(m, s, t.OLrow[idx] + R.r[6]);
            out = lse_val(m, s) + fin + pp - Zbar;
        }
    }
    t.PP[idx] = out;
}

// one warp per row x: log normaliser over the unpaired term and every partner
__global__ void post_norm_kernel(Band t)
{
    const int x = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (x >= t.L) return;
    float m = -INFINITY, s = 0.f;
    if (lane == 0) lse_add(m, s, t.SL[x]);
    for (int d = 1 + lane; d <= t.Wb; d += 32) {
        if (x + d < t.L) lse_add(m, s, t.PP[(size_t)x * t.RS + d]);
        if (x - d >= 0) lse_add(m, s, t.PP[(size_t)(x - d) * t.RS + d]);
    }
    group_reduce<32>(m, s);
    if (lane == 0) t.nrm[x] = lse_val(m, s);
}

__global__ void post_dense_kernel(Band t, double* __restrict__ single, double* __restrict__ pair)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int L = t.L;
    if (idx >= (long long)L * L) return;
    const int x = (int)(idx % L), y = (int)(idx / L);
    const int k = (x > y) ? x - y : y - x;
    double v = 0.0;
    if (k >= 1 && k <= t.Wb) {
        const int i = (x < y) ? x : y;
        const float pp = t.PP[(size_t)i * t.RS + k];
        if (pp != -INFINITY) v = exp((double)pp - (double)t.nrm[x]);
    }
    pair[idx] = v;
    if (y == 0) single[x] = exp((double)t.SL[x] - (double)t.nrm[x]);
}

int run_posteriors(messi_ctx* ctx, const Band& t, double B, double* d_single, double* d_pair)
{
    const Rules R = make_rules(B);
    const long long n = (long long)t.L * t.RS;
    post_cells_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(t, R, B);
    LAUNCH_CHECK(ctx, "post_cells_kernel");
    post_norm_kernel<<<(unsigned)(((long long)t.L * 32 + 255) / 256), 256, 0, ctx->stream>>>(t);
    LAUNCH_CHECK(ctx, "post_norm_kernel");
    const long long nn = (long long)t.L * t.L;
    post_dense_kernel<<<(unsigned)((nn + 255) / 256), 256, 0, ctx->stream>>>(t, d_single, d_pair);
    LAUNCH_CHECK(ctx, "post_dense_kernel");
    return MESSI_OK;
}

// ---------------------------------------------------------------------------
// dense (Julia-layout) tables <-> band tables
// ---------------------------------------------------------------------------
__global__ void dense_inside_kernel(Band t, double* __restrict__ out)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int L = t.L;
    if (idx >= (long long)L * L) return;
    const int i = (int)(idx % L), j = (int)(idx / L);
    double S = -INFINITY, F = -INFINITY, Lv = -INFINITY;
    if (j >= i) {
        const int d = j - i;
        const double base = t.cb[j + 1] - t.cb[i];
        if (d <= t.Wb) {
            const size_t o = (size_t)i * t.RS + d;
            S = (double)t.Srow[o] + base;
            F = (double)t.Frow[o] + base;
            Lv = (double)t.Lrow[o] + base;
        } else if (j == L - 1) {
            S = (double)t.Ssuf[i] + base;
        }
    }
    out[3 * idx] = S;
    out[3 * idx + 1] = F;
    out[3 * idx + 2] = Lv;
}

__global__ void dense_outside_kernel(Band t, double* __restrict__ out)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int L = t.L;
    if (idx >= (long long)L * L) return;
    const int i = (int)(idx % L), j = (int)(idx / L);
    double S = -INFINITY, F = -INFINITY, Lv = -INFINITY;
    if (j >= i) {
        const int d = j - i;
        const double base = t.cb[L] - (t.cb[j + 1] - t.cb[i]);
        if (d <= t.Wb) {
            const size_t o = (size_t)i * t.RS + d;
            S = (double)t.OSrow[o] + base;
            F = (double)t.OFrow[o] + base;
            Lv = (double)t.OLrow[o] + base;
        } else if (j == L - 1) {
            S = (double)t.Osuf[i] + base;
        }
    }
    out[3 * idx] = S;
    out[3 * idx + 1] = F;
    out[3 * idx + 2] = Lv;
}

int launch_dense_inside(messi_ctx* ctx, const Band& t, double* d_out)
{
    const long long n = (long long)t.L * t.L;
    dense_inside_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(t, d_out);
    LAUNCH_CHECK(ctx, "dense_inside_kernel");
    return MESSI_OK;
}

int launch_dense_outside(messi_ctx* ctx, const Band& t, double* d_out)
{
    const long long n = (long long)t.L * t.L;
    dense_outside_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(t, d_out);
    LAUNCH_CHECK(ctx, "dense_outside_kernel");
    return MESSI_OK;
}

__global__ void band_from_dense_inside_kernel(Band t, const double* __restrict__ in)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int L = t.L;
    if (idx >= (long long)L * L) return;
    const int i = (int)(idx % L), j = (int)(idx / L);
    if (j < i) return;
    const int d = j - i;
    const double base = t.cb[j + 1] - t.cb[i];
    const double S = in[3 * idx], F = in[3 * idx + 1], Lv = in[3 * idx + 2];
    if (d <= t.Wb) {
        const float s = (float)(S - base), f = (float)(F - base), l = (float)(Lv - base);
        t.Srow[(size_t)i * t.RS + d] = s;
        t.Scol[(size_t)j * t.RS + d] = s;
        t.Frow[(size_t)i * t.RS + d] = f;
        t.Lrow[(size_t)i * t.RS + d] = l;
        t.Lcol[(size_t)j * t.RS + d] = l;
    }
    if (j == L - 1) t.Ssuf[i] = (float)(S - base);
}

__global__ void band_from_dense_outside_kernel(Band t, const double* __restrict__ in)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int L = t.L;
    if (idx >= (long long)L * L) return;
    const int i = (int)(idx % L), j = (int)(idx / L);
    if (j < i) return;
    const int d = j - i;
    if (d > t.Wb) return;
    const double base = t.cb[L] - (t.cb[j + 1] - t.cb[i]);
    const size_t o = (size_t)i * t.RS + d;
    t.OSrow[o] = (float)(in[3 * idx] - base);
    t.OFrow[o] = (float)(in[3 * idx + 1] - base);
    t.OLrow[o] = (float)(in[3 * idx + 2] - base);
}

int launch_band_from_dense_inside(messi_ctx* ctx, const Band& t, const double* d_in)
{
    const long long n = (long long)t.L * t.L;
    band_from_dense_inside_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(t, d_in);
    LAUNCH_CHECK(ctx, "band_from_dense_inside_kernel");
    return MESSI_OK;
}

int launch_band_from_dense_outside(messi_ctx* ctx, const Band& t, const double* d_out)
{
    const long long n = (long long)t.L * t.L;
    band_from_dense_outside_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(t, d_out);
    LAUNCH_CHECK(ctx, "band_from_dense_outside_kernel");
    return MESSI_OK;
}

}  // namespace messi
