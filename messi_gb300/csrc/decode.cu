// decode.cu -- structures from the SCFG tables: maximum-expected-accuracy
// posterior decoding and stochastic sampling of structures.
//
// Posterior decoding replaces computeposteriordecodingcuda
// (src/InsideCUDA.jl:183-215, kernel posteriordecoding of
// src/cuda/inside.cu:286-321, one launch per span) and the CPU traceback
// posteriordecodingtraceback (src/RNATools.jl:43-72).  The recursion, in FP32
// as the reference's GPU path computes it:
//     e(i,i) = 0
//     e(i,j) = max( single[i] + e(i+1,j),                                  s = -1
//                   alpha*pair(i,j) + e(i+1,j-1),                          s = -2
//                   max_k alpha*pair(i,k) + e(i+1,k-1) + e(k+1,j) )        s = k+1
// with ties to the first alternative and the smallest k.  One persistent
// cooperative launch walks the diagonals of 16 x 16 tiles (a row block waits
// for the next one's flag).  e is kept row-major (the split's second factor) and
// column-major (the output); s is written column-major, the layout the Julia
// caller reads.  The traceback runs on the device in one thread.
//
// Structure sampling replaces samplestructure / samplestructurehelper
// (src/InsideOutsideAlgorithm.jl:570-635): a stochastic traceback through the
// banded inside tables of scfg.cu.  One warp draws one structure: for a span
// (x, y) with parent nonterminal P it weighs every bifurcation x..h | h+1..y
// (P = S, F) and the pair (x, y) (P = S, F, L) by rule x inside x inside,
// samples one by inverse CDF and pushes the sub-spans on a per-warp stack.
// The log-odds baseline of the banded tables is the same for every option
// of a span, so the weights are the reference's up to a common factor.
// Random numbers: SplitMix64 (Steele, Lea and Flood, OOPSLA 2014) over
// (seed, structure, draw).
#include <algorithm>
#include <climits>
#include <cmath>

#include "decode_schedule.h"
#include "internal.h"
#include "wave.cuh"

namespace messi {

namespace {

__device__ __forceinline__ void amax_merge(float& v, int& k, float v2, int k2)
{
    if (v2 > v || (v2 == v && k2 < k)) {
        v = v2;
        k = k2;
    }
}

}  // namespace

__global__ void to_float_kernel(const double* __restrict__ in, float* __restrict__ out, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)in[i];
}

__global__ void to_double_kernel(const float* __restrict__ in, double* __restrict__ out, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (double)in[i];
}

// ---------------------------------------------------------------------------
// Posterior decoding over tiles of 16 x 16 cells.
// pair: L x L as uploaded from the Julia matrix (column-major); it is read as
// pair[i*L + k], the reference kernel's indexing (the matrix is symmetric).
//
// With a(i,k) = alpha*pair(i,k) + e(i+1,k-1), the value of "i pairs k and
// encloses i+1 .. k-1" (which replaces pair(i,k) in memory once known),
//     e(i,j) = max( single(i) + e(i+1,j), a(i,j), max_{i<k<j} a(i,k) + e(k+1,j) ):
// a product of triangular matrices with max for the sum.  The maximum is exact
// and ties go to the smallest k (the reference's loop order) in whatever order
// the split points are taken, so the bits are the reference kernel's.
//
// CTA b owns the rows of the tiles (I, *), I = b, b + grid, ..., and computes
// them in the order of the tile diagonals D = J - I.  Tile (I, J) needs row
// block I + 1 up to diagonal D - 1, which needed row block I + 2 up to D - 2,
// and so on: a CTA publishes its row block's finished diagonals in a flag
// (release) and waits for the flags of the row blocks it reads next (acquire,
// bounded; decode_schedule.h), not for a grid barrier.  Row index r = k + 1 of
// the second factor:
//   * r in a block R strictly between I and J: both factors lie in finished
//     tiles.  Sixteen groups of 64 threads take every sixteenth R; a thread
//     keeps four cells of the tile and reads e(r, j) from L2 once for all four,
//     a(i, .) from shared memory.  R = I + 1 and I + 2 are usually still in the
//     making when the CTA starts the tile, so they come after the wait for row
//     block I + 1 and the rest before it, behind row block I + 3 up to diagonal
//     D - 3.  That is usually long done, and one thread without cells has seen it
//     during the tile before (a look by every warp at the start of the tile
//     instead: 0.66 ms at L = 1,000);
//   * r in I or J: the factors lie in the tile itself (and in the two diagonal
//     tiles).  A thread per cell; the cells become final along the 31
//     anti-diagonals from the lower left corner, and in every step each cell
//     that is not yet final takes the two values that the last step's cells
//     gave it (without branches: with the split index carried along and the
//     stores inside, a step took 530 cycles).
// Bound by the chain of L/16 waits and 31 steps each; a wavefront with one
// grid barrier per two diagonals of cells took 3.61 ms at L = 1,000, this takes
// 0.63 ms.
// ---------------------------------------------------------------------------
constexpr int kDT = 16;          // cells per tile side
constexpr int kDThreads = 1024;  // 16 groups of 64 threads
constexpr int kDGroups = kDThreads / 64;
constexpr float kDecodeInit = -1e10f;  // the reference's initial maximum (with index 0)

struct DecodeSmem {
    float ad[kDT][kDT + 1];      // a of the row block's diagonal tile
    float ed[kDT][kDT + 1];      // e of the column block's diagonal tile
    float et[kDT + 1][kDT + 2];  // e of the tile: column J*16 - 1 at 0, row I*16 + 16 at 16
    float at[kDT][kDT + 2];      // a of the tile: column J*16 - 1 at 0
    float bv[kDGroups][kDT * kDT];
    int bk[kDGroups][kDT * kDT];
    DecodeWait seen;             // a flag and its value, seen during the tile before
};

// Waits (one thread) until the flag is raised; false once any CTA has given up
// waiting (sync[2], the host's error flag).
__device__ bool flag_look(const unsigned int* flags, DecodeWait w, unsigned int* sync)
{
    unsigned int spins = 0;
    while (ld_acquire_u32(flags + w.block) < (unsigned)w.diagonals)
        if (!keep_waiting(spins, sync)) return false;
    return true;
}

// The whole CTA.
__device__ bool flag_wait(const unsigned int* flags, DecodeWait w, unsigned int* sync)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) s_ok = flag_look(flags, w, sync);
    __syncthreads();
    return s_ok != 0;
}

// A warp, apart from the others.
__device__ __forceinline__ bool flag_wait_warp(const unsigned int* flags, DecodeWait w, unsigned int* sync)
{
    bool ok = true;
    if ((threadIdx.x & 31) == 0) ok = flag_look(flags, w, sync);
    __syncwarp();  // the other lanes' reads behind lane 0's look
    return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ void flag_set(unsigned int* flag, unsigned int v)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(v) : "memory");
    }
}

__device__ __forceinline__ void cells_barrier() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// The diagonal tile of row block I: cell (a, b) by thread 16a + b, span by span.
__device__ void decode_diag_tile(DecodeSmem& S, const float* __restrict__ single, float* A, int L, float alpha, int I,
                                 float* erow, float* ecol, int* scol)
{
    const int a = threadIdx.x >> 4, b = threadIdx.x & 15;
    const int i = I * kDT + a, j = I * kDT + b;
    const bool valid = j < L && b >= a;  // j < L implies i < L
    const float p = (valid && b > a) ? A[(size_t)i * L + j] : 0.f;
    const float si = (i < L) ? __ldg(single + i) : 0.f;
    S.et[a][b] = 0.f;
    S.ad[a][b] = -INFINITY;
    for (int d = 1; d < kDT; d++) {
        cells_barrier();
        if (!valid || b - a != d) continue;
        float bv = kDecodeInit;
        int bk = 0;
        for (int c = a + 1; c < b; c++) {
            const float v = S.ad[a][c] + S.et[c + 1][b];
            if (v > bv) {
                bv = v;
                bk = I * kDT + c;
            }
        }
        const float e2 = __fmaf_rn(alpha, p, S.et[a + 1][b - 1]);
        float mv = si + S.et[a + 1][b];
        int sv = -1;
        if (e2 > mv) {
            mv = e2;
            sv = -2;
        }
        if (bv > mv) {
            mv = bv;
            sv = bk + 1;
        }
        S.et[a][b] = mv;
        S.ad[a][b] = e2;
        erow[(size_t)i * L + j] = mv;
        ecol[(size_t)j * L + i] = mv;
        scol[(size_t)j * L + i] = sv;
    }
    cells_barrier();
    if (valid) A[(size_t)i * L + j] = S.ad[a][b];  // -inf on the diagonal: a column never pairs itself
}

// ROWS: the CTA has one row block whose a(i, r - 1) stay in shared memory at
// arow[a * astride + r] (astride a multiple of 4); otherwise they are read from A.
template <bool ROWS>
__global__ void __launch_bounds__(kDThreads) decode_tile_kernel(const float* __restrict__ single, float* A, int L,
                                                                float alpha, float* erow, float* ecol, int* scol,
                                                                int astride, unsigned int* sync, unsigned int* flags)
{
    __shared__ DecodeSmem S;
    extern __shared__ float4 decode_rows[];
    float* arow = reinterpret_cast<float*>(decode_rows);
    const int NB = (L + kDT - 1) / kDT, tid = threadIdx.x;
    for (int I = blockIdx.x; I < NB; I += gridDim.x) {
        if (tid < 256) {
            decode_diag_tile(S, single, A, L, alpha, I, erow, ecol, scol);
            if (ROWS && I * kDT + (tid & 15) < L) arow[(tid >> 4) * astride + I * kDT + (tid & 15) + 1] = S.ad[tid >> 4][tid & 15];
        }
        flag_set(flags + I, 1u);  // D + 1 finished diagonals
    }
    // phase 1: this thread's cells are (a0 + 4m, b)
    const int grp = tid >> 6, b1 = tid & 15, a0 = (tid >> 4) & 3;
    bool lost = false;  // this warp has given up waiting
    DecodeWait seen{-1, 0};
    for (int D = 1; D < NB; D++) {
        for (int I = blockIdx.x; I + D < NB; I += gridDim.x) {
            const int J = I + D;
            const int j1 = min(J * kDT + b1, L - 1);
            float bv[4];
            int bk[4];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                bv[m] = kDecodeInit;
                bk[m] = 0;
            }
            // rows r0 .. r0 + 4n - 1 of block R, four at a time
            auto block = [&](int r0, int n) {
                float ev[kDT];
#pragma unroll
                for (int x = 0; x < kDT; x++) ev[x] = (x < 4 * n) ? __ldcg(erow + (size_t)(r0 + x) * L + j1) : 0.f;
#pragma unroll
                for (int m = 0; m < 4; m++)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (q >= n) break;
                        const int a = a0 + 4 * m, r = r0 + 4 * q;
                        float4 av;
                        if (ROWS) {
                            av = *reinterpret_cast<const float4*>(arow + a * astride + r);
                        } else {
                            const float* g = A + (size_t)(I * kDT + a) * L + r - 1;
                            av = make_float4(g[0], g[1], g[2], g[3]);
                        }
                        const float v[4] = {av.x + ev[4 * q], av.y + ev[4 * q + 1], av.z + ev[4 * q + 2], av.w + ev[4 * q + 3]};
                        const float best = fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3]));
                        if (best >= bv[m])
                            amax_merge(bv[m], bk[m], best,
                                       r - 1 + (v[0] == best ? 0 : (v[1] == best ? 1 : (v[2] == best ? 2 : 3))));
                    }
            };
            const int R0 = decode_early_first(I) + grp;
            const DecodeWait early = decode_early_wait(I, D);
            // (a warp that has given up goes on: the launch is marked as failed)
            if (R0 < J && !(seen.block == early.block && seen.diagonals >= early.diagonals) && !lost)
                lost = !flag_wait_warp(flags, early, sync);
            for (int R = R0; R < J; R += kDGroups) block(R * kDT, 4);
            if (!flag_wait(flags, decode_late_wait(I, D), sync)) return;
            // cell (a, b) of this thread in the tile, and what it needs from the neighbouring tiles
            const int a = tid >> 4, b = tid & 15, i = I * kDT + a, j = J * kDT + b;
            const int jc = min(j, L - 1);
            float p = 0.f, si = 0.f, ved = 0.f, vrow = 0.f, vcol = 0.f, acol = 0.f, vcorner = 0.f;
            if (tid < 256) {  // every load first: one round trip together with the last blocks'
                p = A[(size_t)i * L + jc];
                si = __ldg(single + i);
                ved = __ldcg(erow + (size_t)min(J * kDT + a, L - 1) * L + jc);
                if (a == 0) vrow = __ldcg(erow + (size_t)((I + 1) * kDT) * L + jc);
                if (b == 0) {
                    vcol = __ldcg(erow + (size_t)i * L + J * kDT - 1);
                    acol = A[(size_t)i * L + J * kDT - 1];
                    if (a == 0) vcorner = __ldcg(erow + (size_t)((I + 1) * kDT) * L + J * kDT - 1);
                }
            }
            // the two blocks next to the diagonal, four rows each by eight groups
            if (grp >= 4 && grp < 12) {
                const int R = I + 1 + ((grp - 4) >> 2);
                if (R < J) block(R * kDT + 4 * (grp & 3), 1);
            }
            if (tid < 256) {
                S.ed[a][b] = ved;
                if (!ROWS) S.ad[a][b] = A[(size_t)i * L + I * kDT + b];
                if (a == 0) S.et[kDT][b + 1] = vrow;
                if (b == 0) {
                    S.et[a][0] = vcol;
                    S.at[a][0] = acol;
                    if (a == 0) S.et[kDT][0] = vcorner;
                }
            }
#pragma unroll
            for (int m = 0; m < 4; m++) {
                S.bv[grp][(a0 + 4 * m) * kDT + b1] = bv[m];
                S.bk[grp][(a0 + 4 * m) * kDT + b1] = bk[m];
            }
            __syncthreads();
            float v1 = kDecodeInit, v = 0.f, e1 = 0.f, e2 = 0.f;
            int k1 = 0;
            if (tid < 256) {
                if (D >= 2)
#pragma unroll 4
                    for (int q = 0; q < kDGroups; q++) amax_merge(v1, k1, S.bv[q][tid], S.bk[q][tid]);
                // k = J*16 - 1, the column before the tile
                amax_merge(v1, k1, S.at[a][0] + S.ed[0][b], J * kDT - 1);
                v = v1;
                const int mine = 15 - a + b;  // the step in which this cell becomes final
                for (int t = 0; t < 2 * kDT - 1; t++) {
                    // the values alone: which split point gave them is looked up afterwards
                    const int ar = kDT + b - t;  // cell (ar, b) became final in step t - 1
                    const int bc = t - kDT + a;  // and so did (a, bc)
                    const float x = (ar >= a + 2 && ar < kDT) ? S.ad[a][ar - 1] + S.et[ar][b + 1] : -INFINITY;
                    const float y = (bc >= 0 && bc < b) ? S.at[a][bc + 1] + S.ed[bc + 1][b] : -INFINITY;
                    v = fmaxf(v, fmaxf(x, y));
                    if (mine == t) {
                        e2 = __fmaf_rn(alpha, p, S.et[a + 1][b]);
                        e1 = si + S.et[a + 1][b + 1];
                        float mv = e1;
                        if (e2 > mv) mv = e2;
                        if (v > mv) mv = v;
                        S.et[a][b + 1] = mv;
                        S.at[a][b + 1] = e2;
                    }
                    cells_barrier();
                }
                if (j < L) {
                    erow[(size_t)i * L + j] = S.et[a][b + 1];
                    A[(size_t)i * L + j] = e2;
                    if (ROWS) arow[a * astride + j + 1] = e2;
                }
            } else if (tid == 256) {
                // what the CTA's next tile waits for first
                const bool more = I + (int)gridDim.x + D < NB;
                const int next = more ? I + (int)gridDim.x : (int)blockIdx.x;
                const int block = min(decode_early_wait(next, more ? D : D + 1).block, NB - 1);
                S.seen = DecodeWait{block, (int)ld_acquire_u32(flags + block)};
            }
            flag_set(flags + I, (unsigned)D + 1u);
            seen = S.seen;  // (written again behind the next tile's barriers)
            // what no other tile reads, while the others' values arrive: the
            // column-major copy and the traceback codes
            if (tid < 256 && j < L) {
                int sv = -1;
                float mv = e1;
                if (e2 > mv) {
                    mv = e2;
                    sv = -2;
                }
                if (v > mv) {
                    for (int c = a + 1; c < kDT - 1; c++) amax_merge(v1, k1, S.ad[a][c] + S.et[c + 1][b + 1], I * kDT + c);
                    for (int c = 0; c < b; c++) amax_merge(v1, k1, S.at[a][c + 1] + S.ed[c + 1][b], J * kDT + c);
                    sv = k1 + 1;
                }
                ecol[(size_t)j * L + i] = S.et[a][b + 1];
                scol[(size_t)j * L + i] = sv;
            }
            // (the next tile writes the shared arrays after its wait, which begins with a CTA barrier)
        }
    }
}

// posteriordecodingtraceback (src/RNATools.jl:43-72) on the column-major s:
// paired[c] = 1-based partner of column c, 0 when unpaired.  One thread;
// stack: 2 * (L + 1) ints of scratch.
__global__ void decode_traceback_kernel(const int* __restrict__ scol, int L, int* __restrict__ paired,
                                        int* __restrict__ stack)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    for (int c = 0; c < L; c++) paired[c] = 0;
    int top = 0;
    stack[top++] = 1;
    stack[top++] = L;
    while (top > 0 && top + 2 <= 2 * (L + 1)) {
        const int j = stack[--top];
        const int i = stack[--top];
        const int k = scol[(size_t)(j - 1) * L + (i - 1)];
        if (k == -1) {
            stack[top++] = i + 1;
            stack[top++] = j;
        } else if (k == -2) {
            paired[i - 1] = j;
            paired[j - 1] = i;
            if (i + 1 < j - 1) {
                stack[top++] = i + 1;
                stack[top++] = j - 1;
            }
        } else if (k > 0 && k <= L) {
            if (i < k) {
                paired[i - 1] = k;
                paired[k - 1] = i;
            }
            if (i + 1 <= k - 1) {
                stack[top++] = i + 1;
                stack[top++] = k - 1;
            }
            if (k + 1 <= j) {
                stack[top++] = k + 1;
                stack[top++] = j;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// structure sampling
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x)
{
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__device__ __forceinline__ double uniform01(unsigned long long seed, unsigned long long stream, unsigned long long n)
{
    const unsigned long long h = splitmix64(splitmix64(seed ^ (stream * 0xD1B54A32D192ED03ull)) + n);
    return (double)(h >> 11) * (1.0 / 9007199254740992.0);
}

// Weight of option o of span (x, y) under parent P (0 = S, 1 = F, 2 = L):
// o < nsplit: bifurcation at h = x + o; o == nsplit: the pair (x, y).
__device__ __forceinline__ float option_weight(const Band& t, const Rules& R, int P, int x, int y, int o, int nsplit)
{
    if (o < nsplit) {
        const int h = x + o;
        const float lv = __ldg(t.Lrow + (size_t)x * t.RS + (h - x));
        const int span = y - h - 1;
        float sv;
        // column layout: consecutive h of a warp read consecutive addresses
        if (span <= t.Wb) sv = __ldg(t.Scol + (size_t)y * t.RS + span);
        else if (y == t.L - 1) sv = __ldg(t.Ssuf + h + 1);
        else sv = -INFINITY;
        return ((P == 0) ? R.r[0] : R.r[4]) + lv + sv;
    }
    const int span = y - x;
    if (span < 2 || span > t.Wb) return -INFINITY;
    const float pv = __ldg(t.pb + (size_t)x * t.RS + span);
    const float fv = __ldg(t.Frow + (size_t)(x + 1) * t.RS + (span - 2));
    return ((P == 0) ? R.r[2] : (P == 1 ? R.r[3] : R.r[6])) + pv + fv;
}

constexpr int kCachedRounds = 32;  // options of a span kept in registers: 32 per lane

// One warp per structure.  stack: [nstruct][3 * (L + 1)] ints;
// paired: [nstruct][L] (1-based partners, 0 = unpaired).
// KH99 log rule probabilities in FP64 (the prior of a sampled structure is
// the sum over its derivation: src/InsideOutsideAlgorithm.jl:86-144 parses
// the same rules, unfolded).
struct PriorRules {
    double r[7];
};

__global__ void __launch_bounds__(128) sample_structures_kernel(Band t, Rules R, PriorRules PR, int nstruct,
                                                                unsigned long long seed, int* __restrict__ paired,
                                                                int* __restrict__ stack, double* __restrict__ prior,
                                                                unsigned int* __restrict__ status)
{
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= nstruct) return;
    const int L = t.L;
    int* out = paired + (size_t)warp * L;
    int* stk = stack + (size_t)warp * 3 * (L + 1);
    for (int c = lane; c < L; c += 32) out[c] = 0;
    __syncwarp();
    int top = 0;  // entries of 3 ints: parent, x, y (kept in lane 0's view; every lane follows)
    if (lane == 0) {
        stk[0] = 0;
        stk[1] = 0;
        stk[2] = L - 1;
    }
    top = 1;
    unsigned long long draw = 0;
    double lp = 0.0;  // log prior of the derivation (lane 0's copy is the result)
    while (top > 0) {
        __syncwarp();
        top--;
        const int P = stk[3 * top], x = stk[3 * top + 1], y = stk[3 * top + 2];
        __syncwarp();
        if (x == y) lp += (P == 0) ? PR.r[1] : (P == 2 ? PR.r[5] : -INFINITY);  // S -> s, L -> s
        if (x >= y) continue;
        // bifurcations x..h | h+1..y with L(x, h) in the band; then the pair.
        // Up to kCached options per span keep their weights in registers (one
        // pass of loads); longer option lists are re-read per pass.
        const int nsplit = (P == 2) ? 0 : min(y - x, t.Wb + 1);
        const int nopt = nsplit + 1;
        const bool cached = nopt <= 32 * kCachedRounds;
        float wv[kCachedRounds];
        float m = -INFINITY;
        if (cached) {
#pragma unroll
            for (int q = 0; q < kCachedRounds; q++) {
                const int o = lane + 32 * q;
                wv[q] = (o < nopt) ? option_weight(t, R, P, x, y, o, nsplit) : -INFINITY;
                m = fmaxf(m, wv[q]);
            }
        } else {
            for (int o = lane; o < nopt; o += 32) m = fmaxf(m, option_weight(t, R, P, x, y, o, nsplit));
        }
        for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
        if (m == -INFINITY) {
            if (lane == 0) atomicOr(status, 2u);  // a span with no derivation: the tables are inconsistent
            break;
        }
        double tot = 0.0;
        if (cached) {
#pragma unroll
            for (int q = 0; q < kCachedRounds; q++) tot += (double)__expf(wv[q] - m);
        } else {
            for (int o = lane; o < nopt; o += 32) tot += (double)__expf(option_weight(t, R, P, x, y, o, nsplit) - m);
        }
        for (int off = 16; off > 0; off >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, off);
        const double target = uniform01(seed, (unsigned long long)warp, draw++) * tot;
        // inverse CDF in rounds of 32 options; if rounding leaves the target
        // past the last cumulative sum, the last option of non-zero weight
        int pick = -1, last = -1;
        double run = 0.0;
        // one round of 32 options: returns true once the pick is found
        auto round = [&](int r0, float wo) {
            const int o = r0 + lane;
            const double w = (o < nopt) ? (double)__expf(wo - m) : 0.0;
            double inc = w;
            for (int off = 1; off < 32; off <<= 1) {
                const double n = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= off) inc += n;
            }
            const unsigned int pos = __ballot_sync(0xffffffffu, w > 0.0);
            if (pos) last = r0 + 31 - __clz((int)pos);
            const unsigned int ball = __ballot_sync(0xffffffffu, (w > 0.0) && (run + inc > target));
            if (ball) {
                pick = r0 + __ffs(ball) - 1;
                return true;
            }
            run += __shfl_sync(0xffffffffu, inc, 31);
            return false;
        };
        if (cached) {
            bool found = false;
#pragma unroll
            for (int q = 0; q < kCachedRounds; q++)
                if (!found && 32 * q < nopt) found = round(32 * q, wv[q]);
        } else {
            for (int r0 = 0; r0 < nopt; r0 += 32)
                if (round(r0, (r0 + lane < nopt) ? option_weight(t, R, P, x, y, r0 + lane, nsplit) : -INFINITY)) break;
        }
        if (pick < 0) pick = last;
        const int npush = (pick < nsplit) ? 2 : 1;
        if (pick < 0 || top + npush > L) {
            if (lane == 0) atomicOr(status, 4u);
            break;
        }
        if (pick < nsplit) lp += (P == 0) ? PR.r[0] : PR.r[4];                   // S -> LS, F -> LS
        else lp += (P == 0) ? PR.r[2] : (P == 1 ? PR.r[3] : PR.r[6]);            // pair rules
        if (lane == 0) {
            if (pick < nsplit) {
                const int h = x + pick;
                // the reference pushes the left part, then the right part
                stk[3 * top] = 2;  // L(x, h)
                stk[3 * top + 1] = x;
                stk[3 * top + 2] = h;
                stk[3 * top + 3] = 0;  // S(h+1, y)
                stk[3 * top + 4] = h + 1;
                stk[3 * top + 5] = y;
            } else {
                out[x] = y + 1;
                out[y] = x + 1;
                stk[3 * top] = 1;  // F(x+1, y-1)
                stk[3 * top + 1] = x + 1;
                stk[3 * top + 2] = y - 1;
            }
        }
        top += npush;
    }
    if (lane == 0 && prior) prior[warp] = lp;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
size_t decode_sync_words(int L) { return (size_t)kSyncWords + (L + kDT - 1) / kDT; }

int run_posterior_decoding(messi_ctx* ctx, int L, const double* d_single, const double* d_pair, double alpha,
                           float* d_work, int* d_scol, unsigned int* d_sync, int* d_paired, int* d_stack,
                           double* d_eout)
{
    // d_work: single (L) | pair (L*L) | erow (L*L) | ecol (L*L) floats
    const long long LL = (long long)L * L;
    float* f_single = d_work;
    float* f_pair = d_work + L;
    float* erow = f_pair + LL;
    float* ecol = erow + LL;
    const int bs = 256;
    to_float_kernel<<<(unsigned)((L + bs - 1) / bs), bs, 0, ctx->stream>>>(d_single, f_single, L);
    LAUNCH_CHECK(ctx, "to_float_kernel");
    to_float_kernel<<<(unsigned)((LL + bs - 1) / bs), bs, 0, ctx->stream>>>(d_pair, f_pair, LL);
    LAUNCH_CHECK(ctx, "to_float_kernel");
    cudaError_t e = cudaMemsetAsync(erow, 0, sizeof(float) * 2 * LL, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_scol, 0, sizeof(int) * LL, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_sync, 0, decode_sync_words(L) * sizeof(unsigned int), ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "decoding tables reset");
    if (L > 1) {
        const float a = (float)alpha;
        int Lv = L;
        const int NB = (L + kDT - 1) / kDT;
        // one CTA per row block where the GPU holds that many; its rows of a
        // then stay in shared memory if they fit
        int sms = ctx->num_sms;
        if (sms <= 0) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
        int grid = std::min(NB, std::max(1, sms));
        if (ctx->wave_ctas > 0) grid = std::min(grid, ctx->wave_ctas);
        int astride = NB * kDT + 4;
        unsigned int* d_flags = d_sync + kSyncWords;
        const size_t bytes = (size_t)kDT * astride * sizeof(float);
        const bool rows = grid == NB && bytes <= (size_t)160 * 1024;
        const void* kernel = rows ? (const void*)decode_tile_kernel<true> : (const void*)decode_tile_kernel<false>;
        if (rows) {
            e = allow_smem(ctx->device, kernel, bytes);
            if (e != cudaSuccess) return cuda_fail(ctx, e, "decode_tile_kernel attributes");
        }
        void* args[] = {(void*)&f_single, (void*)&f_pair, &Lv, (void*)&a, &erow, &ecol, &d_scol, &astride, &d_sync, &d_flags};
        e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kDThreads), args, rows ? bytes : 0, ctx->stream);
        ctx->launches++;
        if (e != cudaSuccess) return cuda_fail(ctx, e, "decode_tile_kernel");
    }
    if (d_paired) {
        decode_traceback_kernel<<<1, 32, 0, ctx->stream>>>(d_scol, L, d_paired, d_stack);
        LAUNCH_CHECK(ctx, "decode_traceback_kernel");
    }
    if (d_eout) {
        // the column-major copy is the Julia matrix e[i, j] (zeros below the diagonal)
        to_double_kernel<<<(unsigned)((LL + bs - 1) / bs), bs, 0, ctx->stream>>>(ecol, d_eout, LL);
        LAUNCH_CHECK(ctx, "to_double_kernel");
    }
    return queue_status(ctx, d_sync + 2);
}

int run_sample_structures(messi_ctx* ctx, const Band& t, double B, int nstruct, unsigned long long seed,
                          int* d_paired, int* d_stack, double* d_prior, unsigned int* d_status)
{
    Rules R = make_rules(B);
    PriorRules PR;
    for (int k = 0; k < 7; k++) PR.r[k] = std::log(kKH99Prob[k]);
    cudaError_t e = cudaMemsetAsync(d_status, 0, sizeof(unsigned int), ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "sampler status reset");
    const int warps_per_block = 4;
    const int blocks = (nstruct + warps_per_block - 1) / warps_per_block;
    sample_structures_kernel<<<blocks, 32 * warps_per_block, 0, ctx->stream>>>(t, R, PR, nstruct, seed, d_paired,
                                                                                d_stack, d_prior, d_status);
    LAUNCH_CHECK(ctx, "sample_structures_kernel");
    return MESSI_OK;
}

}  // namespace messi
