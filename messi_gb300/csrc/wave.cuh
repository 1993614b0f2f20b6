// wave.cuh -- device helpers shared by the persistent wavefront kernels
// (SCFG inside/outside, posterior decoding): bounded waits and the split-sum
// group width.
#pragma once

#include "internal.h"

namespace messi {

// each spin is an L2 round trip, later plus a 32 ns sleep (~0.3-0.5 us): a wait
// gives up after one to two seconds
constexpr unsigned int kSpinLimit = 1u << 22;

static __device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* p)
{
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Dataflow waits: a table of FP32 cells filled with kUnwritten before the
// launch, whose cells are their own flags.  The bits are a NaN that no
// arithmetic gives (those are 0x7fffffff), so a cell is complete exactly when
// it reads as anything else, and no fence or barrier need order its write with
// another.  Reads and writes are relaxed at device scope (L2).
constexpr unsigned int kUnwritten = 0xffffffffu;

static __device__ __forceinline__ bool unwritten(float v) { return __float_as_uint(v) == kUnwritten; }

static __device__ __forceinline__ float ld_cell(const float* p)
{
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}

static __device__ __forceinline__ void st_cell(float* p, float v)
{
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

// One more failed look at cells that are not there yet: false (and the
// launch marked failed) once the waiting has taken one to two seconds, or
// some other CTA has given up.
static __device__ __forceinline__ bool keep_waiting(unsigned int& spins, unsigned int* sync,
                                                    unsigned int limit = kSpinLimit)
{
    if (++spins > limit || ((spins & 1023u) == 0u && ld_acquire_u32(&sync[2]) != 0u)) {
        atomicExch(&sync[2], 1u);
        return false;
    }
    if (spins > 64u) __nanosleep(32);
    return true;
}

// The same for a whole warp that waits together: one decision for all 32 lanes.
// Their own looks at sync[2] may differ, and a lane that left alone would leave
// the others in the warp's votes for ever.
static __device__ __forceinline__ bool warp_keep_waiting(unsigned int& spins, unsigned int* sync,
                                                         unsigned int limit = kSpinLimit)
{
    return __all_sync(0xffffffffu, keep_waiting(spins, sync, limit));
}

// Lanes per cell for a split sum of `nterms` terms: at most 8 terms per lane
// up to 256 terms, so a lane's loads are issued together and the sum costs
// one L2 round trip; longer sums use the whole warp.
static __device__ __forceinline__ int group_width(int nterms)
{
    return nterms <= 8 ? 1 : (nterms <= 16 ? 2 : (nterms <= 32 ? 4 : (nterms <= 64 ? 8 : (nterms <= 128 ? 16 : 32))));
}

}  // namespace messi
