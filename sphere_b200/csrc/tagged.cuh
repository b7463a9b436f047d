// Cell values that carry the iteration they belong to, for the Darcy solver's
// Jacobi kernel.
//
// An iteration of that kernel is a few hundred nanoseconds of arithmetic per
// cell, so its cost is the hand-over of the iterates between thread blocks.
// With a flag per block that hand-over is a fence, a store, a poll, a block
// barrier and then the loads; here the value is its own flag: a cell's new
// value and its iteration number go out in one 16-byte store, and a reader
// polls its neighbours' cells until they carry the iteration it needs.  No
// fence and no barrier is left on the path.  One 128-bit access is single-copy
// atomic (PTX ld / st .relaxed.b128), so value and number always match.
//
// Two buffers suffice (iterate i in buffer i & 1): a cell's iterate i + 2
// overwrites its iterate i only after the cell has read iterate i + 1 of its
// neighbours, which they wrote after reading its iterate i; neighbourhoods are
// symmetric.  Numbers are unique over all launches of an engine (launch
// sequence << 32 | iterate), so the buffers are never cleared.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "dev_common.cuh"

namespace sphb {

struct __align__(16) TaggedValue {
    double v;
    unsigned long long tag;
};

__device__ __forceinline__ void tagged_store(TaggedValue *p, double v, unsigned long long tag)
{
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }"
                 :: "l"(p), "l"(__double_as_longlong(v)), "l"(tag) : "memory");
}

__device__ __forceinline__ TaggedValue tagged_load(const TaggedValue *p)
{
    long long v;
    TaggedValue r;
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(v), "=l"(r.tag) : "l"(p) : "memory");
    r.v = __longlong_as_double(v);
    return r;
}

// Global part of the stop rule (zero at launch): maxima of the residuals per
// iteration (bit patterns of non-negative doubles, all ones for a NaN) and the
// number of warps that have reported a check iteration.
constexpr unsigned kFlowRing = 64;
struct FlowSync {
    unsigned long long ring[kFlowRing];
    unsigned arrived;
    unsigned active;          // cells that change during the solve
};

// Largest 64-bit value of a warp, in every lane.
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v)
{
    const unsigned hi = (unsigned)(v >> 32);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)v : 0u);
    return (unsigned long long)mh << 32 | ml;
}

// x / d for a divisor whose correctly rounded reciprocal r is at hand
// (Markstein, IBM Journal of Research and Development 34, 1990: with r =
// RN(1/d), a quotient within one unit and its exact remainder, one fused
// correction rounds as the division does; the first correction brings the
// quotient within one unit).  Operands outside the range in which the
// remainders are exact take the division.
__host__ __device__ __forceinline__ double div_by(double x, double d, double r)
{
    const double a = fabs(x);
    if (!(a > 1e-200 && a < 1e200)) return x / d;
    double q = x * r;
    q = fma(fma(-q, d, x), r, q);
    return fma(fma(-q, d, x), r, q);
}

}  // namespace sphb
