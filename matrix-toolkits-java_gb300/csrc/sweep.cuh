// sweep.cuh -- what the triangular sweeps share (precond.cu: one ticket per
// chunk of a level; lines.cu: one CTA per tile of lines): the pending value
// that marks an x entry as not yet solved, relaxed loads and stores, and the
// bounded wait for an entry.
#pragma once

#include "dev.cuh"

namespace mtjg {

// x entries not yet solved hold this signalling NaN (FP64; kPending32 in the
// FP32 sweeps of the mixed-precision inner solves).
constexpr unsigned long long kPending = 0x7FF40000DEADBEEFull;
constexpr unsigned long long kQuietNaN = 0x7FF8000000000000ull;
constexpr unsigned kPending32 = 0x7FA0BEEFu;
constexpr unsigned kQuietNaN32 = 0x7FC00000u;
constexpr long long kSweepSpinLimit = 1LL << 21;

__device__ __forceinline__ double ld_relaxed(const double *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return __longlong_as_double((long long)v);
}

__device__ __forceinline__ void st_relaxed(double *p, double v)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"((unsigned long long)__double_as_longlong(v))
                 : "memory");
}

__device__ __forceinline__ float ld_relaxed(const float *p)
{
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return __uint_as_float(v);
}

__device__ __forceinline__ void st_relaxed(float *p, float v)
{
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(__float_as_uint(v)) : "memory");
}

__device__ __forceinline__ bool pending(double v) { return (unsigned long long)__double_as_longlong(v) == kPending; }
__device__ __forceinline__ bool pending(float v) { return __float_as_uint(v) == kPending32; }
template <class T>
__device__ __forceinline__ T pending_value();
template <>
__device__ __forceinline__ double pending_value<double>() { return __longlong_as_double((long long)kPending); }
template <>
__device__ __forceinline__ float pending_value<float>() { return __uint_as_float(kPending32); }
// a result that happens to carry the pending pattern is stored as a quiet NaN
__device__ __forceinline__ double unpend(double v) { return pending(v) ? __longlong_as_double((long long)kQuietNaN) : v; }
__device__ __forceinline__ float unpend(float v) { return pending(v) ? __uint_as_float(kQuietNaN32) : v; }

// x_c for a row of the sweep: a relaxed load, polled while it is pending.
// Gives up (bad) after kSweepSpinLimit polls or when another wait has given
// up (the context's error flag is set).
template <class T>
__device__ __forceinline__ T wait_x(const T *x, int c, const int *err, int spin, bool &bad)
{
    T v = ld_relaxed(x + c);
    if (!pending(v)) return v;
    unsigned ns = 32;
    for (long long polls = 1;; ++polls) {
        if (polls > spin) {
            __nanosleep(ns);
            ns = ns < 256 ? 2 * ns : ns;
        }
        v = ld_relaxed(x + c);
        if (!pending(v)) return v;
        if (polls > kSweepSpinLimit || ((polls & 31) == 0 && *(volatile const int *)err)) {
            bad = true;
            return T(0);
        }
    }
}

}  // namespace mtjg
