// Values that are their own ready marks.  A buffer starts as a signalling-NaN bit pattern that no
// arithmetic can produce (results of operations are quiet NaNs, and stores check); a reader polls
// the value itself until it is something else, and a producer needs no flag and no fence: 64-bit
// accesses are single, and no value vouches for another.
#pragma once

#include "bpf_internal.cuh"

namespace bpf {

constexpr unsigned long long kPending = 0x7FF4B0F5B0F5B0F5ull;   // signalling NaN

__device__ __forceinline__ double pending_value() { return __longlong_as_double((long long)kPending); }
__device__ __forceinline__ bool is_pending(double v) { return (unsigned long long)__double_as_longlong(v) == kPending; }
__device__ __forceinline__ double not_pending(double v) {
    return is_pending(v) ? __longlong_as_double(0x7FF8000000000000ll) : v;
}
__device__ __forceinline__ double ld_value(const double *p) {
    unsigned long long b;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b) : "l"(p) : "memory");
    return __longlong_as_double((long long)b);
}
// v = *p once it is not pending; false if the wait gave up (lim polls, or a recorded error).
__device__ __forceinline__ bool poll_value(const double *p, double &v, long long lim, const DevStatus *ds) {
    long long it = 0;
    while (is_pending(v = ld_value(p))) {
        if (++it > lim || ((it & 31) == 0 && ld_relaxed_i32(&ds->err) != 0)) return false;
        __nanosleep(20);
    }
    return true;
}

}  // namespace bpf
