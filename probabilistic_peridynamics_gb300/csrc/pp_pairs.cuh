// pp_pairs.cuh -- records of a pair list (pp_pairs.cu, pp_adjoint.cu).
#pragma once

#include "pp_bond_f64.cuh"

namespace pp {

constexpr int kReversed = (int)0x80000000u;  // slot_pair: the pair's second slot

__device__ __forceinline__ void store_record(double* p, const d3& v) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v.x), "d"(v.y), "d"(v.z),
                 "d"(0.0)
                 : "memory");
}

__device__ __forceinline__ d3 load_record(const double* p) {
    d3 v;
    [[maybe_unused]] double w;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(w)
        : "l"(p));
    return v;
}

// The record at p as slot `sp` sees it: negated for a pair's second slot.  By
// bits: a selected negation is an instruction of the binary64 pipe.
__device__ __forceinline__ d3 signed_record(const double* p, int sp) {
    const d3 v = load_record(p);
    const long long flip = sp < 0 ? (long long)0x8000000000000000ull : 0;
    return d3{__longlong_as_double(__double_as_longlong(v.x) ^ flip),
              __longlong_as_double(__double_as_longlong(v.y) ^ flip),
              __longlong_as_double(__double_as_longlong(v.z) ^ flip)};
}

}  // namespace pp
