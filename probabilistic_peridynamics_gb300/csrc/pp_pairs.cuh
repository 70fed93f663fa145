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

// Reference vector of pair p, r0[j] - r0[i] as pp_pair_fill kept it.
__device__ __forceinline__ d3 pair_reference(const pp_pairs& pr, int64_t p) {
    return d3{pr.vector[p], pr.vector[pr.npairs + p], pr.vector[2 * pr.npairs + p]};
}

// The record at p where `live`, else +0 (without a branch around the load).  Not
// a read-only load: a dependent launch may begin before the records are written.
__device__ __forceinline__ d3 load_record_if(const double* p, bool live) {
    d3 v{0.0, 0.0, 0.0};
    [[maybe_unused]] double w = 0.0;
    asm("{\n\t.reg .pred live;\n\t"
        "setp.ne.s32 live, %5, 0;\n\t"
        "@live ld.global.v4.f64 {%0, %1, %2, %3}, [%4];\n\t}"
        : "+d"(v.x), "+d"(v.y), "+d"(v.z), "+d"(w)
        : "l"(p), "r"((int)live));
    return v;
}

// The record at p as slot `sp` sees it: negated for a pair's second slot, +0
// for sp = -1.  By bits: a selected negation is an instruction of the
// binary64 pipe.  (A component that is zero gets the other sign of zero than the
// slot's own product has: equal as a number, and so are the sums.)
__device__ __forceinline__ d3 signed_record(const double* p, int sp) {
    const d3 v = load_record_if(p, sp != -1);
    const long long flip = sp < -1 ? (long long)0x8000000000000000ull : 0;
    return d3{__longlong_as_double(__double_as_longlong(v.x) ^ flip),
              __longlong_as_double(__double_as_longlong(v.y) ^ flip),
              __longlong_as_double(__double_as_longlong(v.z) ^ flip)};
}

}  // namespace pp
