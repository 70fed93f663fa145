// pp_bond_f64.cuh -- binary64 per-bond arithmetic shared by the plain and
// fused FP64 kernels.
//
// Restates the per-work-item body of bond_force1..4
// (peripy/cl/peridynamics.cl:61-102, 193-233, 323-385, 474-536) with exact
// round-to-nearest intrinsics and the reference association order:
//   xi   = r0[j] - r0[i]                           (:65-67)
//   xe   = (u[j] - u[i]) + xi                      (:69-71)
//   |xi| = sqrt((x*x + y*y) + z*z), |xe| likewise  (:73-74)
//   s    = (|xe| - |xi|) / |xi|                    (:75)
//   PMB:      intact iff s < s0, f = (s*k)[*corr]*vol[j]            (:78-83, :214)
//   n-linear: regime moves by at most one, breaks at r >= nregimes,
//             f = ((s*k[r] + c[r])[*corr])*vol[j]                     (:345-373, :524)
//   force component = f * (xe / |xe|)                                (:79-87)
#pragma once

#include "pp_common.cuh"
#include "pp_exact64.cuh"

namespace pp {

struct F64Bond {
    const double* r0;
    const double* u;
    const double* vols;
    int32_t* nlist;
    const double* sc;         // stiffness corrections or nullptr
    const int32_t* btypes;    // bond types or nullptr
    int32_t* regimes;
    const double* ktab;
    const double* stab;
    const double* ctab;
    const double* xi_len;     // per-slot |xi| (pp_bond_lengths) or nullptr
    double k;
    double s0;
    int nregimes;
};

// Stretch and direction cosines of one bond: s = (y - xi) / xi, q = xe / y.
struct F64Stretch {
    double s, qx, qy, qz;
};

// By the binary64 pipe's own operations: any inputs.
static __device__ __noinline__ void f64_stretch_any(double x, double y, double z, double sq,
                                                    double xi, F64Stretch* out) {
    const double len = dsqrt(sq);
    out->s = ddiv(dsub(len, xi), xi);
    out->qx = ddiv(x, len);
    out->qy = ddiv(y, len);
    out->qz = ddiv(z, len);
}

// The same values by pp_exact64.cuh, which needs no binary64 instruction for
// the root, the difference and the four quotients: ~140 clocks a warp and
// slot of the integer and FP32 pipes instead of ~720 of the binary64 pipe,
// which the other operations of the slot keep busy.  It takes lengths within
// 2^+-200 (squares 2^+-400) that differ by less than a factor of two, and
// components that are zero or above 2^-700, so that no intermediate is
// subnormal or overflows; everything else (NaN and infinities among it)
// goes to f64_stretch_any.
__device__ __forceinline__ F64Stretch f64_stretch(double x, double y, double z, double sq,
                                                  double xi) {
    using namespace exact64;
    const uint64_t xb = double_bits(x), yb = double_bits(y), zb = double_bits(z);
    const uint64_t sb = double_bits(sq), lb = double_bits(xi);
    F64Stretch r;
    uint64_t s;
    bool ok = exponent_in(sb, 1023 - 400, 1023 + 400) && exponent_in(lb, 1023 - 200, 1023 + 200) &&
              (lb >> 63) == 0 && zero_or_above(xb, 1023 - 700) && zero_or_above(yb, 1023 - 700) &&
              zero_or_above(zb, 1023 - 700);
    if (ok) {
        const Divisor len = sqrt_rn(sb);
        ok = relative_difference(len, divisor(lb), s);
        r.s = bits_double(s);
        r.qx = div_signed(xb, len);
        r.qy = div_signed(yb, len);
        r.qz = div_signed(zb, len);
    }
    if (!ok) {
        F64Stretch t;
        f64_stretch_any(x, y, z, sq, xi, &t);
        r = t;
    }
    return r;
}

// |xi| from the squared length, correctly rounded.
__device__ __forceinline__ double f64_length(double sq) {
    using namespace exact64;
    const uint64_t sb = double_bits(sq);
    if (!exponent_in(sb, 1023 - 400, 1023 + 400) || (sb >> 63)) return dsqrt(sq);
    const Divisor d = sqrt_rn(sb);
    return bits_double(pack(d.m, d.e));
}

static __device__ __noinline__ bool f64_less_any(double a, double b) { return a < b; }

// a < b.  A binary64 comparison is an instruction of the binary64 pipe too:
// with b positive and neither a NaN, the bits compare as signed integers.
__device__ __forceinline__ bool f64_less(double a, double b) {
    const int64_t ab = __double_as_longlong(a), bb = __double_as_longlong(b);
    constexpr uint64_t kInf = 0x7FF0000000000000ull;
    if ((uint64_t)(bb - 1) < kInf && ((uint64_t)ab << 1) <= (kInf << 1)) return ab < bb;
    return f64_less_any(a, b);
}

// Contribution of slot `gid` of node i.  Breaks the bond / moves its regime
// in place exactly as the reference kernel does; counts intact bonds.
template <bool CORR, bool TYPES>
__device__ __forceinline__ d3 f64_slot(const F64Ops& op, const F64Bond& b, int64_t gid, d3 ri, d3 ui,
                                       int& intact) {
    const int j = b.nlist[gid];
    if (j == -1) return d3_zero();
    const double* rj = b.r0 + 3 * (int64_t)j;
    const double* uj = b.u + 3 * (int64_t)j;
    const double xi_x = op.sub(rj[0], ri.x);
    const double xi_y = op.sub(rj[1], ri.y);
    const double xi_z = op.sub(rj[2], ri.z);
    const double xe_x = op.add(op.sub(uj[0], ui.x), xi_x);
    const double xe_y = op.add(op.sub(uj[1], ui.y), xi_y);
    const double xe_z = op.add(op.sub(uj[2], ui.z), xi_z);
    // |xi| never changes: read it when cached (the same binary64 value)
    const double xi = b.xi_len ? b.xi_len[gid]
                               : f64_length(op.add(op.add(op.mul(xi_x, xi_x), op.mul(xi_y, xi_y)),
                                                 op.mul(xi_z, xi_z)));
    const F64Stretch st = f64_stretch(
        xe_x, xe_y, xe_z, op.add(op.add(op.mul(xe_x, xe_x), op.mul(xe_y, xe_y)), op.mul(xe_z, xe_z)), xi);
    const double s = st.s;
    double f;
    if constexpr (!TYPES) {
        if (!f64_less(s, b.s0)) {
            b.nlist[gid] = -1;
            return d3_zero();
        }
        f = op.mul(s, b.k);
        if constexpr (CORR) f = op.mul(f, b.sc[gid]);
        f = op.mul(f, b.vols[j]);
    } else {
        const int nr = b.nregimes;
        const int base = b.btypes[gid] * nr;
        int r = b.regimes[gid];
        // A valid bond always has 0 <= r < nregimes; clamp the table reads
        // so that a malformed regimes array cannot read out of bounds.
        const int rc = r < 0 ? 0 : (r >= nr ? nr - 1 : r);
        if (f64_less(s, b.stab[base + rc])) {
            if (r > 0 && rc > 0) {
                if (f64_less(s, b.stab[base + rc - 1])) {
                    r -= 1;
                    b.regimes[gid] = r;
                }
            }
        } else {
            r += 1;
            b.regimes[gid] = r;
        }
        if (r >= nr) {
            b.nlist[gid] = -1;
            return d3_zero();
        }
        const int rr = r < 0 ? 0 : r;
        f = op.add(op.mul(s, b.ktab[base + rr]), b.ctab[base + rr]);
        if constexpr (CORR) f = op.mul(f, b.sc[gid]);
        f = op.mul(f, b.vols[j]);
    }
    intact += 1;
    return d3{op.mul(f, st.qx), op.mul(f, st.qy), op.mul(f, st.qz)};
}

// Euler update of one DOF (peripy/cl/euler.cl:23).
__device__ __forceinline__ double euler_u(double u, double f, int bct, double bcv,
                                          double bc_scale, double dt) {
    return bct == 0 ? dadd(u, dmul(dt, f)) : dmul(bc_scale, bcv);
}

// Euler-Cromer update of one DOF (peripy/cl/euler_cromer.cl:55-58).
__device__ __forceinline__ double euler_cromer_u(double u, double& ud, double& udd, double f,
                                                 int bct, double bcv, double rho,
                                                 double bc_scale, double damping,
                                                 double dt) {
    const double uddi = ddiv(dsub(f, dmul(damping, ud)), rho);
    udd = uddi;
    ud = dadd(ud, dmul(uddi, dt));
    return bct == 0 ? dadd(u, dmul(dt, ud)) : dmul(bc_scale, bcv);
}

// Velocity-Verlet update of one DOF (peripy/cl/velocity_verlet.cl:90-94).
__device__ __forceinline__ double velocity_verlet_u(double u, double& ud, double& udd,
                                                    double f, int bct, double bcv,
                                                    double rho, double bc_scale,
                                                    double damping, double dt) {
    const double half = dmul(dt, 0.5);  // dt / 2
    const double ud1 = dadd(ud, dmul(half, udd));
    const double udd1 = ddiv(dsub(f, dmul(damping, ud1)), rho);
    ud = dadd(ud1, dmul(half, udd1));
    udd = udd1;
    return bct == 0 ? dadd(u, dmul(dt, dadd(ud, dmul(half, udd1)))) : dmul(bc_scale, bcv);
}

// Force with the force boundary condition (peridynamics.cl:127-129).
__device__ __forceinline__ double force_with_bc(double body, int fct, double fcv,
                                                double fc_scale) {
    return fct == 0 ? body : dadd(body, dmul(fc_scale, fcv));
}

// Damage of one node (peridynamics.cl:606-608).
__device__ __forceinline__ double damage_of(int intact, int family) {
    return dsub(1.0, ddiv((double)intact, (double)family));
}

}  // namespace pp
