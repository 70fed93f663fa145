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
#include "pp_fused.cuh"

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

using F64Stretch = exact64::Stretch;

// By the binary64 pipe's own operations: any inputs.
static __device__ __noinline__ void f64_stretch_any(double x, double y, double z, double xi,
                                                    F64Stretch* out) {
    using exact64::double_bits;
    const double len = dsqrt(dadd(dadd(dmul(x, x), dmul(y, y)), dmul(z, z)));
    out->s = double_bits(ddiv(dsub(len, xi), xi));
    out->qx = double_bits(ddiv(x, len));
    out->qy = double_bits(ddiv(y, len));
    out->qz = double_bits(ddiv(z, len));
}

struct F64StretchAny {
    __device__ __forceinline__ void operator()(double x, double y, double z, double xi,
                                               F64Stretch* out) const {
        f64_stretch_any(x, y, z, xi, out);
    }
};

// The same values by pp_exact64.cuh where it takes the operands: ~140 clocks a
// warp and slot of the integer and FP32 pipes instead of ~720 of the binary64
// pipe, which the other operations of the slot keep busy.
//
// kIntSquares: the three squares on the integer pipe too.  The one-kernel
// steps, with 23 binary64 operations a slot, gain by it (400,000 nodes in rows of
// 128 slots: plain 2.51 -> 2.09 ms, fused 1.99 -> 1.97; 90,000 in rows of 32: 170 ->
// 157 us, fused 165 -> 152); the pair step, with 16, does not.
template <bool kIntSquares>
__device__ __forceinline__ F64Stretch f64_stretch(const F64Ops& op, const d3& xe, double xi) {
    return exact64::stretch<kIntSquares>(op, xe, xi, F64StretchAny());
}

// |xi| from the squared length, correctly rounded.
__device__ __forceinline__ double f64_length(double sq) {
    using namespace exact64;
    const uint64_t sb = double_bits(sq);
    if (!positive_in(sb, 1023 - 400, 1023 + 400)) return dsqrt(sq);
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

// The damage law of the bond in slot `gid` at stretch s, towards a neighbour
// of volume vol: breaks the bond / moves its regime in place exactly as the
// reference kernel does.  True when the bond stays; f is then its force.
template <bool CORR, bool TYPES>
__device__ __forceinline__ bool f64_bond_law(const F64Ops& op, const F64Bond& b, int64_t gid,
                                             double s, double vol, double& f) {
    if constexpr (!TYPES) {
        if (!f64_less(s, b.s0)) {
            b.nlist[gid] = -1;
            return false;
        }
        f = op.mul(s, b.k);
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
            return false;
        }
        const int rr = r < 0 ? 0 : r;
        f = op.add(op.mul(s, b.ktab[base + rr]), b.ctab[base + rr]);
    }
    if constexpr (CORR) f = op.mul(f, b.sc[gid]);
    f = op.mul(f, vol);
    return true;
}

// Reference vector of the bond to node j, ri = r0 of its other node.
__device__ __forceinline__ d3 f64_reference(const F64Ops& op, const double* r0, int j, d3 ri) {
    const double* rj = r0 + 3 * (int64_t)j;
    return d3{op.sub(rj[0], ri.x), op.sub(rj[1], ri.y), op.sub(rj[2], ri.z)};
}

// The deformed vector.
__device__ __forceinline__ d3 f64_deformed(const F64Ops& op, const double* u, int j, d3 ui,
                                           const d3& xi) {
    const double* uj = u + 3 * (int64_t)j;
    return d3{op.add(op.sub(uj[0], ui.x), xi.x), op.add(op.sub(uj[1], ui.y), xi.y),
              op.add(op.sub(uj[2], ui.z), xi.z)};
}

__device__ __forceinline__ double f64_square(const F64Ops& op, const d3& v) {
    return op.add(op.add(op.mul(v.x, v.x), op.mul(v.y, v.y)), op.mul(v.z, v.z));
}

__device__ __forceinline__ d3 f64_force(const F64Ops& op, double f, const F64Stretch& st) {
    return d3{op.mul(f, __longlong_as_double(st.qx)), op.mul(f, __longlong_as_double(st.qy)),
              op.mul(f, __longlong_as_double(st.qz))};
}

// Contribution of slot `gid` of node i; counts intact bonds.
template <bool CORR, bool TYPES>
__device__ __forceinline__ d3 f64_slot(const F64Ops& op, const F64Bond& b, int64_t gid, d3 ri,
                                       d3 ui, int& intact) {
    const int j = b.nlist[gid];
    if (j == -1) return d3_zero();
    const d3 xi = f64_reference(op, b.r0, j, ri);
    const d3 xe = f64_deformed(op, b.u, j, ui, xi);
    // |xi| never changes: read it when cached (the same binary64 value)
    const double len = b.xi_len ? b.xi_len[gid] : f64_length(f64_square(op, xi));
    const F64Stretch st = f64_stretch<true>(op, xe, len);
    double f;
    if (!f64_bond_law<CORR, TYPES>(op, b, gid, __longlong_as_double(st.s), b.vols[j], f))
        return d3_zero();
    intact += 1;
    return f64_force(op, f, st);
}

static __device__ __noinline__ double f64_divide_any(double a, double b) { return ddiv(a, b); }

// a / b: on the integer pipe where a and b are within 2^+-400 (a may be
// zero) and b is positive, as densities are; else the binary64 pipe's own.
__device__ __forceinline__ double f64_divide(double a, double b) {
    using namespace exact64;
    const uint64_t ab = double_bits(a), bb = double_bits(b);
    const bool ok = positive_in(bb, 1023 - 400, 1023 + 400) &&
                    (is_zero(ab) || positive_in(ab & 0x7FFFFFFFFFFFFFFFull, 1023 - 400, 1023 + 400));
    if (!ok) return f64_divide_any(a, b);
    return div_signed(ab, divisor(bb));
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
    const double uddi = f64_divide(dsub(f, dmul(damping, ud)), rho);
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
    const double udd1 = f64_divide(dsub(f, dmul(damping, ud1)), rho);
    ud = dadd(ud1, dmul(half, udd1));
    udd = udd1;
    return bct == 0 ? dadd(u, dmul(dt, dadd(ud, dmul(half, udd1)))) : dmul(bc_scale, bcv);
}

// Force with the force boundary condition (peridynamics.cl:127-129).
__device__ __forceinline__ double force_with_bc(double body, int fct, double fcv,
                                                double fc_scale) {
    return fct == 0 ? body : dadd(body, dmul(fc_scale, fcv));
}

// Damage of one node (peridynamics.cl:606-608): 1 - intact / family.  The
// integers become significands directly (a conversion is an instruction of
// the binary64 pipe).
__device__ __forceinline__ double damage_of(int intact, int family) {
    using namespace exact64;
    if (family <= 0 || intact < 0) return dsub(1.0, ddiv((double)intact, (double)family));
    if (intact == 0) return 1.0;
    return dsub(1.0, div_signed(int_bits(intact), divisor(int_bits(family))));
}

// The inputs of a block's node updates, copied to shared memory by cp.async
// while the block computes its bonds: their load latency (and no registers)
// is then hidden behind the bond phase.
constexpr int kMaxNodes = 8;  // nodes (warps) per block
struct NodeStage {
    double u[3 * kMaxNodes], ud[3 * kMaxNodes], udd[3 * kMaxNodes], rho[3 * kMaxNodes];
    double bcv[3 * kMaxNodes], fcv[3 * kMaxNodes];
    double sum[3 * kMaxNodes];  // bond forces
    int bct[3 * kMaxNodes], fct[3 * kMaxNodes];
    int family[kMaxNodes], count[kMaxNodes];
};

template <int Bytes>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(s), "l"(gmem), "n"(Bytes)
                 : "memory");
}

// Started by the block's first threads, one per DOF; f64_node_phase waits.
__device__ __forceinline__ void f64_stage_nodes(const pp_fused_args& a, int parity, int node0,
                                                int nodes, NodeStage& s) {
    const int t = threadIdx.x;
    if (t < 3 * nodes && node0 + t / 3 < a.nnodes) {
        const int64_t o = 3 * (int64_t)node0 + t;
        cp_async<8>(&s.u[t], a.u[parity] + o);
        cp_async<8>(&s.bcv[t], a.bc_values + o);
        cp_async<8>(&s.fcv[t], a.fc_values + o);
        cp_async<4>(&s.bct[t], a.bc_types + o);
        cp_async<4>(&s.fct[t], a.fc_types + o);
        if (a.integrator != PP_EULER) {
            cp_async<8>(&s.ud[t], a.ud + o);
            cp_async<8>(&s.udd[t], a.udd + o);
            cp_async<8>(&s.rho[t], a.densities + o);
        }
    }
    if (t < nodes && node0 + t < a.nnodes) cp_async<4>(&s.family[t], a.family + node0 + t);
}

// Node updates of a block's `nodes` nodes from their bond forces and intact
// counts: one thread per DOF, then one per node for the damage (a warp-wide
// update of one node's three DOFs would hold the binary64 pipe as long).
// Called by every thread of the block.
__device__ __forceinline__ void f64_node_phase(const pp_fused_args& a, int parity,
                                               const StepMags& m, int node0, int nodes,
                                               NodeStage& s) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int t = threadIdx.x;
    if (t < 3 * nodes) {
        const int64_t o = 3 * (int64_t)node0 + t;
        if (node0 + t / 3 < a.nnodes) {
            const double body = s.sum[t];
            a.body_force[o] = body;
            const double frc = force_with_bc(body, s.fct[t], s.fcv[t], m.force);
            a.force[o] = frc;
            const int bct = s.bct[t];
            const double bcv = s.bcv[t];
            const double u = s.u[t];
            double unew;
            if (a.integrator == PP_EULER) {
                unew = euler_u(u, frc, bct, bcv, m.disp, a.dt);
            } else {
                double v = s.ud[t];
                double acc = s.udd[t];
                if (a.integrator == PP_EULER_CROMER)
                    unew = euler_cromer_u(u, v, acc, frc, bct, bcv, s.rho[t], m.disp, a.damping,
                                          a.dt);
                else
                    unew = velocity_verlet_u(u, v, acc, frc, bct, bcv, s.rho[t], m.disp,
                                             a.damping, a.dt);
                a.ud[o] = v;
                a.udd[o] = acc;
            }
            a.u[parity ^ 1][o] = unew;
        }
    } else if (t < 4 * nodes) {
        const int li = t - 3 * nodes;
        if (node0 + li < a.nnodes) {
            a.n_neigh[node0 + li] = s.count[li];
            a.damage[node0 + li] = damage_of(s.count[li], s.family[li]);
        }
    }
}

}  // namespace pp
