// pp_adjoint.cu -- reverse (adjoint) step of the Euler time step with
// per-bond stiffness and a frozen bond set, for gradients of a
// displacement loss.
//
// Forward step (run with pp_fused_step, PP_FLOAT64, stiffness corrections =
// per-bond stiffness k_b, bond_stiffness = 1, critical_stretch = +inf so
// the bond set stays frozen):
//   u'_m = u_m + dt f_m(u)   on free DOFs,   u'_m = c * bc_values on BC DOFs
//   f_m  = sum_{b=(m,j)} k_b vol_j s_b p_b/|p_b|,  p_b = xi_b + u_j - u_m,
//   s_b  = (|p_b| - |xi_b|)/|xi_b|            (peridynamics.cl:65-87, :214)
// Reverse of one step, with mu = lambda' masked to the free DOFs:
//   lambda_m = mu_m + dt sum_{b=(m,j)} G_b (k_(j,m) vol_m mu_j - k_b vol_j mu_m)
//   G(p)     = p^ p^T / |xi| + (s/|p|)(I - p^ p^T)      (symmetric, even in p)
//   dL/dk_b += dt vol_j s_b (mu_m . p^_b)
// The first sum gathers the contribution of the reverse bond (j, m) from
// row m itself: G is the same for both directions of a bond, and the
// reverse bond's stiffness is found through the partner slot.  One warp per
// node, no atomics: the gradient is deterministic.
//
// On a pair list (pp_pairs.cu) whose pairs all have two slots the reverse
// step computes each bond once: the contribution G v to node m is the negative
// of the one to node j.  k_adjoint_pairs writes it as a record and adds to
// both slots' gradients (kept per pair, so that the additions are coalesced;
// pp_pair_gradient spreads them at the end); k_adjoint_nodes sums the records.
// A rollout's steps are queued from here (pp_rollout_forward / _backward).
#include "pp_pairs.cuh"

namespace pp {
namespace {

constexpr int kWarps = 8;

__global__ void __launch_bounds__(kWarps * 32)
    k_partner_slots(const int32_t* __restrict__ nlist, int nnodes, int L,
                    int32_t* __restrict__ partner) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (i >= nnodes) return;
    for (int s = lane; s < L; s += 32) {
        const int j = nlist[(int64_t)i * L + s];
        int found = -1;
        if (j >= 0 && j < nnodes) {
            const int32_t* row = nlist + (int64_t)j * L;
            for (int q = 0; q < L; ++q)
                if (row[q] == i) {
                    found = q;
                    break;
                }
        }
        partner[(int64_t)i * L + s] = found;
    }
}

__global__ void __launch_bounds__(kWarps * 32)
    k_adjoint_backward(pp_adjoint_args a, const double* __restrict__ u,
                       const double* __restrict__ lam_next, double* __restrict__ lam,
                       double* __restrict__ grad_k) {
    const int lane = threadIdx.x & 31;
    const int m = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (m >= a.nnodes) return;  // warp-uniform
    const int L = a.max_neigh;
    const int64_t o3 = 3 * (int64_t)m;
    const double rmx = a.r0[o3], rmy = a.r0[o3 + 1], rmz = a.r0[o3 + 2];
    const double umx = u[o3], umy = u[o3 + 1], umz = u[o3 + 2];
    // mu = lambda_next on the free DOFs of node m
    const double mmx = a.bc_types[o3] ? 0.0 : lam_next[o3];
    const double mmy = a.bc_types[o3 + 1] ? 0.0 : lam_next[o3 + 1];
    const double mmz = a.bc_types[o3 + 2] ? 0.0 : lam_next[o3 + 2];
    const double vol_m = a.vols[m];
    double ax = 0.0, ay = 0.0, az = 0.0;
    for (int s = lane; s < L; s += 32) {
        const int64_t gid = (int64_t)m * L + s;
        const int j = a.nlist[gid];
        if (j == -1) continue;
        const int64_t j3 = 3 * (int64_t)j;
        const double xx = a.r0[j3] - rmx, xy = a.r0[j3 + 1] - rmy, xz = a.r0[j3 + 2] - rmz;
        const double px = u[j3] - umx + xx, py = u[j3 + 1] - umy + xy, pz = u[j3 + 2] - umz + xz;
        const double xi = sqrt(xx * xx + xy * xy + xz * xz);
        const double y = sqrt(px * px + py * py + pz * pz);
        const double st = (y - xi) / xi;
        const double hx = px / y, hy = py / y, hz = pz / y;
        const double mjx = a.bc_types[j3] ? 0.0 : lam_next[j3];
        const double mjy = a.bc_types[j3 + 1] ? 0.0 : lam_next[j3 + 1];
        const double mjz = a.bc_types[j3 + 2] ? 0.0 : lam_next[j3 + 2];
        const double kb = a.stiffness[gid];
        const int q = a.partner[gid];
        const double krev =
            (q >= 0 && a.nlist[(int64_t)j * L + q] == m) ? a.stiffness[(int64_t)j * L + q] : 0.0;
        // v = k_(j,m) vol_m mu_j - k_b vol_j mu_m
        const double vol_j = a.vols[j];
        const double vx = krev * vol_m * mjx - kb * vol_j * mmx;
        const double vy = krev * vol_m * mjy - kb * vol_j * mmy;
        const double vz = krev * vol_m * mjz - kb * vol_j * mmz;
        // G v = (h.v)/|xi| h + (s/|p|)(v - (h.v) h)
        const double hv = hx * vx + hy * vy + hz * vz;
        const double c1 = hv / xi, c2 = st / y;
        ax += c1 * hx + c2 * (vx - hv * hx);
        ay += c1 * hy + c2 * (vy - hv * hy);
        az += c1 * hz + c2 * (vz - hv * hz);
        // dL/dk_b += dt vol_j s_b (mu_m . h)
        grad_k[gid] += a.dt * vol_j * st * (mmx * hx + mmy * hy + mmz * hz);
    }
    for (int off = 16; off >= 1; off >>= 1) {
        ax += __shfl_xor_sync(kFull, ax, off);
        ay += __shfl_xor_sync(kFull, ay, off);
        az += __shfl_xor_sync(kFull, az, off);
    }
    if (lane == 0) {
        lam[o3] = mmx + a.dt * ax;
        lam[o3 + 1] = mmy + a.dt * ay;
        lam[o3 + 2] = mmz + a.dt * az;
    }
}

constexpr int kPairThreads = 128;

// What a bond's reverse step needs of its geometry: s and 1/|p|.
struct AdjointBond {
    uint64_t s, inv_y;
};

static __device__ __noinline__ AdjointBond adjoint_bond_any(double sq, double xi) {
    using exact64::double_bits;
    const double y = sqrt(sq);
    return {double_bits((y - xi) / xi), double_bits(1.0 / y)};
}

// On the integer pipe (pp_exact64.cuh) within the limits of f64_stretch.
__device__ __forceinline__ AdjointBond adjoint_bond(double sq, double xi) {
    using namespace exact64;
    const uint64_t sb = double_bits(sq), lb = double_bits(xi);
    constexpr uint64_t kOne = 0x3FF0000000000000ull;
    AdjointBond r{0, 0};
    bool ok = positive_in(sb, 1023 - 400, 1023 + 400) && positive_in(lb, 1023 - 200, 1023 + 200);
    if (ok) {
        const Divisor y = sqrt_rn(sb);
        ok = relative_difference(y, divisor(lb), r.s);
        r.inv_y = div_bits(kOne, y);
    }
    if (!ok) r = adjoint_bond_any(sq, xi);
    return r;
}

// x, or zero where `off`: selected as integers (a selected double takes a
// slot of the binary64 pipe).
__device__ __forceinline__ double zero_if(bool off, const double* x) {
    const long long bits = *reinterpret_cast<const long long*>(x);
    return __longlong_as_double(off ? 0ll : bits);
}

// What the reverse step reads of a node, 32 bytes: lambda on the free DOFs
// (zero on the others) and the volume.
struct NodeMu {
    d3 mu;
    double vol;
};

__device__ __forceinline__ NodeMu load_mu(const double* __restrict__ mu, int64_t i) {
    NodeMu r;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(r.mu.x), "=d"(r.mu.y), "=d"(r.mu.z), "=d"(r.vol)
        : "l"(mu + 4 * i));
    return r;
}

__global__ void k_adjoint_pack(const double* __restrict__ grad_u, const int32_t* __restrict__ bc,
                               const double* __restrict__ vols, int nnodes,
                               double* __restrict__ mu) {
    const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (g >= 4 * (int64_t)nnodes) return;
    const int64_t i = g >> 2, o = 3 * i + (g & 3);
    mu[g] = (g & 3) == 3 ? vols[i] : zero_if(bc[o] != 0, grad_u + o);
}

__device__ __forceinline__ double dot(const d3& a, const d3& b) {
    return __fma_rn(a.x, b.x, __fma_rn(a.y, b.y, a.z * b.z));
}

// One thread per pair.  s/|p| = 1/|xi| - 1/|p|, so with c = s/|p|
//   G v = c v + (p.v) p / |p|^3,   v = k_(j,m) vol_m mu_j - k_(m,j) vol_j mu_m
// and both p.v and the gradients follow from p.mu_m and p.mu_j.  Bound by the
// binary64 pipe: 39 operations a bond (fused multiply-adds; root and
// quotients on the integer pipe) instead of some 130 from each end, six of
// them divisions and two square roots.  What it gathers of a node is one load
// (NodeMu) besides u.  A pass of the 12,500-node rollout (500 steps forward,
// recomputed and reversed): 353 ms with k_fused_f64 of the time and
// k_adjoint_backward, 228 ms after the forward steps' arithmetic moved, 79 ms
// with both on pairs, 73 ms with this algebra, the nodes' records and
// tree_block_f64 (this kernel 46 -> 43 us, k_adjoint_nodes 19 -> 17), 68 ms
// with the forward kernels launched ahead (pp_pairs.cu).
__global__ void __launch_bounds__(kPairThreads)
    k_adjoint_pairs(pp_adjoint_args a, pp_pairs pr, int shift, const double* __restrict__ u,
                    const double* __restrict__ mu, double* __restrict__ grad_pair) {
    __shared__ double s_one;
    if (threadIdx.x == 0) s_one = 1.0;
    __syncthreads();
    const F64Ops op(&s_one);
    const int64_t q = blockIdx.x * (int64_t)kPairThreads + threadIdx.x;
    if (q >= pr.npairs) return;
    const int2 gh = reinterpret_cast<const int2*>(pr.slots)[q];
    const bool live_g = a.nlist[gh.x] != -1, live_h = a.nlist[gh.y] != -1;
    if (!live_g && !live_h) return;
    const int m = gh.x >> shift, j = gh.y >> shift;
    const int64_t om = 3 * (int64_t)m;
    const NodeMu nm = load_mu(mu, m), nj = load_mu(mu, j);
    const d3 mu_m = nm.mu, mu_j = nj.mu;
    const double vol_m = nm.vol, vol_j = nj.vol;
    const double kj = zero_if(!live_h, a.stiffness + gh.y);
    const double km = zero_if(!live_g, a.stiffness + gh.x);
    double2* const g = reinterpret_cast<double2*>(grad_pair) + q;
    const double2 old = *g;
    const d3 p = f64_deformed(op, u, j, d3{u[om], u[om + 1], u[om + 2]},
                              pair_reference(pr, q));
    const AdjointBond bond = adjoint_bond(dot(p, p), pr.length[q]);
    const double inv_y = __longlong_as_double(bond.inv_y);
    const double c = __longlong_as_double(bond.s) * inv_y;
    const double pm = dot(p, mu_m), pj = dot(p, mu_j);
    const double cj = kj * vol_m, cm = -(km * vol_j);
    const double e = __fma_rn(cj, pj, cm * pm) * inv_y * inv_y * inv_y;
    const double wj = c * cj, wm = c * cm;
    store_record(pr.force + 4 * q, d3{__fma_rn(wj, mu_j.x, __fma_rn(wm, mu_m.x, e * p.x)),
                                      __fma_rn(wj, mu_j.y, __fma_rn(wm, mu_m.y, e * p.y)),
                                      __fma_rn(wj, mu_j.z, __fma_rn(wm, mu_m.z, e * p.z))});
    // dL/dk += dt vol s (mu . p)/|p|, p reversed for the second slot; a
    // broken direction's stays as it is
    const double t = a.dt * c;
    const double gx = __fma_rn(t * vol_j, pm, old.x);
    const double gy = __fma_rn(-(t * vol_m), pj, old.y);
    longlong2 sum;
    sum.x = live_g ? __double_as_longlong(gx) : __double_as_longlong(old.x);
    sum.y = live_h ? __double_as_longlong(gy) : __double_as_longlong(old.y);
    *reinterpret_cast<longlong2*>(g) = sum;
}

// lam = mu + dt (sum of the node's records), one warp per node; kept on the
// free DOFs, with the volume.  A lane's slots go in batches of B, the loads of
// a batch in flight together.
template <int B>
__global__ void __launch_bounds__(kWarps * 32)
    k_adjoint_nodes(pp_adjoint_args a, pp_pairs pr, const double* __restrict__ mu_next,
                    double* __restrict__ mu) {
    __shared__ double s_one, s_sum[3 * kWarps], s_part[3 * 32 * kWarps];
    if (threadIdx.x == 0) s_one = 1.0;
    __syncthreads();
    const F64Ops op(&s_one);
    const int m = blockIdx.x * kWarps + (threadIdx.x >> 5);
    const int64_t row = (int64_t)m * a.max_neigh;
    d3 v = d3_zero();
    for (int s0 = m < a.nnodes ? threadIdx.x & 31 : a.max_neigh; s0 < a.max_neigh;
         s0 += 32 * B) {
        int sp[B], j[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            sp[b] = pr.slot_pair[row + s0 + 32 * b];
            j[b] = a.nlist[row + s0 + 32 * b];
        }
        d3 w[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            if (j[b] == -1) sp[b] = -1;
            w[b] = signed_record(pr.force + 4 * (int64_t)(sp[b] & 0x7FFFFFFF), sp[b]);
        }
#pragma unroll
        for (int b = 0; b < B; ++b)
            v = d3{op.add(v.x, w[b].x), op.add(v.y, w[b].y), op.add(v.z, w[b].z)};
    }
    tree_block_put(s_part, v);
    __syncthreads();
    const int t = (threadIdx.x - 96 * blockIdx.x) & (kWarps * 32 - 1);
    if (t < 96) tree_block_f64(op, t, s_part, s_sum);
    __syncthreads();
    const int64_t g = 4 * (int64_t)blockIdx.x * kWarps + threadIdx.x;
    if (threadIdx.x >= 4 * kWarps || g >= 4 * (int64_t)a.nnodes) return;
    const int node = threadIdx.x >> 2, comp = threadIdx.x & 3;
    const double lam = __fma_rn(a.dt, s_sum[comp < 3 ? 3 * node + comp : 0], mu_next[g]);
    const bool off = comp == 3 || a.bc_types[3 * (g >> 2) + comp] != 0;
    mu[g] = off ? mu_next[g] : lam;  // (zero and the volume stay)
}

// The gradient of every slot from those kept per pair (zero elsewhere).
__global__ void k_pair_gradient(const int32_t* __restrict__ slot_pair, int64_t nslots,
                                const double* __restrict__ grad_pair, double* __restrict__ grad) {
    const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (g >= nslots) return;
    const int sp = slot_pair[g];
    grad[g] = sp == -1 ? 0.0 : grad_pair[2 * (int64_t)(sp & 0x7FFFFFFF) + (sp < 0 ? 1 : 0)];
}

// First step at which each slot is seen broken.
__global__ void k_mark_breaks(const int32_t* __restrict__ nlist, int32_t* __restrict__ break_step,
                              int64_t nslots, int32_t t) {
    const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (g < nslots && nlist[g] == -1 && break_step[g] > t) break_step[g] = t;
}

// The bond set in force during step t.
__global__ void k_bonds_at_step(const int32_t* __restrict__ nlist0,
                                const int32_t* __restrict__ break_step, int64_t nslots,
                                int32_t t, int32_t* __restrict__ nlist_t) {
    const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (g < nslots) nlist_t[g] = break_step[g] > t ? nlist0[g] : -1;
}

}  // namespace
}  // namespace pp

using namespace pp;

extern "C" int pp_mark_breaks(const int32_t* nlist, int32_t* break_step, int64_t nslots,
                              int32_t t, void* stream) {
    if (nslots < 0) return PP_ERROR_INVALID_VALUE;
    if (nslots == 0) return PP_SUCCESS;
    if (!nlist || !break_step) return PP_ERROR_INVALID_VALUE;
    k_mark_breaks<<<(unsigned)((nslots + 255) / 256), 256, 0,
                    static_cast<cudaStream_t>(stream)>>>(nlist, break_step, nslots, t);
    return launch_status();
}

extern "C" int pp_bonds_at_step(const int32_t* nlist0, const int32_t* break_step, int64_t nslots,
                                int32_t t, int32_t* nlist_t, void* stream) {
    if (nslots < 0) return PP_ERROR_INVALID_VALUE;
    if (nslots == 0) return PP_SUCCESS;
    if (!nlist0 || !break_step || !nlist_t) return PP_ERROR_INVALID_VALUE;
    k_bonds_at_step<<<(unsigned)((nslots + 255) / 256), 256, 0,
                      static_cast<cudaStream_t>(stream)>>>(nlist0, break_step, nslots, t,
                                                           nlist_t);
    return launch_status();
}

extern "C" int pp_partner_slots(const int32_t* nlist, int32_t nnodes, int32_t max_neigh,
                                int32_t* partner, void* stream) {
    if (nnodes < 0) return PP_ERROR_INVALID_VALUE;
    if (!is_pow2_le_1024(max_neigh)) return PP_ERROR_MAX_NEIGH;
    if (nnodes == 0) return PP_SUCCESS;
    if (!nlist || !partner) return PP_ERROR_INVALID_VALUE;
    k_partner_slots<<<(nnodes + kWarps - 1) / kWarps, kWarps * 32, 0,
                      static_cast<cudaStream_t>(stream)>>>(nlist, nnodes, max_neigh, partner);
    return launch_status();
}

extern "C" int pp_adjoint_backward(const pp_adjoint_args* args, const double* u,
                                   const double* lam_next, double* lam, double* grad_k,
                                   void* stream) {
    if (!args) return PP_ERROR_INVALID_VALUE;
    const pp_adjoint_args& a = *args;
    if (a.nnodes < 0) return PP_ERROR_INVALID_VALUE;
    if (!is_pow2_le_1024(a.max_neigh)) return PP_ERROR_MAX_NEIGH;
    if (a.nnodes == 0) return PP_SUCCESS;
    if (!a.r0 || !a.vols || !a.nlist || !a.partner || !a.bc_types || !a.stiffness || !u ||
        !lam_next || !lam || !grad_k || lam == lam_next)
        return PP_ERROR_INVALID_VALUE;
    k_adjoint_backward<<<(a.nnodes + kWarps - 1) / kWarps, kWarps * 32, 0,
                         static_cast<cudaStream_t>(stream)>>>(a, u, lam_next, lam, grad_k);
    return launch_status();
}

namespace pp {
namespace {

int adjoint_pair_step(const pp_adjoint_args& a, const pp_pairs& pr, const double* u,
                      const double* mu_next, double* mu, double* grad_pair, cudaStream_t st) {
    const int shift = 31 - __builtin_clz((unsigned)a.max_neigh);
    if (pr.npairs > 0)
        k_adjoint_pairs<<<(unsigned)((pr.npairs + kPairThreads - 1) / kPairThreads), kPairThreads,
                          0, st>>>(a, pr, shift, u, mu_next, grad_pair);
    const auto nodes = a.max_neigh >= 128  ? k_adjoint_nodes<4>
                       : a.max_neigh >= 64 ? k_adjoint_nodes<2>
                                           : k_adjoint_nodes<1>;
    nodes<<<(a.nnodes + kWarps - 1) / kWarps, kWarps * 32, 0, st>>>(a, pr, mu_next, mu);
    return launch_status();
}

int check_rollout(const pp_fused_args* args, const pp_pairs* pairs, const pp_rollout* r) {
    if (!args || !pairs || !r || r->steps < 0 || r->every < 1) return PP_ERROR_INVALID_VALUE;
    const int v = validate_pairs(*args, *pairs);
    if (v != PP_SUCCESS) return v;
    // each pair's two directions have their own stiffness
    if (args->integrator != PP_EULER || args->bond_types || pairs->symmetric)
        return PP_ERROR_INVALID_VALUE;
    if (r->steps > 0 && (!r->mags || !r->checkpoints)) return PP_ERROR_INVALID_VALUE;
    return PP_SUCCESS;
}

Launch at_magnitude(double mag) { return Launch{mag, 0.0, nullptr, nullptr, nullptr, 0}; }

}  // namespace
}  // namespace pp

extern "C" int pp_rollout_forward(const pp_fused_args* args, const pp_pairs* pairs,
                                  const pp_rollout* r, void* stream) {
    const int v = check_rollout(args, pairs, r);
    if (v != PP_SUCCESS || args->nnodes == 0) return v;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t size = 3 * (size_t)args->nnodes;
    pp_pairs pr = *pairs;
    pr.break_step = r->break_step;
    for (int t = 0; t < r->steps; ++t) {
        const int p = t & 1;
        if (t % r->every == 0 &&
            cudaMemcpyAsync(r->checkpoints + (t / r->every) * size, args->u[p],
                            size * sizeof(double), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            return PP_ERROR_CUDA;
        pr.step = t;
        const int rc = launch_pair_step(*args, pr, p, at_magnitude(r->mags[t]), st);
        if (rc != PP_SUCCESS) return rc;
    }
    return PP_SUCCESS;
}

extern "C" int pp_rollout_backward(const pp_fused_args* args, const pp_pairs* pairs,
                                   const pp_rollout* r, const pp_adjoint_args* adjoint,
                                   const int32_t* nlist0, const double* grad_u, double* mu0,
                                   double* mu1, double* grad_pair, void* stream) {
    int v = check_rollout(args, pairs, r);
    if (v != PP_SUCCESS || args->nnodes == 0) return v;
    if (!adjoint || adjoint->nnodes != args->nnodes || adjoint->max_neigh != args->max_neigh ||
        adjoint->nlist != args->nlist || !adjoint->r0 || !adjoint->vols || !adjoint->bc_types ||
        !adjoint->stiffness || !grad_u || !mu0 || !mu1 || mu0 == mu1 || !grad_pair ||
        (r->every > 1 && !r->states) || (r->break_step && !nlist0) ||
        ((reinterpret_cast<uintptr_t>(mu0) | reinterpret_cast<uintptr_t>(mu1)) & 31u) ||
        (reinterpret_cast<uintptr_t>(grad_pair) & 15u))
        return PP_ERROR_INVALID_VALUE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t size = 3 * (size_t)args->nnodes;
    const int64_t nslots = (int64_t)args->nnodes * args->max_neigh;
    pp_fused_args a = *args;
    pp_pairs pr = *pairs;
    pr.break_step = nullptr;
    double* mu[2] = {mu0, mu1};
    k_adjoint_pack<<<(unsigned)((4 * (int64_t)a.nnodes + 255) / 256), 256, 0, st>>>(
        grad_u, adjoint->bc_types, adjoint->vols, a.nnodes, mu0);
    if ((v = launch_status()) != PP_SUCCESS) return v;
    int p = 0;
    // the bond set in force during step t
    auto bonds = [&](int t) {
        return r->break_step ? pp_bonds_at_step(nlist0, r->break_step, nslots, t, a.nlist, stream)
                             : PP_SUCCESS;
    };
    for (int t0 = r->steps > 0 ? (r->steps - 1) / r->every * r->every : -1; t0 >= 0;
         t0 -= r->every) {
        const int t1 = r->steps - t0 < r->every ? r->steps : t0 + r->every;
        double* first = r->checkpoints + (t0 / r->every) * size;
        auto state = [&](int t) { return t == t0 ? first : r->states + (t - t0 - 1) * size; };
        for (int t = t0; t < t1 - 1; ++t) {
            if ((v = bonds(t)) != PP_SUCCESS) return v;
            a.u[0] = state(t);
            a.u[1] = state(t + 1);
            if ((v = launch_pair_step(a, pr, 0, at_magnitude(r->mags[t]), st)) != PP_SUCCESS)
                return v;
        }
        for (int t = t1 - 1; t >= t0; --t) {
            if ((v = bonds(t)) != PP_SUCCESS) return v;
            if ((v = adjoint_pair_step(*adjoint, pr, state(t), mu[p], mu[p ^ 1], grad_pair, st)) != PP_SUCCESS)
                return v;
            p ^= 1;
        }
    }
    return PP_SUCCESS;
}

extern "C" int pp_pair_gradient(const pp_pairs* pairs, int64_t nslots, const double* grad_pair,
                                double* grad, void* stream) {
    if (!pairs || nslots < 0) return PP_ERROR_INVALID_VALUE;
    if (nslots == 0) return PP_SUCCESS;
    if (!pairs->slot_pair || !grad_pair || !grad) return PP_ERROR_INVALID_VALUE;
    k_pair_gradient<<<(unsigned)((nslots + 255) / 256), 256, 0,
                      static_cast<cudaStream_t>(stream)>>>(pairs->slot_pair, nslots, grad_pair,
                                                           grad);
    return launch_status();
}
