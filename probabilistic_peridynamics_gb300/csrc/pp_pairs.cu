// pp_pairs.cu -- the PP_FLOAT64 step with each bond computed once.
//
// Both directions of a bond (i, j) have the same length, stretch and, up to
// the sign, direction cosines, bit for bit: r0[j] - r0[i] and u[j] - u[i]
// change sign exactly.  A pair list names the two slots of every bond:
//
//  k_pair_bonds  one thread per pair: the binary64 bond arithmetic of
//                pp_bond_f64.cuh once, the damage law of each live side, and
//                the force vectors of both directions into a 32-byte record
//                (one record when they are exact negatives of each other:
//                PMB bonds between nodes of equal volume and correction);
//  k_pair_nodes  one warp per node: the records of its slots summed in the
//                work-group tree order (pp_common.cuh), then the node update.
//
// Both kernels are bound by the binary64 pipe (88 and 92 % busy on the plate of
// 400,000 nodes in rows of 128 slots: 0.62 + 0.32 ms), so halving the bond
// work (1.95 ms in one kernel) outweighs writing and gathering the records (32 bytes
// a pair written, 32 gathered per slot).  What that pipe does not have to do is
// kept off it: roots and quotients (pp_exact64.cuh), the reference vectors
// (24 bytes a pair read instead of three subtractions, 0.66 -> 0.63 ms), signs
// and selects.
//
// The pair list depends only on the bonds that exist when it is built; a
// slot that is -1 at a step is dead whoever broke it.  A slot without a
// counterpart (a one-sided list), the later copies of a neighbour listed
// twice and a node listed as its own neighbour form pairs of one side.
#include "pp_pairs.cuh"

namespace pp {
namespace {

constexpr int kRowWarps = 8;
constexpr int kPairThreads = 128;
// The step's kernels are launched ahead of their predecessor's end
// (pp_common.cuh: 2,000 nodes 9.2 us a step against 9.7, 800 nodes in rows of 256
// slots 9.7 against 10.1).  From so many pairs on they also let the next one in
// before their last stores (42.7M bonds 0.944 against 0.968 ms, 6.1M bonds in rows
// of 32 slots 0.179 against 0.194, 1.0M bonds 30.1 against 30.4 us); with fewer its
// waiting blocks crowd the SMs (470,000 bonds 16.3 against 15.1 us, 36,500 bonds
// 10.6 against 6.9).
constexpr int kReleasePairs = 400'000;
constexpr int kSingle = -2;    // build: owner of a pair of one side
constexpr int kPartner = -3;   // build: the pair's other slot owns it

// Valid entries of a row that is strictly ascending with its -1 entries at
// the end; -1 for any other row.  One warp per row.
__global__ void __launch_bounds__(kRowWarps * 32)
    k_row_order(const int32_t* __restrict__ nlist, int nnodes, int L, int32_t* __restrict__ len) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
    if (i >= nnodes) return;
    const int32_t* row = nlist + (int64_t)i * L;
    bool ok = true;
    int count = 0;
    for (int s = lane; s < L; s += 32) {
        const int j = row[s];
        const int before = s > 0 ? row[s - 1] : -1;
        if (j >= 0 && j < nnodes) {
            ++count;
            ok = ok && (s == 0 || (before >= 0 && before < j));
        } else {
            ok = ok && j == -1;
        }
    }
    count = __reduce_add_sync(kFull, count);
    ok = __all_sync(kFull, ok);
    if (lane == 0) len[i] = ok ? count : -1;
}

// The first slot of row r that holds key, or -1.
__device__ __forceinline__ int find_first(const int32_t* __restrict__ row, int L, int len,
                                          int key) {
    if (len >= 0) {
        int lo = 0, hi = len;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (row[mid] < key)
                lo = mid + 1;
            else
                hi = mid;
        }
        return lo < len && row[lo] == key ? lo : -1;
    }
    for (int s = 0; s < L; ++s)
        if (row[s] == key) return s;
    return -1;
}

// Every slot's counterpart: slot_pair = the counterpart's slot, or kSingle,
// where the slot owns its pair; kPartner where the counterpart does; -1
// where there is no bond.  Owners per row go to row_start[i + 1].
__global__ void __launch_bounds__(kRowWarps * 32)
    k_pair_partners(const int32_t* __restrict__ nlist, const int32_t* __restrict__ len, int nnodes,
                    int L, int32_t* __restrict__ slot_pair, int32_t* __restrict__ row_start) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
    if (i >= nnodes) return;
    const int64_t base = (int64_t)i * L;
    const int32_t* row = nlist + base;
    const int own = len[i];
    int owners = 0;
    for (int s = lane; s < L; s += 32) {
        const int j = row[s];
        int v = -1;
        if (j >= 0 && j < nnodes) {
            v = kSingle;
            if (j != i && (own >= 0 || find_first(row, L, -1, j) == s)) {
                const int q = find_first(nlist + (int64_t)j * L, L, len[j], i);
                if (q >= 0) v = i < j ? j * L + q : kPartner;
            }
            owners += v != kPartner;
        }
        slot_pair[base + s] = v;
    }
    owners = __reduce_add_sync(kFull, owners);
    if (lane == 0) row_start[i + 1] = owners;
}

// In-place inclusive scan of start[1..n], start[0] = 0; one CTA of 1024
// threads.  Set-up only.
__global__ void k_pair_scan(int32_t* __restrict__ start, int n) {
    __shared__ int warp_tot[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ int carry;
    if (tid == 0) {
        carry = 0;
        start[0] = 0;
    }
    __syncthreads();
    for (int k0 = 0; k0 < n; k0 += 1024) {
        const int k = k0 + tid;
        int v = k < n ? start[k + 1] : 0;
        for (int off = 1; off < 32; off <<= 1) {
            const int w = __shfl_up_sync(kFull, v, off);
            if (lane >= off) v += w;
        }
        if (lane == 31) warp_tot[warp] = v;
        __syncthreads();
        if (warp == 0) {
            int w = warp_tot[lane];
            for (int off = 1; off < 32; off <<= 1) {
                const int x = __shfl_up_sync(kFull, w, off);
                if (lane >= off) w += x;
            }
            warp_tot[lane] = w;
        }
        __syncthreads();
        v += carry + (warp > 0 ? warp_tot[warp - 1] : 0);
        if (k < n) start[k + 1] = v;
        __syncthreads();
        if (tid == 1023) carry = v;
        __syncthreads();
    }
}

// The pairs of a row's owner slots, in slot order from row_start[i].  Sets
// *differ where the two directions of a bond do not have equal volumes and
// corrections.
__global__ void __launch_bounds__(kRowWarps * 32)
    k_pair_fill(const int32_t* __restrict__ nlist, const double* __restrict__ r0,
                const double* __restrict__ vols, const double* __restrict__ sc, int nnodes, int L,
                const int32_t* __restrict__ row_start, pp_pairs pr, int32_t* __restrict__ differ) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
    if (i >= nnodes) return;
    const int64_t base = (int64_t)i * L;
    const int64_t o = 3 * (int64_t)i;
    int next = row_start[i];
    bool diff = false;
    for (int s0 = 0; s0 < L; s0 += 32) {
        const int s = s0 + lane;
        const int v = s < L ? pr.slot_pair[base + s] : -1;
        const bool owner = v >= 0 || v == kSingle;
        const unsigned m = __ballot_sync(kFull, owner);
        if (owner) {
            const int p = next + __popc(m & ((1u << lane) - 1u));
            const int g = (int)(base + s);
            const int j = nlist[g];
            reinterpret_cast<int2*>(pr.slots)[p] = make_int2(g, v >= 0 ? v : -1);
            pr.slot_pair[g] = p;
            const double x = dsub(r0[3 * (int64_t)j], r0[o]);
            const double y = dsub(r0[3 * (int64_t)j + 1], r0[o + 1]);
            const double z = dsub(r0[3 * (int64_t)j + 2], r0[o + 2]);
            pr.length[p] = f64_length(dadd(dadd(dmul(x, x), dmul(y, y)), dmul(z, z)));
            pr.vector[p] = x;
            pr.vector[pr.npairs + p] = y;
            pr.vector[2 * pr.npairs + p] = z;
            if (v >= 0) {
                pr.slot_pair[v] = p | kReversed;
                diff |= __double_as_longlong(vols[i]) != __double_as_longlong(vols[j]);
                if (sc) diff |= __double_as_longlong(sc[g]) != __double_as_longlong(sc[v]);
            }
        }
        next += __popc(m);
    }
    if (__any_sync(kFull, diff) && lane == 0) atomicOr(differ, 1);
}

template <bool CORR, bool TYPES, bool SYM>
__global__ void __launch_bounds__(kPairThreads, 8)
    k_pair_bonds(pp_fused_args a, pp_pairs pr, int parity, int shift) {
    __shared__ double s_one;
    if (threadIdx.x == 0) s_one = 1.0;
    __syncthreads();
    const F64Ops op(&s_one);
    const int64_t p = blockIdx.x * (int64_t)kPairThreads + threadIdx.x;
    grid_wait();
    if (p >= pr.npairs) return;
    const int2 gh = reinterpret_cast<const int2*>(pr.slots)[p];
    const int jg = a.nlist[gh.x];
    const int jh = gh.y >= 0 ? a.nlist[gh.y] : -1;
    if (jg == -1 && jh == -1) return;
    const int i = gh.x >> shift;
    const int j = jg != -1 ? jg : gh.y >> shift;
    F64Bond b{a.r0,
              a.u[parity],
              a.vols,
              a.nlist,
              a.stiffness_corrections,
              a.bond_types,
              a.regimes,
              a.bond_stiffness_table,
              a.critical_stretch_table,
              a.plus_cs,
              nullptr,
              a.bond_stiffness,
              a.critical_stretch,
              a.nregimes};
    const int64_t oi = 3 * (int64_t)i;
    const d3 ui{b.u[oi], b.u[oi + 1], b.u[oi + 2]};
    const d3 xe = f64_deformed(op, b.u, j, ui, pair_reference(pr, p));
    const F64Stretch st = f64_stretch<false>(op, xe, pr.length[p]);
    if (pr.npairs >= kReleasePairs) grid_release();
    bool live_g = jg != -1, live_h = jh != -1;
    const double s = __longlong_as_double(st.s);
    if constexpr (SYM) {
        // the same force either way; each side breaks by itself
        if (live_g && !f64_less(s, a.node_instance ? a.instance_s0[a.node_instance[i]] : b.s0)) {
            live_g = false;
            a.nlist[gh.x] = -1;
            if (pr.break_step) pr.break_step[gh.x] = pr.step;
        }
        if (live_h && !f64_less(s, a.node_instance ? a.instance_s0[a.node_instance[j]] : b.s0)) {
            live_h = false;
            a.nlist[gh.y] = -1;
            if (pr.break_step) pr.break_step[gh.y] = pr.step;
        }
        if (!live_g && !live_h) return;
        double f = op.mul(s, b.k);
        if constexpr (CORR) f = op.mul(f, b.sc[gh.x]);
        store_record(pr.force + 4 * p, f64_force(op, op.mul(f, b.vols[j]), st));
    } else {
        double f;
        if (live_g) {
            if (!TYPES && a.node_instance) b.s0 = a.instance_s0[a.node_instance[i]];
            if (f64_bond_law<CORR, TYPES>(op, b, gh.x, s, b.vols[j], f))
                store_record(pr.force + 8 * p, f64_force(op, f, st));
            else if (pr.break_step)
                pr.break_step[gh.x] = pr.step;
        }
        if (live_h) {
            if (!TYPES && a.node_instance) b.s0 = a.instance_s0[a.node_instance[j]];
            if (f64_bond_law<CORR, TYPES>(op, b, gh.y, s, b.vols[i], f))
                store_record(pr.force + 8 * p + 4, f64_force(op, f, st));
            else if (pr.break_step)
                pr.break_step[gh.y] = pr.step;
        }
    }
}

// Latency-bound until four slots' loads are in flight and the node updates'
// inputs are staged (0.56 -> 0.43 ms); then 32 registers, so that 64 warps
// are resident (0.39 ms; rows of 256 slots hold more and do better with 48:
// 0.354 against 0.369 ms a step at 68,000 nodes), then the last steps of a
// block's sums together (tree_block_f64: 0.34 ms).
template <int SL, bool SYM>
__global__ void __launch_bounds__(kRowWarps * 32, SL <= 4 ? 8 : 6)
    k_pair_nodes(pp_fused_args a, pp_pairs pr, int parity, Launch l) {
    __shared__ NodeStage stage;
    __shared__ double s_one;
    extern __shared__ double s_stack[];
    if (threadIdx.x == 0) s_one = 1.0;
    __syncthreads();
    const F64Ops op(&s_one);
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int node0 = blockIdx.x * kRowWarps;
    const int i = node0 + warp;
    grid_wait();
    const bool whole = SL > 1 || a.max_neigh == 32;  // a word for every lane
    f64_stage_nodes(a, parity, node0, kRowWarps, stage);
    if (i < a.nnodes) {  // warp-uniform
        const int64_t row = (int64_t)i * a.max_neigh;
        int intact = 0;
        constexpr int kBatch = SL < 4 ? SL : 4;
        const d3 part = tree_lane_f64<SL, kBatch>(
            op, lane, a.max_neigh, s_stack + threadIdx.x, kRowWarps * 32,
            [&](const int(&k)[kBatch], d3(&v)[kBatch]) {
                // all indices of a batch, then all its records
                int sp[kBatch];
#pragma unroll
                for (int b = 0; b < kBatch; ++b) {
                    sp[b] = pr.slot_pair[row + k[b]];
                    if (a.nlist[row + k[b]] == -1) sp[b] = -1;
                }
#pragma unroll
                for (int b = 0; b < kBatch; ++b) {
                    intact += sp[b] != -1;
                    const int64_t p = sp[b] & 0x7FFFFFFF;
                    v[b] = signed_record(pr.force + (SYM ? 4 * p : 8 * p + (sp[b] < 0 ? 4 : 0)),
                                         sp[b]);
                }
            });
        const int count = __reduce_add_sync(kFull, intact);
        if (lane == 0) stage.count[warp] = count;
        if (whole) {
            tree_block_put(s_stack, part);
        } else {
            const double f = tree_warp_f64(op, lane, a.max_neigh, part);
            if (lane == 0) stage.sum[3 * warp] = f;
            if (lane == 16) stage.sum[3 * warp + 1] = f;
            if (lane == 8) stage.sum[3 * warp + 2] = f;
        }
    }
    if (whole) {
        __syncthreads();
        // on other warps from block to block (0.981 against 1.013 ms)
        const int t = (threadIdx.x - 96 * blockIdx.x) & (kRowWarps * 32 - 1);
        if (t < 96) tree_block_f64(op, t, s_stack, stage.sum);
    }
    if (pr.npairs >= kReleasePairs) grid_release();
    f64_node_phase(a, parity, step_mags(l), node0, kRowWarps, stage);
}

template <bool CORR, bool TYPES, bool SYM>
void launch_bonds(const pp_fused_args& a, const pp_pairs& pr, int parity, cudaStream_t st) {
    const int shift = 31 - __builtin_clz((unsigned)a.max_neigh);
    const int64_t grid = (pr.npairs + kPairThreads - 1) / kPairThreads;
    if (grid > 0)
        launch_dependent(k_pair_bonds<CORR, TYPES, SYM>, (unsigned)grid, kPairThreads, 0, st, a, pr,
                         parity, shift);
}

template <int SL>
void launch_nodes(const pp_fused_args& a, const pp_pairs& pr, int parity, const Launch& l,
                  cudaStream_t st) {
    const unsigned grid = (unsigned)((a.nnodes + kRowWarps - 1) / kRowWarps);
    constexpr size_t dyn = tree_stack_bytes<SL == 1 ? 2 : SL>(kRowWarps * 32);
    if (pr.symmetric)
        launch_dependent(k_pair_nodes<SL, true>, grid, kRowWarps * 32, dyn, st, a, pr, parity, l);
    else
        launch_dependent(k_pair_nodes<SL, false>, grid, kRowWarps * 32, dyn, st, a, pr, parity, l);
}

}  // namespace

int validate_pairs(const pp_fused_args& a, const pp_pairs& pr) {
    const int v = validate_fused(a);
    if (v != PP_SUCCESS) return v;
    if (a.precision != PP_FLOAT64) return PP_ERROR_UNSUPPORTED;
    if (pr.npairs < 0 || pr.npairs >= (1ll << 30) || pr.reserved != 0 ||
        pr.reserved2 != 0) return PP_ERROR_INVALID_VALUE;
    if ((int64_t)a.nnodes * a.max_neigh > 0x7FFFFFFFll) return PP_ERROR_UNSUPPORTED;
    if (a.nnodes == 0) return PP_SUCCESS;
    if (!pr.slot_pair || (pr.npairs > 0 && (!pr.slots || !pr.length || !pr.vector || !pr.force)))
        return PP_ERROR_INVALID_VALUE;
    if (pr.symmetric && a.bond_types) return PP_ERROR_INVALID_VALUE;
    if (!aligned32(pr.force) || (reinterpret_cast<uintptr_t>(pr.slots) & 7u)) return PP_ERROR_MISALIGNED;
    return PP_SUCCESS;
}

int launch_pair_step(const pp_fused_args& a, const pp_pairs& pr, int parity, const Launch& l,
                     cudaStream_t st) {
    const bool corr = a.stiffness_corrections != nullptr;
    if (a.bond_types) {
        if (corr)
            launch_bonds<true, true, false>(a, pr, parity, st);
        else
            launch_bonds<false, true, false>(a, pr, parity, st);
    } else if (pr.symmetric) {
        if (corr)
            launch_bonds<true, false, true>(a, pr, parity, st);
        else
            launch_bonds<false, false, true>(a, pr, parity, st);
    } else {
        if (corr)
            launch_bonds<true, false, false>(a, pr, parity, st);
        else
            launch_bonds<false, false, false>(a, pr, parity, st);
    }
    const int rc = launch_status();
    if (rc != PP_SUCCESS) return rc;
    switch (a.max_neigh > 32 ? a.max_neigh / 32 : 1) {
        case 1: launch_nodes<1>(a, pr, parity, l, st); break;
        case 2: launch_nodes<2>(a, pr, parity, l, st); break;
        case 4: launch_nodes<4>(a, pr, parity, l, st); break;
        case 8: launch_nodes<8>(a, pr, parity, l, st); break;
        case 16: launch_nodes<16>(a, pr, parity, l, st); break;
        case 32: launch_nodes<32>(a, pr, parity, l, st); break;
        default: return PP_ERROR_MAX_NEIGH;
    }
    return launch_status();
}

}  // namespace pp

using namespace pp;

static int check_pair_arrays(const pp_fused_args& a) {
    if (a.nnodes < 0) return PP_ERROR_INVALID_VALUE;
    if (!is_pow2_le_1024(a.max_neigh)) return PP_ERROR_MAX_NEIGH;
    if ((int64_t)a.nnodes * a.max_neigh > 0x7FFFFFFFll) return PP_ERROR_UNSUPPORTED;
    if (a.nnodes > 0 && (!a.nlist || !a.r0 || !a.vols)) return PP_ERROR_INVALID_VALUE;
    return PP_SUCCESS;
}

extern "C" int pp_pair_count(const pp_fused_args* args, int32_t* slot_pair, int32_t* row_start,
                             int32_t* scratch, void* stream) {
    if (!args) return PP_ERROR_INVALID_VALUE;
    const int v = check_pair_arrays(*args);
    if (v != PP_SUCCESS) return v;
    if (!row_start) return PP_ERROR_INVALID_VALUE;
    const pp_fused_args& a = *args;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (a.nnodes > 0) {
        if (!slot_pair || !scratch) return PP_ERROR_INVALID_VALUE;
        const unsigned grid = (unsigned)((a.nnodes + kRowWarps - 1) / kRowWarps);
        k_row_order<<<grid, kRowWarps * 32, 0, st>>>(a.nlist, a.nnodes, a.max_neigh, scratch);
        k_pair_partners<<<grid, kRowWarps * 32, 0, st>>>(a.nlist, scratch, a.nnodes, a.max_neigh,
                                                        slot_pair, row_start);
    }
    k_pair_scan<<<1, 1024, 0, st>>>(row_start, a.nnodes);
    return launch_status();
}

extern "C" int pp_pair_fill(const pp_fused_args* args, const pp_pairs* pairs,
                            const int32_t* row_start, int32_t* differ, void* stream) {
    if (!args || !pairs || !differ) return PP_ERROR_INVALID_VALUE;
    const int v = check_pair_arrays(*args);
    if (v != PP_SUCCESS) return v;
    const pp_fused_args& a = *args;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(differ, 0, sizeof(int32_t), st) != cudaSuccess) return PP_ERROR_CUDA;
    if (a.nnodes == 0) return PP_SUCCESS;
    if (!row_start || !pairs->slot_pair || (pairs->npairs > 0 && (!pairs->slots || !pairs->length || !pairs->vector)))
        return PP_ERROR_INVALID_VALUE;
    k_pair_fill<<<(unsigned)((a.nnodes + kRowWarps - 1) / kRowWarps), kRowWarps * 32, 0, st>>>(
        a.nlist, a.r0, a.vols, a.stiffness_corrections, a.nnodes, a.max_neigh, row_start, *pairs,
        differ);
    return launch_status();
}
