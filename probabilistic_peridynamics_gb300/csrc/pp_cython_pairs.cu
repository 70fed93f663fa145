// pp_cython_pairs.cu -- the step of pp_cython.cu with each bond computed once
// and the ordered sums taken by one thread per component.
//
// The Cython loops compute a bond once, with its lower node first, and give
// both nodes that force (peridynamics.pyx:34-99).  Here:
//
//  k_cyp_bonds  one thread per pair (i < j): length, strain, the break test
//               and the terms F vol[j] (added to i) and F vol[i] (subtracted
//               from j) into 32-byte records (one record where the volumes
//               are equal).  Root and quotients come from pp_exact64.cuh: the
//               binary64 pipe is left with 15 additions and products a pair.
//               A pair that breaks marks both rows.
//  k_cyp_rows   one warp per marked or unordered row (the others leave at
//               once): the swap-removals of pp_cython.cu's k_cy_break, then
//               the ordered sum if the row's entries no longer ascend.
//  k_cyp_nodes  one thread per node and component: a row whose entries
//               ascend is summed in row order, which is the reference's
//               order (lower neighbours ascending, then upper ones in row
//               order); force boundary condition, displacement update and
//               new position.  A warp's 32 sums advance together, where a
//               warp per node holds the binary64 pipe for a whole warp per
//               three sums.
#include "pp_pairs.cuh"

namespace pp {
namespace {

constexpr int kPairThreads = 128;
constexpr int kBuildWarps = 8;
constexpr int kRowWarps = 8;  // at most: 48 KB of shared memory a block
constexpr int kNodeThreads = 192;  // 64 nodes
constexpr int kMarked = 1;     // row state: a bond of the row broke this step
constexpr int kUnordered = 2;  // row state: the entries do not ascend

constexpr int kLower = 1;   // entry j < i
constexpr int kUpper = 2;   // entry j > i
constexpr int kBroken = 4;  // the bond breaks this step

__device__ __forceinline__ bool is_bond(int j, int i, int n) { return j >= 0 && j < n && j != i; }

__device__ __forceinline__ int row_count(const int32_t* n_neigh, int i, int width) {
    return min(max(n_neigh[i], 0), width);
}

// Do the first cnt entries of the row name other nodes in ascending order?
// (All lanes of a warp; the answer is the warp's.)
template <class Entry>
__device__ __forceinline__ bool ascends(int lane, int cnt, int i, int n, Entry&& entry) {
    bool ok = true;
    for (int p = lane; p < cnt; p += 32) {
        const int j = entry(p);
        ok = ok && is_bond(j, i, n) && (p == 0 || entry(p - 1) < j);
    }
    return __all_sync(kFull, ok);
}

// Row states, and the pairs each row owns: its entries j > i.
__global__ void __launch_bounds__(kBuildWarps * 32)
    k_cyp_count(const int32_t* __restrict__ nlist, const int32_t* __restrict__ n_neigh, int n,
                int width, int32_t* __restrict__ state, int32_t* __restrict__ row_start) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kBuildWarps + (threadIdx.x >> 5);
    if (i >= n) return;
    const int32_t* row = nlist + (int64_t)i * width;
    const int cnt = row_count(n_neigh, i, width);
    int own = 0;
    for (int p = lane; p < cnt; p += 32) own += row[p] > i && row[p] < n;
    own = __reduce_add_sync(kFull, own);
    const bool up = ascends(lane, cnt, i, n, [&](int p) { return row[p]; });
    if (lane == 0) {
        state[i] = up ? 0 : kUnordered;
        row_start[i + 1] = own;
    }
}

// In-place inclusive scan of start[1..n], start[0] = 0; one CTA.
__global__ void k_cyp_scan(int32_t* __restrict__ start, int n) {
    __shared__ int warp_tot[32];
    __shared__ int carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
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

// The pairs of row i's upper entries, in row order from row_start[i].
__global__ void __launch_bounds__(kBuildWarps * 32)
    k_cyp_fill(const double* __restrict__ coords, const double* __restrict__ vol,
               const int32_t* __restrict__ nlist, const int32_t* __restrict__ n_neigh, int n,
               int width, const int32_t* __restrict__ row_start, pp_cy_pairs pr,
               int32_t* __restrict__ differ) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kBuildWarps + (threadIdx.x >> 5);
    if (i >= n) return;
    const int64_t base = (int64_t)i * width;
    const int cnt = row_count(n_neigh, i, width);
    int next = row_start[i];
    bool diff = false;
    for (int p0 = 0; p0 < cnt; p0 += 32) {
        const int p = p0 + lane;
        const int j = p < cnt ? nlist[base + p] : -1;
        const bool upper = j > i && j < n;
        const unsigned m = __ballot_sync(kFull, upper);
        if (upper) {
            const int q = next + __popc(m & ((1u << lane) - 1u));
            reinterpret_cast<int2*>(pr.nodes)[q] = make_int2(i, j);
            pr.slot_pair[base + p] = q;
            const int64_t oi = 3 * (int64_t)i, oj = 3 * (int64_t)j;
            const double x = dsub(coords[oj], coords[oi]);
            const double y = dsub(coords[oj + 1], coords[oi + 1]);
            const double z = dsub(coords[oj + 2], coords[oi + 2]);
            pr.length[q] = f64_length(dadd(dadd(dmul(x, x), dmul(y, y)), dmul(z, z)));
            diff |= __double_as_longlong(vol[i]) != __double_as_longlong(vol[j]);
        }
        next += __popc(m);
    }
    if (__any_sync(kFull, diff) && lane == 0) atomicOr(differ, 1);
}

// The pair of every lower entry (j < i): the one row j owns for i (the first
// of them, should j list i several times: their values are the same).
__global__ void __launch_bounds__(kBuildWarps * 32)
    k_cyp_lower(const int32_t* __restrict__ nlist, const int32_t* __restrict__ n_neigh, int n,
                int width, const int32_t* state, pp_cy_pairs pr) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kBuildWarps + (threadIdx.x >> 5);
    if (i >= n) return;
    const int64_t base = (int64_t)i * width;
    const int cnt = row_count(n_neigh, i, width);
    for (int p = lane; p < cnt; p += 32) {
        const int j = nlist[base + p];
        if (j > i && j < n) continue;
        int found = -1;
        if (is_bond(j, i, n)) {
            const int32_t* row = nlist + (int64_t)j * width;
            const int len = row_count(n_neigh, j, width);
            if (!(state[j] & kUnordered)) {
                int lo = 0, hi = len;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (row[mid] < i)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                if (lo < len && row[lo] == i) found = lo;
            } else {
                for (int q = 0; q < len && found < 0; ++q)
                    if (row[q] == i) found = q;
            }
            if (found >= 0)
                found = pr.slot_pair[(int64_t)j * width + found] | kReversed;
            else  // (a symmetric list has none) left out by k_cyp_rows
                atomicOr(pr.row_state + i, kUnordered);
        }
        pr.slot_pair[base + p] = found;
    }
}

__global__ void k_cyp_positions(const double* __restrict__ coords, const double* __restrict__ u,
                                double* __restrict__ pos, int64_t ndof) {
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o < ndof) pos[o] = dadd(coords[o], u[o]);
}

// l, strain and fn = strain k / l of a bond of squared length sq.
struct CyBond {
    uint64_t strain, fn;
};

static __device__ __noinline__ CyBond cy_bond_any(double sq, double l0, double k) {
    const double l = dsqrt(sq);
    const double strain = ddiv(dsub(l, l0), l0);
    return {exact64::double_bits(strain), exact64::double_bits(ddiv(dmul(strain, k), l))};
}

// The same from the integer pipe, within the limits of f64_stretch and with
// strain k zero or above 2^-700.
__device__ __forceinline__ CyBond cy_bond(const F64Ops& op, double sq, double l0, double k) {
    using namespace exact64;
    const uint64_t sb = double_bits(sq), lb = double_bits(l0);
    CyBond r{0, 0};
    bool ok = positive_in(sb, 1023 - 400, 1023 + 400) && positive_in(lb, 1023 - 200, 1023 + 200);
    if (ok) {
        const Divisor len = sqrt_rn(sb);
        ok = relative_difference(len, divisor(lb), r.strain);
        const uint64_t num = double_bits(op.mul(bits_double(r.strain), k));
        ok = ok && (is_zero(num) ||
                    positive_in(num & 0x7FFFFFFFFFFFFFFFull, 1023 - 700, 1023 + 700));
        r.fn = div_bits(num, len);
    }
    if (!ok) r = cy_bond_any(sq, l0, k);
    return r;
}

template <bool SYM>
__global__ void __launch_bounds__(kPairThreads, 7)
    k_cyp_bonds(pp_cy_pairs pr, const double* __restrict__ vol, double k, double critical) {
    __shared__ double s_one;
    if (threadIdx.x == 0) s_one = 1.0;
    __syncthreads();
    const F64Ops op(&s_one);
    const int64_t q = blockIdx.x * (int64_t)kPairThreads + threadIdx.x;
    if (q >= pr.npairs) return;
    const int2 ij = reinterpret_cast<const int2*>(pr.nodes)[q];
    if (ij.x < 0) return;  // broken in an earlier step
    const double* ri = pr.position + 3 * (int64_t)ij.x;
    const double* rj = pr.position + 3 * (int64_t)ij.y;
    const d3 d{op.sub(rj[0], ri[0]), op.sub(rj[1], ri[1]), op.sub(rj[2], ri[2])};
    const CyBond b = cy_bond(op, f64_square(op, d), pr.length[q], k);
    double* rec = pr.term + (SYM ? 4 : 8) * q;
    // |strain| < critical, or the bond breaks
    const double size = __longlong_as_double(b.strain & 0x7FFFFFFFFFFFFFFFull);
    if (!f64_less(size, critical)) {
        pr.nodes[2 * q] = -1;
        rec[3] = 1.0;
        atomicOr(pr.row_state + ij.x, kMarked);
        atomicOr(pr.row_state + ij.y, kMarked);
        return;
    }
    const double fn = __longlong_as_double(b.fn);
    const d3 f{op.mul(fn, d.x), op.mul(fn, d.y), op.mul(fn, d.z)};
    const double vj = vol[ij.y];
    store_record(rec, d3{op.mul(f.x, vj), op.mul(f.y, vj), op.mul(f.z, vj)});
    if constexpr (!SYM) {
        const double vi = vol[ij.x];
        store_record(rec + 4, d3{op.mul(f.x, vi), op.mul(f.y, vi), op.mul(f.z, vi)});
    }
}

template <bool SYM>
__device__ __forceinline__ const double* term_of(const pp_cy_pairs& pr, int sp) {
    const int64_t q = sp & 0x7FFFFFFF;
    return pr.term + (SYM ? 4 * q : 8 * q + (sp < 0 ? 4 : 0));
}

// Shared memory per warp and entry: entry, slot pair, flag, order (int32).
template <bool SYM>
__global__ void __launch_bounds__(kRowWarps * 32)
    k_cyp_rows(pp_cy_pairs pr, int32_t* __restrict__ nlist, int32_t* __restrict__ n_neigh, int n,
               int width, double* __restrict__ force) {
    extern __shared__ int32_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * (blockDim.x >> 5) + warp;
    if (i >= n) return;  // warp-uniform
    int state = pr.row_state[i];
    if (state == 0) return;
    int32_t* row = smem + (size_t)warp * 4 * width;
    int32_t* sp = row + width;
    int32_t* flag = sp + width;
    int32_t* order = flag + width;
    int32_t* g = nlist + (int64_t)i * width;
    int32_t* gsp = pr.slot_pair + (int64_t)i * width;
    int cnt = row_count(n_neigh, i, width);
    for (int p = lane; p < cnt; p += 32) {
        const int j = g[p], s = gsp[p];
        int f = 0;
        if (is_bond(j, i, n) && s != -1) {
            f = j < i ? kLower : kUpper;
            // (either record of a pair: both sides break together)
            if ((state & kMarked) && pr.term[(SYM ? 4 : 8) * (int64_t)(s & 0x7FFFFFFF) + 3] != 0.0)
                f |= kBroken;
        }
        row[p] = j;
        sp[p] = s;
        flag[p] = f;
    }
    __syncwarp();
    if (state & kMarked) {
        const int cnt0 = cnt;
        auto move = [&](int to, int from) {
            row[to] = row[from];
            sp[to] = sp[from];
            flag[to] = flag[from];
        };
        // removals by the lower neighbours, in ascending neighbour index
        while (true) {
            int best = INT32_MAX;
            for (int p = lane; p < cnt; p += 32)
                if ((flag[p] & (kLower | kBroken)) == (kLower | kBroken) && row[p] < best)
                    best = row[p];
            best = __reduce_min_sync(kFull, best);
            if (best == INT32_MAX) break;
            int hit = -1;
            for (int p0 = 0; p0 < cnt && hit < 0; p0 += 32) {
                const int p = p0 + lane;
                const unsigned m = __ballot_sync(kFull, p < cnt && row[p] == best);
                if (m) hit = p0 + __ffs(m) - 1;
            }
            if (hit >= 0) {
                if (lane == 0) move(hit, cnt - 1);
                --cnt;
            }
            __syncwarp();
        }
        // the row's own scan: broken upper bonds are swap-removed
        int next = 0;
        while (true) {
            int hit = -1;
            for (int p0 = next; p0 < cnt && hit < 0; p0 += 32) {
                const int p = p0 + lane;
                const unsigned m = __ballot_sync(
                    kFull, p < cnt && (flag[p] & (kUpper | kBroken)) == (kUpper | kBroken));
                if (m) hit = p0 + __ffs(m) - 1;
            }
            if (hit < 0) break;
            if (lane == 0) move(hit, cnt - 1);
            --cnt;
            next = hit;
            __syncwarp();
        }
        __syncwarp();
        for (int p = lane; p < cnt0; p += 32) {
            g[p] = row[p];
            gsp[p] = sp[p];
        }
        state = ascends(lane, cnt, i, n, [&](int p) { return row[p]; }) ? 0 : kUnordered;
        if (lane == 0) {
            n_neigh[i] = cnt;
            pr.row_state[i] = state;
        }
    }
    if (!(state & kUnordered)) return;
    // order of the sum: lower neighbours ascending, then upper ones in row
    // order; entries without a bond are left out
    int lower = 0, used = 0;
    for (int p0 = 0; p0 < cnt; p0 += 32) {
        const int p = p0 + lane;
        const int f = p < cnt ? flag[p] : 0;
        lower += __popc(__ballot_sync(kFull, (f & kLower) != 0));
        used += __popc(__ballot_sync(kFull, (f & (kLower | kUpper)) != 0));
    }
    int upper = lower;
    for (int p0 = 0; p0 < cnt; p0 += 32) {
        const int p = p0 + lane;
        const int f = p < cnt ? flag[p] : 0;
        const unsigned m = __ballot_sync(kFull, (f & kUpper) != 0);
        if (f & kUpper) order[upper + __popc(m & ((1u << lane) - 1u))] = p;
        upper += __popc(m);
        if (f & kLower) {
            // (a neighbour listed twice: its copies in row order; their
            // terms are equal)
            int rank = 0;
            for (int q = 0; q < cnt; ++q)
                rank += (flag[q] & kLower) && (row[q] < row[p] || (row[q] == row[p] && q < p));
            order[rank] = p;
        }
    }
    __syncwarp();
    if (lane < 3) {
        double acc = 0.0;
        for (int r = 0; r < used; ++r) {
            const int s = sp[order[r]];
            const double t = term_of<SYM>(pr, s)[lane];
            acc = s < 0 ? dsub(acc, t) : dadd(acc, t);
        }
        force[3 * (int64_t)i + lane] = acc;
    }
}

template <bool SYM>
__global__ void __launch_bounds__(kNodeThreads)
    k_cyp_nodes(pp_cy_pairs pr, const double* __restrict__ coords,
                const int32_t* __restrict__ n_neigh, int n, int width,
                const double* __restrict__ fc_values, const int32_t* __restrict__ fc_types,
                double fc_scale, const double* __restrict__ bc_values,
                const int32_t* __restrict__ bc_types, double bc_scale, double dt,
                double* __restrict__ force, double* __restrict__ u) {
    __shared__ double s_one;
    if (threadIdx.x == 0) s_one = 1.0;
    __syncthreads();
    const F64Ops op(&s_one);
    const int64_t o = blockIdx.x * (int64_t)kNodeThreads + threadIdx.x;
    if (o >= 3 * (int64_t)n) return;
    const int i = (int)(o / 3), c = (int)(o - 3 * (int64_t)i);
    double acc = 0.0;
    if (pr.row_state[i] & kUnordered) {
        acc = force[o];
    } else {
        const int32_t* sp = pr.slot_pair + (int64_t)i * width;
        const int cnt = row_count(n_neigh, i, width);
        constexpr int kAhead = 4;
        int p = 0;
        for (; p + kAhead <= cnt; p += kAhead) {
            int s[kAhead];
            double t[kAhead];
#pragma unroll
            for (int a = 0; a < kAhead; ++a) s[a] = sp[p + a];
#pragma unroll
            for (int a = 0; a < kAhead; ++a) t[a] = term_of<SYM>(pr, s[a])[c];
#pragma unroll
            for (int a = 0; a < kAhead; ++a) {
                // acc -+ t, the sign flipped by bits
                const long long flip = s[a] < 0 ? (long long)0x8000000000000000ull : 0;
                acc = op.add(__longlong_as_double(__double_as_longlong(t[a]) ^ flip), acc);
            }
        }
        for (; p < cnt; ++p) {
            const int s = sp[p];
            const long long flip = s < 0 ? (long long)0x8000000000000000ull : 0;
            acc = op.add(__longlong_as_double(__double_as_longlong(term_of<SYM>(pr, s)[c]) ^ flip),
                         acc);
        }
    }
    if (fc_types[o] != 0) acc = dadd(acc, dmul(fc_scale, fc_values[o]));
    force[o] = acc;
    const double x = bc_types[o] == 0 ? op.add(u[o], op.mul(dt, acc)) : dmul(bc_scale, bc_values[o]);
    u[o] = x;
    pr.position[o] = op.add(coords[o], x);
}

int check_pairs(const pp_cy_pairs* pr, int32_t nnodes, int32_t width) {
    if (!pr || nnodes < 0 || width < 0) return PP_ERROR_INVALID_VALUE;
    if (width > 1024) return PP_ERROR_MAX_NEIGH;
    if ((int64_t)nnodes * width > 0x7FFFFFFFll) return PP_ERROR_UNSUPPORTED;
    if (pr->npairs < 0 || pr->npairs >= (1ll << 30) || pr->reserved != 0)
        return PP_ERROR_INVALID_VALUE;
    if (nnodes == 0) return PP_SUCCESS;
    if (!pr->row_state || !pr->position || (width > 0 && !pr->slot_pair) ||
        (pr->npairs > 0 && (!pr->nodes || !pr->length)))
        return PP_ERROR_INVALID_VALUE;
    return PP_SUCCESS;
}

}  // namespace
}  // namespace pp

using namespace pp;

extern "C" int pp_cy_pair_count(const int32_t* nlist, const int32_t* n_neigh, int32_t nnodes,
                                int32_t width, int32_t* row_state, int32_t* row_start,
                                void* stream) {
    if (nnodes < 0 || width < 0 || !row_start) return PP_ERROR_INVALID_VALUE;
    if (width > 1024) return PP_ERROR_MAX_NEIGH;
    if ((int64_t)nnodes * width > 0x7FFFFFFFll) return PP_ERROR_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (nnodes > 0) {
        if ((width > 0 && !nlist) || !n_neigh || !row_state) return PP_ERROR_INVALID_VALUE;
        k_cyp_count<<<(unsigned)((nnodes + kBuildWarps - 1) / kBuildWarps), kBuildWarps * 32, 0,
                      st>>>(nlist, n_neigh, nnodes, width, row_state, row_start);
    }
    k_cyp_scan<<<1, 1024, 0, st>>>(row_start, nnodes);
    return launch_status();
}

extern "C" int pp_cy_pair_fill(const double* coords, const double* u, const double* volume,
                               const int32_t* nlist, const int32_t* n_neigh, int32_t nnodes,
                               int32_t width, const int32_t* row_start, const pp_cy_pairs* pairs,
                               int32_t* differ, void* stream) {
    const int v = check_pairs(pairs, nnodes, width);
    if (v != PP_SUCCESS) return v;
    if (!differ) return PP_ERROR_INVALID_VALUE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(differ, 0, sizeof(int32_t), st) != cudaSuccess) return PP_ERROR_CUDA;
    if (nnodes == 0) return PP_SUCCESS;
    if (!coords || !u || !volume || (width > 0 && !nlist) || !n_neigh || !row_start)
        return PP_ERROR_INVALID_VALUE;
    const unsigned grid = (unsigned)((nnodes + kBuildWarps - 1) / kBuildWarps);
    k_cyp_fill<<<grid, kBuildWarps * 32, 0, st>>>(coords, volume, nlist, n_neigh, nnodes, width,
                                                  row_start, *pairs, differ);
    k_cyp_lower<<<grid, kBuildWarps * 32, 0, st>>>(nlist, n_neigh, nnodes, width, pairs->row_state,
                                                   *pairs);
    const int64_t ndof = 3 * (int64_t)nnodes;
    k_cyp_positions<<<(unsigned)((ndof + 255) / 256), 256, 0, st>>>(coords, u, pairs->position,
                                                                    ndof);
    return launch_status();
}

namespace pp {
namespace {

template <bool SYM>
int cy_pair_step(const pp_cy_pairs& pr, const pp_cy_step& a, cudaStream_t st) {
    if (pr.npairs > 0)
        k_cyp_bonds<SYM><<<(unsigned)((pr.npairs + kPairThreads - 1) / kPairThreads), kPairThreads,
                           0, st>>>(pr, a.volume, a.bond_stiffness, a.critical_strain);
    const size_t per_warp = (size_t)(a.width > 0 ? a.width : 1) * 4 * sizeof(int32_t);
    int warps = kRowWarps;  // (a row of 1024 entries takes 16 KB)
    while (warps * per_warp > 48 * 1024) warps >>= 1;
    k_cyp_rows<SYM><<<(unsigned)((a.nnodes + warps - 1) / warps), warps * 32, warps * per_warp,
                      st>>>(pr, a.nlist, a.n_neigh, a.nnodes, a.width, a.force);
    const int64_t ndof = 3 * (int64_t)a.nnodes;
    k_cyp_nodes<SYM><<<(unsigned)((ndof + kNodeThreads - 1) / kNodeThreads), kNodeThreads, 0,
                       st>>>(pr, a.coords, a.n_neigh, a.nnodes, a.width, a.force_bc_values,
                             a.force_bc_types, a.force_bc_scale, a.bc_values, a.bc_types,
                             a.bc_scale, a.dt, a.force, a.u);
    return launch_status();
}

}  // namespace
}  // namespace pp

extern "C" int pp_cy_pair_step(const pp_cy_step* args, const pp_cy_pairs* pairs, void* stream) {
    if (!args) return PP_ERROR_INVALID_VALUE;
    const pp_cy_step& a = *args;
    const int v = check_pairs(pairs, a.nnodes, a.width);
    if (v != PP_SUCCESS) return v;
    if (a.nnodes == 0) return PP_SUCCESS;
    if (!a.coords || !a.u || !a.volume || (a.width > 0 && !a.nlist) || !a.n_neigh || !a.force ||
        !a.force_bc_values || !a.force_bc_types || !a.bc_values || !a.bc_types)
        return PP_ERROR_INVALID_VALUE;
    if (pairs->npairs > 0 && !pairs->term) return PP_ERROR_INVALID_VALUE;
    if (!aligned32(pairs->term) || (reinterpret_cast<uintptr_t>(pairs->nodes) & 7u))
        return PP_ERROR_MISALIGNED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return pairs->symmetric ? cy_pair_step<true>(*pairs, a, st) : cy_pair_step<false>(*pairs, a, st);
}
