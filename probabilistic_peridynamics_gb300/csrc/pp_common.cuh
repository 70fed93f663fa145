// pp_common.cuh -- device helpers shared by the step kernels.
//
// * Exact binary64 operations (__dadd_rn & co.) so that no compiler flag can
//   contract or reorder the reference arithmetic of peripy/cl/*.cl.
// * The work-group tree reduction of peripy/cl/peridynamics.cl:105-115,
//   restated for one warp per node: lane l owns slots l, l+32, l+64, ...;
//   the first log2(max_neigh/32) tree steps combine a lane's own slots in
//   registers, the last five are warp shuffles.  The association order is
//   the same as the work-group tree, so binary64 sums are bit-identical.
// * Double-float ("FP32 pair") arithmetic for the mixed-precision node state
//   (error-free transformations: Knuth's TwoSum, Dekker's Fast2Sum and the
//   FMA-based TwoProduct; the pair operations follow the double-double
//   algorithms of Hida, Li and Bailey's QD library, restated for float).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/pp_gb300.h"

namespace pp {

constexpr unsigned kFull = 0xffffffffu;

// ---------------------------------------------------------------- binary64
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double dsqrt(double a) { return __dsqrt_rn(a); }

struct d3 {
    double x, y, z;
};

__device__ __forceinline__ d3 d3_zero() { return d3{0.0, 0.0, 0.0}; }
__device__ __forceinline__ d3 d3_add(d3 a, d3 b) {
    return d3{dadd(a.x, b.x), dadd(a.y, b.y), dadd(a.z, b.z)};
}
__device__ __forceinline__ d3 d3_shfl_down(d3 v, int off) {
    return d3{__shfl_down_sync(kFull, v.x, off), __shfl_down_sync(kFull, v.y, off),
              __shfl_down_sync(kFull, v.z, off)};
}

// Additions and products as fused multiply-adds: a + b = fma(a, 1, b) and
// a b = fma(a, b, -0) are the same correctly rounded values (signed zeros
// included).  On GB300 a DFMA whose three operands are registers issues every
// 17 clocks per warp and SM, a DADD or DMUL every 20 (measured 1.89 against
// 1.59 lanes/clk/SM), so the constants are kept in registers that the
// compiler cannot see through.
struct F64Ops {
    double one, nzero;
    // `word`: a shared word of the block, written before a barrier
    __device__ __forceinline__ explicit F64Ops(const volatile double* word) {
        one = *word;
        nzero = __longlong_as_double(__double_as_longlong(one) ^ 0xBFF0000000000000ll);
    }
    __device__ __forceinline__ double add(double a, double b) const { return __fma_rn(a, one, b); }
    __device__ __forceinline__ double sub(double a, double b) const { return __fma_rn(-b, one, a); }
    __device__ __forceinline__ double mul(double a, double b) const { return __fma_rn(a, b, nzero); }
};

// Programmatic dependent launch: a kernel launched by launch_dependent may be
// brought up before the one before it in the stream has ended; each of its
// threads calls grid_wait() before it reads or writes memory, which returns
// when that one is complete and its writes are visible.  Not for kernels with
// `const __restrict__` parameters or read-only loads at addresses known before
// the wait, which the compiler may move ahead of it.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The next kernel may be brought up when every block has come here or ended.
__device__ __forceinline__ void grid_release() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... Params, class... Args>
void launch_dependent(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem,
                      cudaStream_t st, const Args&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, Params(args)...);  // (launch_status() has its error)
}

__device__ __forceinline__ double shfl_xor(double v, int off) {
    return __shfl_xor_sync(kFull, v, off);
}

// Levels of pending sums that tree_reduce_f64 keeps per thread.
template <int SL>
struct TreeLevels {
    static constexpr int value = 1 + TreeLevels<SL / 2>::value;
};
template <>
struct TreeLevels<1> {
    static constexpr int value = 0;
};

// Bytes of tree_reduce_f64's stack for a block.
template <int SL>
constexpr size_t tree_stack_bytes(int threads) {
    return sizeof(double) * 3 * TreeLevels<SL>::value * threads;
}

// Reduce per-slot binary64 vectors of one node held by one warp, in the
// work-group tree order, down to one vector a lane.  SL = slots per lane =
// max(1, L/32).  `slot(k)` returns the contribution of slot k and is called
// exactly once for every slot < L (and for no other), on all lanes together.
//
// A lane's slots come in bit-reversed order, so that the tree's first
// log2(SL) steps need one pending sum per level: `stack` (shared memory, 3
// log2(SL) words per thread, `stride` threads) holds the finished left half
// of the pair that a later slot completes.  The loop stays rolled (one copy
// of the slot's code, whatever SL), and the additions are branched around,
// not predicated: a predicated DADD still takes the binary64 pipe's time.
//
// B slots of a lane are asked for together: slot(k, v) fills v[b] for slots
// k[b], b < B (a power of two up to SL).  One at a time keeps the registers of
// long slot code down; four at once keep four loads in flight.
template <int SL, int B, class SlotFn>
__device__ __forceinline__ d3 tree_lane_f64(const F64Ops& op, int lane, int L, double* stack,
                                            int stride, SlotFn&& slot) {
    static_assert(SL % B == 0, "whole batches");
    d3 v = d3_zero();
    if constexpr (SL == 1) {
        if (lane < L) {
            const int k[1] = {lane};
            d3 one[1];
            slot(k, one);
            v = one[0];
        }
    } else {
        auto add = [&](const d3& a, const d3& b) {
            return d3{op.add(a.x, b.x), op.add(a.y, b.y), op.add(a.z, b.z)};
        };
#pragma unroll 1
        for (int n = 0; n < SL / B; ++n) {
            int k[B];
            d3 w[B];
#pragma unroll
            for (int b = 0; b < B; ++b)
                k[b] = lane + 32 * static_cast<int>(__brev(n * B + b) >>
                                                    (32 - TreeLevels<SL>::value));
            slot(k, w);
            // the batch's own levels of the tree
#pragma unroll
            for (int s = 1; s < B; s <<= 1) {
#pragma unroll
                for (int b = 0; b < B; b += 2 * s) w[b] = add(w[b], w[b + s]);
            }
            v = w[0];
            double* p = stack;
            int m = n;
#pragma unroll 1
            while (m & 1) {
                v = add(d3{p[0], p[stride], p[2 * stride]}, v);
                p += 3 * stride;
                m >>= 1;
            }
            if (n != SL / B - 1) {
                p[0] = v.x;
                p[stride] = v.y;
                p[2 * stride] = v.z;
            }
        }
    }
    return v;
}

// The last steps of the tree, over the lanes of a node's warp.  Returns the
// sum's x on lane 0, z on lane 8 and y on lane 16.  Rows of 32 slots or more
// pack the components: a step's lower half computes one component while the
// upper half computes another (addition commutes, so the sums are the tree's
// own): 6 additions a warp instead of 15.
__device__ __forceinline__ double tree_warp_f64(const F64Ops& op, int lane, int L, d3 v) {
    if (L < 32) {
        for (int off = L >> 1; off >= 1; off >>= 1) v = d3_add(v, d3_shfl_down(v, off));
        const double y = __shfl_sync(kFull, v.y, 0), z = __shfl_sync(kFull, v.z, 0);
        return lane == 0 ? v.x : (lane == 8 ? z : y);
    }
    const bool up16 = lane & 16, up8 = lane & 8;
    const double xy = op.add(up16 ? v.y : v.x, shfl_xor(up16 ? v.x : v.y, 16));
    const double z = op.add(v.z, shfl_xor(v.z, 16));
    double t = op.add(up8 ? z : xy, shfl_xor(up8 ? xy : z, 8));
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1) t = op.add(t, shfl_xor(t, off));
    return t;
}

// Both parts of the tree.
template <int SL, int B, class SlotFn>
__device__ __forceinline__ double tree_reduce_f64(const F64Ops& op, int lane, int L, double* stack,
                                                  int stride, SlotFn&& slot) {
    return tree_warp_f64(op, lane, L, tree_lane_f64<SL, B>(op, lane, L, stack, stride, slot));
}

// tree_warp_f64 for the eight nodes of a block of eight warps together (rows
// of 32 slots or more): 24 sums of 32 words, four lanes a sum, on three of
// the warps.  27 additions a block instead of 48 (the step on pairs: 400,000
// nodes in rows of 128 slots 0.981 ms with, 1.020 without; 200,000 nodes in
// rows of 32 0.201 and 0.223; 2,000 nodes 9.7 us and 10.4).  The words lie
// where the lanes' stacks are: room of their own leaves less L1 to the records
// (0.307 against 0.297 ms where every direction has a record).
__device__ __forceinline__ void tree_block_put(double* stack, const d3& v) {
    double* p = stack + threadIdx.x;
    p[0] = v.x;
    p[256] = v.y;
    p[512] = v.z;
}

// After a barrier, by threads t = 0 .. 95: sum[3 node + component].  A sum's
// lane takes words a + 4 (k ^ node): the steps of the tree pair k with k ^ 4,
// k ^ 2 and k ^ 1, whatever k counts from, and eight sums read all banks.
__device__ __forceinline__ void tree_block_f64(const F64Ops& op, int t, const double* stack,
                                               double* sum) {
    const int node = (t >> 2) & 7;
    const double* p = stack + (t >> 5) * 256 + node * 32 + (t & 3);
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = p[4 * (k ^ node)];
#pragma unroll
    for (int s = 4; s >= 1; s >>= 1) {
#pragma unroll
        for (int k = 0; k < s; ++k) v[k] = op.add(v[k], v[k + s]);
    }
    double w = op.add(v[0], shfl_xor(v[0], 2));
    w = op.add(w, shfl_xor(w, 1));
    if ((t & 3) == 0) sum[3 * node + (t >> 5)] = w;
}

// ------------------------------------------------------------ double-float
struct df {
    float hi, lo;
};

// Knuth's TwoSum: s + e == a + b exactly.
__device__ __forceinline__ df two_sum(float a, float b) {
    float s = __fadd_rn(a, b);
    float bb = __fsub_rn(s, a);
    float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return df{s, e};
}
// Dekker's Fast2Sum (requires |a| >= |b| or a == 0).
__device__ __forceinline__ df fast_two_sum(float a, float b) {
    float s = __fadd_rn(a, b);
    float e = __fsub_rn(b, __fsub_rn(s, a));
    return df{s, e};
}
__device__ __forceinline__ df df_add(df a, df b) {
    df s = two_sum(a.hi, b.hi);
    df t = two_sum(a.lo, b.lo);
    s.lo = __fadd_rn(s.lo, t.hi);
    s = fast_two_sum(s.hi, s.lo);
    s.lo = __fadd_rn(s.lo, t.lo);
    return fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ df df_add_f(df a, float b) {
    df s = two_sum(a.hi, b);
    s.lo = __fadd_rn(s.lo, a.lo);
    return fast_two_sum(s.hi, s.lo);
}
// TwoProduct via FMA, plus cross terms.
__device__ __forceinline__ df df_mul(df a, df b) {
    float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    return fast_two_sum(p, e);
}
__device__ __forceinline__ df df_mul_f(df a, float b) {
    float p = __fmul_rn(a.hi, b);
    float e = __fmaf_rn(a.hi, b, -p);
    e = __fmaf_rn(a.lo, b, e);
    return fast_two_sum(p, e);
}
__device__ __forceinline__ df df_from_double(double x) {
    float hi = __double2float_rn(x);
    float lo = __double2float_rn(x - (double)hi);
    return df{hi, lo};
}
__device__ __forceinline__ double df_to_double(df a) {
    return (double)a.hi + (double)a.lo;  // exact: |lo| <= ulp(hi)/2
}

// ------------------------------------------------------------- utilities
__device__ __forceinline__ float4 ldg_f4(const float* p, int64_t i) {
    return __ldg(reinterpret_cast<const float4*>(p) + i);
}
__device__ __forceinline__ int4 ldg_i4(const int32_t* p, int64_t i) {
    return __ldg(reinterpret_cast<const int4*>(p) + i);
}

inline bool is_pow2_le_1024(int32_t x) { return x >= 1 && x <= 1024 && (x & (x - 1)) == 0; }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }

inline int launch_status() {
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PP_SUCCESS : PP_ERROR_CUDA;
}

}  // namespace pp
