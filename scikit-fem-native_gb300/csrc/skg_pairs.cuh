// Pair plan: sums of symmetric element matrices into a square CSR pattern.
//
// A pattern whose row and column DOFs coincide has a symmetric structure, and
// every symmetric element matrix adds the same number to (r, c) and (c, r)
// (three components per node: a 3 x 3 block and its transpose).  The plan
// lists, for each node pair r <= c of the pattern, the positions of its
// contributions in the packed element matrices (upper triangle of node blocks,
// n (n + 1) / 2 per element): one thread sums an entry of a pair in element
// order and writes both places.  No atomics and no accumulators in shared
// memory; each value is written once, by one thread, in a fixed order of
// additions: bitwise reproducible.
//
// Why pairs: an FP64 instruction costs the pipe the same for 1 lane as for 32
// (9.3 to 9.7 ns per DADD, warp and SM, for 1 to 32 active lanes), and walking the
// rows' incidences issues additions for warps whose rows end at different
// times, with a load and a store of shared memory for each.  A pair needs one
// addition less than it has contributions, in nearly full warps, and half of
// the entries are neither stored, loaded nor added: 42 FP64 additions per P2
// element (32^3, counted) instead of 95, 440 bytes per element matrix instead of 800.
//
// Slices: the pairs are taken in row order in windows of kPairWindow; inside a
// window they are sorted by their number of contributions, so that the 32
// pairs of a slice have about the same number, and a slice's positions are
// stored transposed (contribution k of the 32 pairs together): index loads
// coalesce and few lanes idle.  The windows are ordered by the last element
// they need, so that the sums can follow the element pass step by step.
#pragma once

#include <algorithm>
#include <type_traits>
#include <vector>

#include "skg_common.cuh"
#include "skg_df64.cuh"
#include "skg_rows.cuh"

namespace skg {

constexpr int kPairWindow = 1024;
constexpr uint32_t kPairNone = 0xffffffffu;
// Plans of three components: set in the codes of the contributions whose first
// node is the later local node (the stored block is read transposed).
constexpr uint32_t kPairTurned = 0x80000000u;
// Elements per tile (one block) of the element passes.
constexpr int kTile = 128;

// Packed element matrices lie entry by entry: entry (block) t of element e at
// t * stride + e, so that the threads of an element pass (one element each)
// store whole lines without a stage in shared memory, whose size would limit
// the warps that keep the FP64 pipe fed.
inline int64_t block_stride(int64_t ne) { return (ne + kTile - 1) / kTile * kTile; }

// Packed upper triangle of an n x n (block) matrix, a <= b.
__host__ __device__ constexpr int tri_index(int n, int a, int b) { return a * n - a * (a - 1) / 2 + (b - a); }

// Scale exponent and range flag of the FP32-pair modes, set to 0x80 bytes
// before (none, in range; see launch_scale_exponent): the FP64 passes take
// over when a value left the FP32 range or no coordinate gave a scale.
__device__ __forceinline__ bool out_of_range(const int *__restrict__ misc) {
    return misc[1] == 1 || misc[0] < -(1 << 20);
}

// ------------------------------------------------------------------- sums
// Sums run in T: FP64, or double-float (FP32 pairs) for the FP32-pair modes.

__device__ __forceinline__ void pair_add(double &a, double v) { a += v; }
__device__ __forceinline__ void pair_add(df64 &a, df64 v) {  // renormalised once, by `finish`
    const df64 sm = two_sum(a.hi, v.hi);
    a.hi = sm.hi;
    a.lo += sm.lo + v.lo;
}

// -0.0 leaves any sum unchanged: the value of the missing contributions.
template <class T>
__device__ __forceinline__ T pair_zero();
template <>
__device__ __forceinline__ double pair_zero<double>() { return -0.0; }
template <>
__device__ __forceinline__ df64 pair_zero<df64>() { return df64{-0.f, -0.f}; }

// Entry `code` of the packed element matrices (FP64, (hi, lo) pairs, FP32).
__device__ __forceinline__ void pair_load(const double *__restrict__ K, uint32_t code, double &v) {
    v = __ldg(K + code);
}
__device__ __forceinline__ void pair_load(const float2 *__restrict__ K, uint32_t code, df64 &v) {
    const float2 x = __ldg(K + code);
    v = df64{x.x, x.y};
}
__device__ __forceinline__ void pair_load(const float *__restrict__ K, uint32_t code, df64 &v) {
    v = df64{__ldg(K + code), 0.f};
}

// Lower-triangle buffer of the element matrices (same packing, entry (b, a) at
// the position of (a, b)); read only when `any` is set, for the elements of
// the tiles (of kTile consecutive elements) that are flagged.
template <class E>
struct PairLower {
    const E *K = nullptr;
    const int *any = nullptr;
    const uint8_t *tiles = nullptr;
    uint32_t stride = 1;
};

struct PairArrays {
    const int32_t *slice_ptr;
    const uint32_t *codes, *orient;
    const uint2 *slots;
    const uint4 *slots3;
};

inline PairArrays pair_arrays(const PairPlan &p) {
    return PairArrays{p.slice_ptr, p.codes, p.orient, p.slots, p.slots3};
}

struct PairIdentity {
    __device__ double operator()(double v) const { return v; }
};

// Double-float sums in units scaled by 2^-*s: exact conversion.
struct PairUnscale {
    const int *s;
    __device__ double operator()(df64 v) const { return df_to_double(fast_two_sum(v.hi, v.lo), *s); }
};

constexpr int kPairWarps = 16;
constexpr int kPairSlices = kPairWindow / 32 / kPairWarps;  // of a window, per warp

// Scalar plans (block 1): one block per window, each warp takes two of its
// slices at once, so that their chains of dependent loads (slice -> codes ->
// entries) overlap.  T: the sums' type, E: the stored entries'; `finish`
// converts a sum to the FP64 value.  With `redo`, the pass runs only when the
// FP32-pair pass before it left its range (and its blocks walk the windows:
// the launch that finds nothing to do is small; otherwise windows go to the
// blocks in order, which keeps the element data and the values of neighbouring
// rows in L2 together).
template <class T, class E, class F>
__global__ void __launch_bounds__(kPairWarps * 32) k_pair_sum(int w0, int w1, PairArrays p, const E *__restrict__ K,
                                                             PairLower<E> lower, F finish,
                                                             const int *__restrict__ redo,
                                                             double *__restrict__ values) {
    if (redo && !out_of_range(redo)) return;
    const bool general = lower.any && *lower.any == 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int w = w0 + blockIdx.x; w < w1; w += gridDim.x) {
        const int s = w * (kPairWindow / 32) + warp;
        if (general) {  // an element matrix is not symmetric: the two values are summed apart
            for (int q = 0; q < kPairSlices; ++q) {
                const int sq = s + q * kPairWarps;
                const int32_t k0 = p.slice_ptr[sq], n = p.slice_ptr[sq + 1] - k0;
                const uint32_t *cs = p.codes + (int64_t)k0 * 32 + lane;
                const uint2 to = p.slots[(int64_t)sq * 32 + lane];
                T up = pair_zero<T>(), lo = pair_zero<T>();
                for (int k = 0; k < n; ++k) {
                    const uint32_t c = __ldg(cs + k * 32);
                    if (c == kPairNone) continue;
                    const bool turned = (__ldg(p.orient + k0 + k) >> lane) & 1u;
                    T a, b;
                    pair_load(K, c, a);
                    b = a;
                    if (lower.tiles[c % lower.stride / (uint32_t)kTile]) pair_load(lower.K, c, b);
                    pair_add(up, turned ? b : a);
                    pair_add(lo, turned ? a : b);
                }
                if (to.x != kPairNone) values[to.x] = finish(up);
                if (to.y != kPairNone) values[to.y] = finish(lo);
            }
            continue;
        }
        int32_t k0[kPairSlices], n[kPairSlices];
        uint2 to[kPairSlices];
        uint32_t c[kPairSlices][2];
        T v[kPairSlices][2];
#pragma unroll
        for (int q = 0; q < kPairSlices; ++q) {
            k0[q] = p.slice_ptr[s + q * kPairWarps];
            n[q] = p.slice_ptr[s + q * kPairWarps + 1] - k0[q];
            to[q] = __ldcs(p.slots + (int64_t)(s + q * kPairWarps) * 32 + lane);
        }
#pragma unroll
        for (int q = 0; q < kPairSlices; ++q)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                c[q][j] = j < n[q] ? __ldcs(p.codes + (int64_t)(k0[q] + j) * 32 + lane) : kPairNone;
#pragma unroll
        for (int q = 0; q < kPairSlices; ++q)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                v[q][j] = pair_zero<T>();
                if (c[q][j] != kPairNone) pair_load(K, c[q][j], v[q][j]);
            }
#pragma unroll
        for (int q = 0; q < kPairSlices; ++q) {
            T sum = v[q][0];
            if (n[q] > 1) pair_add(sum, v[q][1]);
            const uint32_t *cs = p.codes + (int64_t)(k0[q] + 2) * 32 + lane;
            const auto batch = [&](auto count) {  // whole batches: no instruction is issued for nothing
                constexpr int N = decltype(count)::value;
                uint32_t d[N];
                T x[N];
#pragma unroll
                for (int j = 0; j < N; ++j) d[j] = __ldcs(cs + j * 32);
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    x[j] = pair_zero<T>();
                    if (d[j] != kPairNone) pair_load(K, d[j], x[j]);
                }
#pragma unroll
                for (int j = 0; j < N; ++j) pair_add(sum, x[j]);
                cs += N * 32;
            };
            int left = n[q] - 2;
            for (; left >= 4; left -= 4) batch(std::integral_constant<int, 4>{});
            if (left == 3) batch(std::integral_constant<int, 3>{});
            if (left == 2) batch(std::integral_constant<int, 2>{});
            if (left == 1) batch(std::integral_constant<int, 1>{});
            const double r = finish(sum);
            if (to[q].x != kPairNone) values[to[q].x] = r;
            if (to[q].y != kPairNone) values[to[q].y] = r;
        }
    }
}

// Slices [s0, s1), whole windows.
template <class T, class E, class F>
inline void pair_sum(const PairPlan &plan, int s0, int s1, const E *K, const PairLower<E> &lower, F finish,
                     const int *redo, double *values, cudaStream_t s) {
    const int w0 = s0 / (kPairWindow / 32), w1 = s1 / (kPairWindow / 32);
    if (w1 <= w0) return;
    const unsigned n = (unsigned)(w1 - w0);
    k_pair_sum<T><<<redo ? std::min(n, 4u * kSmCount) : n, kPairWarps * 32, 0, s>>>(w0, w1, pair_arrays(plan), K, lower,
                                                                                    finish, redo, values);
    SKG_LAUNCH_CHECK("pair_sum");
}

// Three components per node: packed blocks (np, stride, 3, 3); the blocks t of
// 32 elements are one contiguous, 16-byte aligned range.  A block of threads
// per slice, nine threads per pair.
constexpr int kPairBlock3 = 288;

__global__ void __launch_bounds__(kPairBlock3) k_pair_sum3(int s0, PairArrays p, const double *__restrict__ K,
                                                           double *__restrict__ values);

// Packed triangles / blocks to full matrices, for patterns without a plan.
void expand_packed(int64_t ne, int n, const double *K, double *full, cudaStream_t s);
void expand_blocks(int64_t ne, int n, const double *K, double *full, cudaStream_t s);

inline void pair_sum3(const PairPlan &plan, int s0, int s1, const double *K, double *values, cudaStream_t s) {
    if (s1 <= s0) return;
    k_pair_sum3<<<(unsigned)(s1 - s0), kPairBlock3, 0, s>>>(s0, pair_arrays(plan), K, values);
    SKG_LAUNCH_CHECK("pair_sum3");
}

// A plan of the packed 3 x 3 blocks of `nodes` nodes: by pairs of nodes, or (four
// nodes) by pairs of DOFs that are not numbered node by node.
inline bool has_block_plan(const skg_pattern *pat, int nodes) {
    return (pat->pairs.block == 3 && pat->pairs.nodes == nodes) ||
           (nodes == 4 && pat->pairs.block == 1 && pat->pairs.nodes == 12);
}

inline void block_sums(const PairPlan &plan, int s0, int s1, const double *K, double *values, cudaStream_t s) {
    if (plan.block == 3) pair_sum3(plan, s0, s1, K, values, s);
    else pair_sum<double>(plan, s0, s1, K, PairLower<double>{}, PairIdentity{}, nullptr, values, s);
}

// ----------------------------------------------------------------- passes

// Element pass and pair sums; elem(e0, e1) launches the element pass over
// elements [e0, e1) on s (e0 a multiple of kTile), sums(slice0, slice1, s) the
// sums of a range of slices.
//
// Device output, or a host output of fewer than kHostChunkMinNnz values: one
// launch of each pass, then one copy.  (In steps the passes lose more to their
// launches' first and last waves than meeting in L2 or running side by side
// gains: P2 FP64 at 64^3 1.01 ms in one step, 1.10 in four and 1.22 in eight
// on one stream, 1.60 in eight on two streams.)  Large host output: in steps on
// s, each followed by the copies of the row chunks that it completes on the
// copy stream, which hide the steps.  tail(cs) queues what follows the sums on
// s; what it copies to the host goes on cs (ordered after s when it is another
// stream), before the values' last copies are waited for.
struct NoTail {
    void operator()(cudaStream_t) const {}
};

template <class FE, class FS, class FT = NoTail>
void run_pair_passes(const skg_pattern *pat, int64_t ne, double *d_values, double *h_values, cudaStream_t s, FE &&elem,
                     FS &&sums, FT &&tail = NoTail{}) {
    const PairPlan &plan = pat->pairs;
    if (!h_values || plan.copies.empty()) {
        if (ne) elem((int64_t)0, ne);
        sums(0, plan.n_slices, s);
        tail(s);
        if (h_values && pat->nnz)
            SKG_CUDA(cudaMemcpyAsync(h_values, d_values, (size_t)pat->nnz * sizeof(double), cudaMemcpyDeviceToHost, s));
        return;
    }
    EventSet ev;
    cudaStream_t cs = side_stream(Side::copy);
    try {
        ev.order(s, cs);  // the previous call's use of the host values
        int64_t done = 0;
        int32_t slice = 0;
        size_t copied = 0;
        for (const PairStep &st : plan.steps) {
            const int64_t to = std::min(ne, (st.ready + kTile - 1) / kTile * kTile);  // whole tiles
            if (to > done) {
                elem(done, to);
                done = to;
            }
            sums(slice, st.slice, s);
            slice = st.slice;
            bool waits = false;
            for (; copied < plan.copies.size() && plan.copies[copied].slice <= slice; ++copied) {
                const PairCopy &c = plan.copies[copied];
                if (!waits) ev.order(s, cs);
                waits = true;
                if (c.slot1 > c.slot0)
                    SKG_CUDA(cudaMemcpyAsync(h_values + c.slot0, d_values + c.slot0,
                                             (size_t)(c.slot1 - c.slot0) * sizeof(double), cudaMemcpyDeviceToHost, cs));
            }
        }
        if (done < ne) elem(done, ne);  // elements no row references
        tail(cs);
        ev.order(cs, s);
    } catch (...) {
        // scratch freed on s after this call must outlive the queued work
        cudaEvent_t e;
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess) {
            cudaEventRecord(e, cs);
            cudaStreamWaitEvent(s, e, 0);
            cudaEventDestroy(e);
        }
        throw;
    }
}

// A block's element vectors, staged in shared memory (16-byte aligned), to
// global memory as one bulk copy: the tile is one contiguous range, and the
// copy engine writes it without load / store instructions of the threads.
// Every thread of the block calls it after its last store to the stage; the
// stage may be written again, and the block may end, when it returns.  `dst`
// is 16-byte aligned; the bytes past a multiple of 16 go by plain stores.
__device__ __forceinline__ void store_tile(const void *stage, void *dst, int bytes) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    const int bulk = bytes & ~15;
    for (int i = bulk / 4 + (int)threadIdx.x; i < bytes / 4; i += blockDim.x)
        static_cast<uint32_t *>(dst)[i] = static_cast<const uint32_t *>(stage)[i];
    if (threadIdx.x == 0 && bulk) {
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                     "r"((uint32_t)__cvta_generic_to_shared(stage)), "r"(bulk)
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    __syncthreads();
}

// One warp's blocks t of its 32 elements (n of them valid), 9 doubles per lane
// at stage + 9 * lane, to global memory as one bulk copy.  Two stages per warp:
// `turn` counts the copies issued, and the stage about to be written was last
// read by the copy before the previous one.
struct WarpStore {
    double *stages;  // two of kStage doubles each, 16-byte aligned
    int turn = 0;
    static constexpr int kStage = 32 * 12;

    __device__ __forceinline__ double *next() {
        if ((threadIdx.x & 31) == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        __syncwarp();
        return stages + (turn & 1) * kStage;
    }
    // `per` doubles per lane are in the stage
    __device__ __forceinline__ void store(double *dst, int n, int per) {
        const double *stage = stages + (turn & 1) * kStage;
        ++turn;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        const int bytes = n * per * 8, bulk = bytes & ~15;
        if ((threadIdx.x & 31) == 0) {
            if (bulk)
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                             "r"((uint32_t)__cvta_generic_to_shared(stage)), "r"(bulk)
                             : "memory");
            if (bulk < bytes) dst[bulk / 8] = stage[bulk / 8];
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    }
    __device__ __forceinline__ void finish() {
        if ((threadIdx.x & 31) == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
};

}  // namespace skg
