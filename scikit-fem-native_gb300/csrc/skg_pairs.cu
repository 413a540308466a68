// Builds the pair plan of a pattern (see skg_pairs.cuh) and holds the sums of
// plans with three components per node.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "skg_common.cuh"
#include "skg_fp64.cuh"
#include "skg_pairs.cuh"

namespace skg {

// Nine threads per pair; a contribution is 72 contiguous bytes, so that the
// nine loads of a pair share its sectors.  Bound by the FP64 pipe (three
// quarters busy; an addition costs the same for a partly filled warp), the
// reads and issue together: additions are fused multiply-adds, the orientation
// is the top bit of the code, and the contributions come in whole batches (one
// slice per block: its count is the same for every thread).  Vector P1 48^3:
// 158 -> 139 us; batches of 2 or 8 instead of 4: 154, 142; predicated batches of
// 4, 8, 12: 149, 173, 242; codes staged in shared memory: no faster.
__global__ void __launch_bounds__(kPairBlock3) k_pair_sum3(int s0, PairArrays p, const double *__restrict__ K,
                                                           double *__restrict__ values) {
    const double one = Fp64::unit();
    const int s = s0 + blockIdx.x;
    const int l = threadIdx.x / 9, en = threadIdx.x - l * 9, i = en / 3, k = en - i * 3;
    const int32_t k0 = p.slice_ptr[s], n = p.slice_ptr[s + 1] - k0;
    const uint4 to = p.slots3[(int64_t)s * 32 + l];
    const uint32_t *cs = p.codes + (int64_t)k0 * 32 + l;
    const double *at = K + en, *turned = K + k * 3 + i;
    double sum = -0.0;
    // the next N contributions, the first of all without an addition: whole
    // batches, so that no instruction is issued for nothing
    const auto batch = [&](auto count, bool first) {
        constexpr int N = decltype(count)::value;
        uint32_t c[N];
        double v[N];
#pragma unroll
        for (int j = 0; j < N; ++j) c[j] = __ldg(cs + 32 * j);
#pragma unroll
        for (int j = 0; j < N; ++j)  // -0.0 leaves any sum unchanged
            v[j] = c[j] != kPairNone ? __ldg((c[j] & kPairTurned ? turned : at) + (uint64_t)(c[j] & ~kPairTurned) * 9)
                                     : -0.0;
        sum = first ? v[0] : fma(sum, one, v[0]);
#pragma unroll
        for (int j = 1; j < N; ++j) sum = fma(sum, one, v[j]);
        cs += 32 * N;
    };
    switch (n & 3) {
        case 1: batch(std::integral_constant<int, 1>{}, true); break;
        case 2: batch(std::integral_constant<int, 2>{}, true); break;
        case 3: batch(std::integral_constant<int, 3>{}, true); break;
        default:
            if (n) batch(std::integral_constant<int, 4>{}, true);
    }
    for (int f = (n - 1) >> 2; f > 0; --f) batch(std::integral_constant<int, 4>{}, false);
    if (to.x == kPairNone) return;
    values[to.x + i * to.y + k] = sum;
    if (to.z != kPairNone) values[to.z + k * to.w + i] = sum;
}

namespace {

// Full matrices (E, n, n) from packed upper triangles: patterns without a plan.
__global__ void k_expand_packed(int64_t ne, int64_t stride, int n, const double *__restrict__ K,
                                double *__restrict__ full) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ne * n * n) return;
    const int64_t e = i / (n * n);
    const int q = (int)(i - e * n * n), a = q / n, b = q - a * n;
    full[i] = K[(a <= b ? tri_index(n, a, b) : tri_index(n, b, a)) * stride + e];
}

// Full element matrices (E, 3n, 3n) from packed blocks, likewise.
__global__ void k_expand_blocks(int64_t ne, int64_t stride, int n, const double *__restrict__ K,
                                double *__restrict__ full) {
    const int L = 3 * n;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ne * L * L) return;
    const int64_t e = i / (L * L);
    const int q = (int)(i - e * L * L), r = q / L, c = q - r * L, a = r / 3, b = c / 3, x = r % 3, y = c % 3;
    const int64_t t = a <= b ? tri_index(n, a, b) : tri_index(n, b, a);
    full[i] = K[(t * stride + e) * 9 + (a <= b ? x * 3 + y : y * 3 + x)];
}

// Node-level view of a pattern, by kind of plan.  1: DOFs of a symmetric
// pattern; 3: nodes of three components; 2: the DOFs of four nodes of three
// components that are not numbered node by node, whose pairs are entries of
// the nodes' packed blocks; 0: DOFs of a pattern whose element matrices are summed
// whole.
template <int K>
struct NodeView {
    static constexpr int C = K == 3 ? 3 : 1;
    const int32_t *cols, *indptr, *indices, *inc_ptr, *inc;
    int32_t L, Lc, n;  // local rows, local columns, local column nodes
    __device__ int32_t node(int64_t e, int b) const { return cols[e * Lc + C * b] / C; }
    __device__ int32_t begin(int32_t r) const { return indptr[C * r]; }
    __device__ int32_t length(int32_t r) const { return indptr[C * r + 1] - indptr[C * r]; }  // DOF columns
    __device__ int32_t col(int32_t rb, int p) const { return indices[rb + C * p] / C; }
    // position of node c in row r (its columns are sorted)
    __device__ int32_t position(int32_t r, int32_t c) const {
        const int32_t rb = begin(r);
        int lo = 0, hi = length(r) / C;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (col(rb, mid) < c) lo = mid + 1; else hi = mid;
        }
        return lo;
    }
};

__global__ void k_block_check(int64_t total, const int32_t *__restrict__ dofs, int32_t *bad) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t first = dofs[i / 3 * 3];
        if (first % 3 != 0 || dofs[i] != first + (int32_t)(i % 3)) *bad = 1;
    }
}

template <int K>
__global__ void k_upper_count(NodeView<K> v, int32_t rows, int32_t *__restrict__ n_upper) {
    const int32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    n_upper[r] = v.length(r) / v.C - (K == 0 ? 0 : v.position(r, r));
}

template <int K>
__global__ void k_pair_rows(NodeView<K> v, int32_t rows, const int32_t *__restrict__ pair_ptr,
                            int32_t *__restrict__ pair_row) {
    const int32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    for (int32_t j = pair_ptr[r]; j < pair_ptr[r + 1]; ++j) pair_row[j] = r;
}

// Calls f(element, a, b) for every contribution of pair (r, c), in the order
// of row r's incidences (ascending elements).
template <int K, class F>
__device__ __forceinline__ void each_contribution(const NodeView<K> &v, int32_t r, int32_t c, F &&f) {
    constexpr int C = NodeView<K>::C;
    for (int32_t it = v.inc_ptr[C * r]; it < v.inc_ptr[C * r + 1]; ++it) {
        const int32_t item = v.inc[it];
        const int32_t e = item / v.L;
        const int a = (item - e * v.L) / C;
        for (int b = 0; b < v.n; ++b)
            if (v.node(e, b) == c) f(e, a, b);
    }
}

template <int K>
__device__ __forceinline__ int32_t pair_column(const NodeView<K> &v, int32_t r, int32_t j, const int32_t *pair_ptr) {
    // the pairs of row r are the last columns of the row
    return v.col(v.begin(r), v.length(r) / v.C - (pair_ptr[r + 1] - j));
}

// Contributions of every pair; per window, the last element (+ 1) it needs.
template <int K>
__global__ void __launch_bounds__(256) k_pair_count(NodeView<K> v, int32_t n_pairs,
                                                    const int32_t *__restrict__ pair_ptr,
                                                    const int32_t *__restrict__ pair_row, int32_t *__restrict__ count,
                                                    int32_t *__restrict__ ready) {
    static_assert(kPairWindow % 256 == 0, "a block lies in one window");
    const int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x;
    int32_t n = 0, last = 0;
    if (j < n_pairs) {
        const int32_t r = pair_row[j], c = pair_column(v, r, (int32_t)j, pair_ptr);
        each_contribution(v, r, c, [&](int32_t e, int, int) {
            ++n;
            last = e + 1;
        });
        count[j] = n;
    }
    last = __reduce_max_sync(0xffffffffu, last);
    if ((threadIdx.x & 31) == 0) atomicMax(ready + j / kPairWindow, last);
}

// One block per window: stable counting sort by min(count, 31), then each
// slice's width (its largest count).  Block b writes window windows[b] at b.
__global__ void __launch_bounds__(kPairWindow) k_window_sort(int32_t n_pairs, const int32_t *__restrict__ windows,
                                                             const int32_t *__restrict__ count,
                                                             int32_t *__restrict__ order,
                                                             int32_t *__restrict__ width) {
    __shared__ int32_t hist[32 * 32], base[32], sorted[kPairWindow];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int64_t j = (int64_t)windows[blockIdx.x] * kPairWindow + t;
    const int32_t n = j < n_pairs ? count[j] : 0;
    const int bin = j < n_pairs ? min(n, 31) : 31;  // threads past the end sort last
    hist[t] = 0;
    __syncthreads();
    const unsigned same = __match_any_sync(0xffffffffu, bin);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (rank == 0) hist[bin * 32 + warp] = __popc(same);
    __syncthreads();
    // exclusive scan over (bin, warp)
    const int32_t h = hist[t];
    int32_t x = h;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) base[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int32_t b = base[lane];
        const int32_t own = b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) b += y;
        }
        base[lane] = b - own;
    }
    __syncthreads();
    hist[t] = base[warp] + x - h;
    __syncthreads();
    const int pos = hist[bin * 32 + warp] + rank;
    sorted[pos] = n;
    order[(int64_t)blockIdx.x * kPairWindow + pos] = j < n_pairs ? (int32_t)j : -1;
    __syncthreads();
    const int32_t w = __reduce_max_sync(0xffffffffu, sorted[t]);
    if (lane == 0) width[(int64_t)blockIdx.x * 32 + warp] = w;
}

// First rows of the host-output chunks, of about equal slot counts.
template <int K>
__global__ void k_copy_rows(NodeView<K> v, int32_t rows, int64_t nnz, int n_chunks, int32_t *__restrict__ first,
                            int32_t *__restrict__ slot) {
    const int k = threadIdx.x;
    if (k > n_chunks) return;
    const int64_t target = nnz * k / n_chunks;
    int lo = 0, hi = rows;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (v.begin(mid) < target) lo = mid + 1; else hi = mid;
    }
    first[k] = k == n_chunks ? rows : lo;
    slot[k] = v.indptr[v.C * first[k]];
}

__device__ __forceinline__ int chunk_of(const int32_t *first, int n_chunks, int32_t row) {
    int k = 0;
    while (k + 1 < n_chunks && first[k + 1] <= row) ++k;
    return k;
}

// Codes, orientations and targets of every slice lane; one block per window.
// done[k]: windows after which host-output chunk k is complete.
template <int K>
__global__ void __launch_bounds__(kPairWindow) k_pair_fill(NodeView<K> v, const int32_t *__restrict__ pair_ptr,
                                                           const int32_t *__restrict__ pair_row,
                                                           const int32_t *__restrict__ order,
                                                           const int32_t *__restrict__ slice_ptr, int np, int64_t stride,
                                                           uint32_t *__restrict__ codes,
                                                           uint32_t *__restrict__ orient, uint2 *__restrict__ slots,
                                                           uint4 *__restrict__ slots3, int n_chunks,
                                                           const int32_t *__restrict__ first,
                                                           int32_t *__restrict__ done) {
    constexpr int C = NodeView<K>::C;
    __shared__ unsigned touched;
    if (threadIdx.x == 0) touched = 0;
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * kPairWindow + threadIdx.x;
    const int32_t j = order[i], lane = (int32_t)(i & 31), s = (int32_t)(i >> 5);
    const int32_t k1 = slice_ptr[s + 1];
    int32_t k = slice_ptr[s];
    unsigned mask = 0;
    uint2 to = make_uint2(kPairNone, kPairNone), len = make_uint2(0, 0);
    if (j >= 0) {
        const int32_t r = pair_row[j], c = pair_column(v, r, j, pair_ptr);
        each_contribution(v, r, c, [&](int32_t e, int a, int b) {
            if (K == 2) {  // entry (x, y) of block (na, nb), or (y, x) of block (nb, na)
                const int na = a / 3, nb = b / 3, x = a - 3 * na, y = b - 3 * nb;
                const uint32_t t = (uint32_t)tri_index(4, min(na, nb), max(na, nb));
                codes[(int64_t)k * 32 + lane] =
                    (t * (uint32_t)stride + (uint32_t)e) * 9u + (uint32_t)(na <= nb ? 3 * x + y : 3 * y + x);
                ++k;
                return;
            }
            const uint32_t t = (uint32_t)(K == 0 ? a * v.n + b : tri_index(v.n, min(a, b), max(a, b)));
            codes[(int64_t)k * 32 + lane] =
                K == 0 ? (uint32_t)e * (uint32_t)np + t
                       : (t * (uint32_t)stride + (uint32_t)e) | (K == 3 && a > b ? kPairTurned : 0u);
            if (K == 1 && a > b) atomicOr(orient + k, 1u << lane);
            ++k;
        });
        to.x = (uint32_t)(v.begin(r) + v.length(r) - C * (pair_ptr[r + 1] - j));
        len.x = (uint32_t)v.length(r);
        if (K != 0 && r != c) {
            to.y = (uint32_t)(v.begin(c) + C * v.position(c, r));
            len.y = (uint32_t)v.length(c);
        }
        if (n_chunks) mask = 1u << chunk_of(first, n_chunks, r) | 1u << chunk_of(first, n_chunks, c);
    }
    for (; k < k1; ++k) codes[(int64_t)k * 32 + lane] = kPairNone;
    if (C == 1) slots[i] = to;
    else slots3[i] = make_uint4(to.x, len.x, to.y, len.y);
    if (!n_chunks) return;
    mask = __reduce_or_sync(0xffffffffu, mask);
    if (lane == 0 && mask) atomicOr(&touched, mask);
    __syncthreads();
    if (threadIdx.x < n_chunks && (touched >> threadIdx.x & 1u)) atomicMax(done + threadIdx.x, (int)blockIdx.x + 1);
}

template <class T>
void download(std::vector<T> &h, const T *d, size_t n, cudaStream_t s) {
    h.resize(n);
    SKG_CUDA(cudaMemcpyAsync(h.data(), d, n * sizeof(T), cudaMemcpyDeviceToHost, s));
    SKG_CUDA(cudaStreamSynchronize(s));
}

template <int K>
PairPlan build(const skg_pattern *p, cudaStream_t s) {
    constexpr int C = NodeView<K>::C;
    const NodeView<K> v{p->col_dofs.get(), p->indptr.get(), p->indices.get(), p->inc_ptr.get(),
                        p->inc.get(),      p->row_local,    p->col_local,     p->col_local / C};
    const int32_t rows = (int32_t)(p->n_rows / C);
    PairPlan plan;
    plan.nodes = v.n;
    plan.np = K == 0 ? p->row_local * p->col_local : v.n * (v.n + 1) / 2;
    DevBuf<int32_t> n_upper(rows + 1, s), pair_ptr(rows + 1, s);
    k_upper_count<K><<<grid_for(rows, 256), 256, 0, s>>>(v, rows, n_upper.get());
    SKG_LAUNCH_CHECK("upper_count");
    exclusive_scan_i32(n_upper.get(), pair_ptr.get(), rows, s);
    std::vector<int32_t> h;
    download(h, pair_ptr.get() + rows, 1, s);
    const int32_t n_pairs = h[0];
    if (n_pairs <= 0) return PairPlan{};
    const int32_t n_windows = (n_pairs - 1) / kPairWindow + 1;
    const int64_t n_lanes = (int64_t)n_windows * kPairWindow;
    plan.n_slices = (int32_t)(n_lanes / 32);
    DevBuf<int32_t> pair_row(n_pairs, s), count(n_pairs, s), ready(n_windows, s), windows(n_windows, s);
    DevBuf<int32_t> order(n_lanes, s), width(plan.n_slices + 1, s);
    SKG_CUDA(cudaMemsetAsync(ready.get(), 0, (size_t)n_windows * 4, s));
    k_pair_rows<K><<<grid_for(rows, 256), 256, 0, s>>>(v, rows, pair_ptr.get(), pair_row.get());
    SKG_LAUNCH_CHECK("pair_rows");
    k_pair_count<K><<<grid_for(n_pairs, 256), 256, 0, s>>>(v, n_pairs, pair_ptr.get(), pair_row.get(), count.get(),
                                                          ready.get());
    SKG_LAUNCH_CHECK("pair_count");
    // windows by the elements they need
    std::vector<int32_t> need, by(n_windows);
    if (n_windows > 1) {
        download(need, ready.get(), n_windows, s);
        for (int32_t i = 0; i < n_windows; ++i) by[i] = i;
        std::stable_sort(by.begin(), by.end(), [&](int32_t a, int32_t b) { return need[a] < need[b]; });
        SKG_CUDA(cudaMemcpyAsync(windows.get(), by.data(), (size_t)n_windows * 4, cudaMemcpyHostToDevice, s));
    } else {
        SKG_CUDA(cudaMemsetAsync(windows.get(), 0, 4, s));
    }
    k_window_sort<<<n_windows, kPairWindow, 0, s>>>(n_pairs, windows.get(), count.get(), order.get(), width.get());
    SKG_LAUNCH_CHECK("window_sort");
    DevBuf<int32_t> slice_ptr(plan.n_slices + 1, s);
    exclusive_scan_i32(width.get(), slice_ptr.get(), plan.n_slices, s);
    download(h, slice_ptr.get() + plan.n_slices, 1, s);
    const int32_t total = h[0];
    const size_t ptr_bytes = ((size_t)plan.n_slices + 1) * 4, orient_bytes = K == 1 ? (size_t)total * 4 : 0;
    const size_t slot_bytes = (size_t)n_lanes * (C == 1 ? sizeof(uint2) : sizeof(uint4));
    const size_t code_bytes = (size_t)total * 32 * 4;
    plan.store = DevBuf<unsigned char>::owned(slot_bytes + code_bytes + orient_bytes + ptr_bytes);
    unsigned char *at = plan.store.get();
    plan.slots = C == 1 ? reinterpret_cast<uint2 *>(at) : nullptr;
    plan.slots3 = C == 1 ? nullptr : reinterpret_cast<uint4 *>(at);
    plan.codes = reinterpret_cast<uint32_t *>(at += slot_bytes);
    plan.orient = reinterpret_cast<uint32_t *>(at += code_bytes);
    plan.slice_ptr = reinterpret_cast<int32_t *>(at += orient_bytes);
    SKG_CUDA(cudaMemcpyAsync(plan.slice_ptr, slice_ptr.get(), ptr_bytes, cudaMemcpyDeviceToDevice, s));
    if (orient_bytes) SKG_CUDA(cudaMemsetAsync(plan.orient, 0, orient_bytes, s));
    const int n_chunks = K != 0 && p->nnz >= kHostChunkMinNnz ? kHostChunks : 0;
    DevBuf<int32_t> chunk(3 * (kHostChunks + 1), s);  // first rows, first slots, windows done
    int32_t *first = chunk.get(), *slot = first + kHostChunks + 1, *done = slot + kHostChunks + 1;
    if (n_chunks) {
        SKG_CUDA(cudaMemsetAsync(chunk.get(), 0, 3 * (kHostChunks + 1) * 4, s));
        k_copy_rows<K><<<1, 32, 0, s>>>(v, rows, p->nnz, n_chunks, first, slot);
        SKG_LAUNCH_CHECK("copy_rows");
    }
    k_pair_fill<K><<<n_windows, kPairWindow, 0, s>>>(v, pair_ptr.get(), pair_row.get(), order.get(),
                                                    plan.slice_ptr, plan.np, block_stride(p->n_elements), plan.codes,
                                                    plan.orient, plan.slots, plan.slots3, n_chunks, first, done);
    SKG_LAUNCH_CHECK("pair_fill");
    if (n_chunks) {
        download(h, chunk.get(), 3 * (kHostChunks + 1), s);
        for (int k = 0; k < n_chunks; ++k) {
            PairCopy c;
            c.slot0 = h[kHostChunks + 1 + k];
            c.slot1 = k + 1 < n_chunks ? h[kHostChunks + 2 + k] : (int32_t)p->nnz;
            c.slice = h[2 * (kHostChunks + 1) + k] * (kPairWindow / 32);
            plan.copies.push_back(c);
        }
        std::stable_sort(plan.copies.begin(), plan.copies.end(),
                         [](const PairCopy &a, const PairCopy &b) { return a.slice < b.slice; });
        // one step per copy (of at least E / 96 elements): the first copy starts
        // as soon as its own elements and windows are done
        for (const PairCopy &c : plan.copies) {
            if (c.slice == 0) continue;
            const PairStep st{c.slice, need[by[c.slice / (kPairWindow / 32) - 1]]};
            if (!plan.steps.empty() && st.ready - plan.steps.back().ready < p->n_elements / 96) plan.steps.pop_back();
            plan.steps.push_back(st);
        }
        if (plan.steps.empty() || plan.steps.back().slice < plan.n_slices)
            plan.steps.push_back(PairStep{plan.n_slices, p->n_elements});
    }
    plan.block = C;
    return plan;
}

}  // namespace

void expand_packed(int64_t ne, int n, const double *K, double *full, cudaStream_t s) {
    if (ne == 0) return;
    k_expand_packed<<<grid_for(ne * n * n, 256), 256, 0, s>>>(ne, block_stride(ne), n, K, full);
    SKG_LAUNCH_CHECK("expand_packed");
}

void expand_blocks(int64_t ne, int n, const double *K, double *full, cudaStream_t s) {
    if (ne == 0) return;
    k_expand_blocks<<<grid_for(ne * 9 * n * n, 256), 256, 0, s>>>(ne, block_stride(ne), n, K, full);
    SKG_LAUNCH_CHECK("expand_blocks");
}

// Plans of a pattern: the pair plan when its row and column DOFs are the same
// (`square`) and its shape is one that is assembled symmetric (four nodes of
// three components in any numbering, by entries where it is not node by node);
// the whole sums for the shapes that no row group serves.  None when the positions exceed
// 32 bits (the assemblies then walk the rows).
void build_pair_plan(skg_pattern *p, bool square, cudaStream_t s) {
    if (p->n_rows == 0 || p->n_elements == 0) return;
    const int L = p->row_local, C = L == 12 || L == 30 ? 3 : 1;
    const int64_t n = L / C, total = p->n_elements * L;
    if (square && (C == 3 ? p->n_rows % 3 == 0 : L == 4 || L == 6 || L == 10) &&
        block_stride(p->n_elements) * (n * (n + 1) / 2) < (int64_t)(C == 3 ? kPairTurned - 1 : kPairNone)) {
        if (C == 1) {
            p->pairs = build<1>(p, s);
            return;
        }
        DevBuf<int32_t> bad(1, s);
        SKG_CUDA(cudaMemsetAsync(bad.get(), 0, 4, s));
        k_block_check<<<grid_for(total, 256), 256, 0, s>>>(total, p->row_dofs.get(), bad.get());
        SKG_LAUNCH_CHECK("block_check");
        std::vector<int32_t> h;
        download(h, bad.get(), 1, s);
        if (h[0] == 0) {
            p->pairs = build<3>(p, s);
            return;
        }
        if (L == 12 && block_stride(p->n_elements) * 90 < (int64_t)kPairNone) p->pairs = build<2>(p, s);
    }
    const bool grouped = p->max_row_len > 0 && L == p->col_local && (L == 4 || L == 6 || L == 10 || L == 12);
    if (!grouped && p->n_elements * L * (int64_t)p->col_local < (int64_t)kPairNone) p->whole = build<0>(p, s);
}

}  // namespace skg
