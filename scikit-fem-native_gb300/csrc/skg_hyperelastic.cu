// Neo-Hookean residual and tangent on vector P1 tetrahedra.
//
// The reference keeps the law as scikit-fem forms
// (benchmarks/skfem_neo_hookean.py:8-52):
//   P = mu (F - F^-T) + lambda ln J F^-T,
//   A_iJkL = mu d_ik d_JL + (mu - lambda ln J) F^-T_iL F^-T_kJ + lambda F^-T_iJ F^-T_kL,
// assembled with NativeLinearForm (residual, linear_form_assembler.cpp:41-154)
// and NativeCrossBilinearForm.assemble_tensor (tangent,
// cross_bilinear_assembler.cpp:207-247).  For P1, F = I + grad u is constant
// on an element, so with g_a = grad lambda_a, h_a = F^-T g_a and the element
// measure V = |det J| * (sum of the rule's weights):
//   r_(a,c)          = V sum_j P_cj g_a,j
//   K_(a,i),(b,k)    = V [ mu d_ik (g_a . g_b) + (mu - lambda ln J) h_b,i h_a,k
//                          + lambda h_a,i h_b,k ]
// (the contraction of A with g_a and g_b written out).
//
// Plain law: one thread per element writes the packed blocks of the tangent
// and the residual entries (k_nh_packed); the pair sums (skg_pairs.cuh) and a
// gather per DOF add them in element order.  The results are bitwise
// reproducible (no atomics).
//
// The surrogate entry point replaces the law by a small MLP on the
// invariants (see skg_mlp.cu) with a per-element fallback to this law.
#include "skg_common.cuh"
#include "skg_df64.cuh"
#include "skg_fp64.cuh"
#include "skg_nh.cuh"
#include "skg_pairs.cuh"

namespace skg {

void gather_element_matrices(const skg_pattern *pat, const double *Ke, double *values, cudaStream_t s);

namespace {

constexpr int kNhBlock = 64;

// Element tangent (packed 3 x 3 blocks of the node pairs a <= b, see
// skg_pairs.cuh) and residual (E, 12) of the plain law, thread per element.
//
// The kernel is bound by the FP64 pipe, so the law is evaluated in a form with
// few FP64 instructions that keeps the stress of small strains:
// * h_a = F^-T grad lambda_a is the gradient of lambda_a on the displaced
//   tetrahedron (edges j_k = e_k + d_k, d_k = u_k - u_0): its cofactors over its
//   determinant, without F, its inverse or the products with it.
// * det F - 1 is made of terms with one displacement difference each, exchanging
//   one edge at a time: (d_1 . j_2 x j_3 + d_2 . j_3 x e_1 + d_3 . e_1 x e_2) / det,
//   and ln J = log1p of it (of the determinants' ratio itself where it is far
//   from 1).
// * With H = grad u = sum_k d_k g_k^T: F g_a = g_a + H g_a and g_a - h_a = H^T h_a
//   (g_a = F^T h_a), so the residual is r_a = V P g_a = mu V (H g_a + H^T h_a) +
//   lambda ln J V h_a = sum_k (d_k G_ka + mu V g_k (d_k . h_a)) + lambda ln J V h_a
//   with G_ab = mu V g_a . g_b; r_0 from the zero sum.  Every term carries a
//   displacement difference: the residual is zero without displacement, and its
//   error is relative to the strain (formed as F - F^-T, or from the displaced
//   edges whole, it is a difference of numbers of size one: at strain 1e-6 on
//   elements of aspect ratio 1000 4e-9 or 2e-6 of the largest entry instead of
//   4e-11, and 1e-11 instead of zero at the undeformed state; the worst of 200
//   random tetrahedra).  426 FP64 instructions, 1105 us at 64^3 (94 % of the pipe's
//   rate); by the displaced edges whole 352 and 921 us, by the stress and tangent
//   tensors 535 and 1543 us.
// * With p_a = (mu - lambda ln J) V h_a, q_a = lambda V h_a, t_a = p_a + q_a
//   the entries are p_a,k h_b,i + q_a,i h_b,k (i != k), t_a,i h_b,i + G_ab
//   (i = k), and t_a,k h_a,i in the diagonal blocks (symmetric).
// Ke or re may be NULL (that output is skipped).
__global__ void __launch_bounds__(kNhBlock, 8) k_nh_packed(int64_t ne, int64_t e_begin, int64_t e_end, int64_t stride,
                                                       const double *__restrict__ p, int64_t npts,
                                                       const int32_t *__restrict__ t, const int32_t *__restrict__ dofs,
                                                       const double *__restrict__ u, double mu, double lmbda,
                                                       double wsum, double *__restrict__ Ke, double *__restrict__ re) {
    __shared__ __align__(16) double stages[kNhBlock / 32 * 2 * WarpStore::kStage];
    const int lane = threadIdx.x & 31;
    const int64_t e0 = e_begin + (int64_t)blockIdx.x * kNhBlock + (threadIdx.x & ~31);
    const int n = (int)(e_end - e0 < 32 ? e_end - e0 : 32);
    if (n <= 0) return;
    const int64_t e = lane < n ? e0 + lane : e0;  // the lanes past the end repeat the first element, unwritten
    const Fp64 F = Fp64::load();
    WarpStore out{stages + (threadIdx.x >> 5) * 2 * WarpStore::kStage};
    int32_t v[4];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = t[k * ne + e];
        ok = ok && v[k] >= 0 && v[k] < npts;
    }
    if (!ok) v[0] = v[1] = v[2] = v[3] = 0;
    double d[9];              // [coordinate * 3 + edge]: displacement differences
    double c[4][3], h[4][3];  // rows 1..3 of the adjugates: the determinant times grad lambda_k
    double det, detj, grown;  // grown: det (det F - 1)
    {
        double J[9], j[9];  // edges of the element, and displaced
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double x0 = p[i * npts + v[0]], u0 = u[dofs[e * 12 + i]];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                J[i * 3 + k] = F.sub(p[i * npts + v[k + 1]], x0);
                d[i * 3 + k] = F.sub(u[dofs[e * 12 + 3 * (k + 1) + i]], u0);
                j[i * 3 + k] = F.add(J[i * 3 + k], d[i * 3 + k]);
            }
        }
        det = F.adjugate(J, c);
        detj = F.adjugate(j, h);
        // row 2 of the adjugate with the first edge as it was and the third displaced
        const double m[3] = {F.cross(j[5], J[6], J[3], j[8]), F.cross(J[0], j[8], j[2], J[6]),
                             F.cross(j[2], J[3], J[0], j[5])};
        grown = F.mul(d[0], h[1][0]);
        grown = fma(d[3], h[1][1], grown);
        grown = fma(d[6], h[1][2], grown);
#pragma unroll
        for (int i = 0; i < 3; ++i) grown = fma(d[i * 3 + 2], c[3][i], fma(d[i * 3 + 1], m[i], grown));
    }
    const double id = ok ? 1.0 / det : __longlong_as_double(0x7ff8000000000000LL);
    const double idj = 1.0 / detj;
    const double rise = grown * id;
    // far from 1 the ratio of the determinants has the smaller relative error
    const double lnJ = fabs(rise) < 0.5 ? log1p(rise) : log(detj * id);
    const double V = fabs(det) * wsum;
    const double c2V = (mu - lmbda * lnJ) * V, lamV = lmbda * V, tV = c2V + lamV;
    double G[4][4];
    const double gs = mu * V * id * id;
#pragma unroll
    for (int a = 1; a < 4; ++a)
#pragma unroll
        for (int b = a; b < 4; ++b) {
            G[a][b] = F.mul(gs, F.dot(c[a], c[b]));
            G[b][a] = G[a][b];
        }
#pragma unroll
    for (int b = 1; b < 4; ++b) G[0][b] = -F.add3(G[1][b], G[2][b], G[3][b]);
    G[0][0] = -F.add3(G[0][1], G[0][2], G[0][3]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int a = 1; a < 4; ++a) h[a][i] = F.mul(h[a][i], idj);
        h[0][i] = -F.add3(h[1][i], h[2][i], h[3][i]);
    }
    if (re) {
        double *st = out.next() + 12 * lane;
        const double gV = mu * V * id, lnV = lmbda * lnJ * V;
        double sum[3];
#pragma unroll
        for (int a = 1; a < 4; ++a) {
            double r[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) r[i] = F.mul(lnV, h[a][i]);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                // d_k . h_a
                const double dh = F.mul(gV, fma(d[6 + k], h[a][2], fma(d[3 + k], h[a][1], F.mul(d[k], h[a][0]))));
#pragma unroll
                for (int i = 0; i < 3; ++i) r[i] = fma(d[i * 3 + k], G[k + 1][a], fma(c[k + 1][i], dh, r[i]));
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                st[a * 3 + i] = r[i];
                sum[i] = a == 1 ? r[i] : F.add(sum[i], r[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) st[i] = -sum[i];
        out.store(re + e0 * 12, n, 12);
    }
    if (Ke) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            double pa[3], qa[3], ta[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                pa[i] = F.mul(c2V, h[a][i]);
                qa[i] = F.mul(lamV, h[a][i]);
                ta[i] = F.mul(tV, h[a][i]);
            }
#pragma unroll
            for (int b = a; b < 4; ++b) {
                double *st = out.next() + 9 * lane;
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        if (i == k) {
                            st[i * 3 + k] = fma(ta[i], h[b][i], G[a][b]);
                        } else if (b > a) {
                            st[i * 3 + k] = fma(pa[k], h[b][i], F.mul(qa[i], h[b][k]));
                        } else if (k > i) {
                            const double x = F.mul(ta[k], h[a][i]);
                            st[i * 3 + k] = x;
                            st[k * 3 + i] = x;
                        }
                    }
                out.store(Ke + (tri_index(4, a, b) * stride + e0) * 9, n, 9);
            }
        }
    }
    out.finish();
}

// Residual gather: thread per DOF over its incidence list (element order).
__global__ void k_vector_gather(int64_t n_rows, const int32_t *__restrict__ inc_ptr, const int32_t *__restrict__ inc,
                                const double *__restrict__ re, double *__restrict__ out) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    double acc = 0.0;
    for (int32_t it = inc_ptr[r]; it < inc_ptr[r + 1]; ++it) acc += re[inc[it]];
    out[r] = acc;
}

// ----------------------------------------------------- sums of the learned law

// Value of a sum of FP32 entries in double-float, converted by integer
// arithmetic (no FP64 pipe) unless it is subnormal, infinite or not a number.
__device__ __forceinline__ double closure_value(df64 v) {
    const unsigned ex = (__float_as_uint(v.hi) >> 23) & 0xffu;
    if (ex == 0xffu) return (double)v.hi;
    v = fast_two_sum(v.hi, v.lo);
    const unsigned b = __float_as_uint(v.hi);
    if ((b & 0x7f800000u) == 0 && (b & 0x7fffffu) != 0) return (double)v.hi + (double)v.lo;
    return df_to_double(v, 0);
}

// Pair sums of the learned law's tangent: packed FP32 blocks, summed in
// double-float in element order.  The elements that the plain law served
// (flags, read when the call's count `fallbacks` is set) have the low parts of
// their FP64 entries at the same positions of `low`.  Bound by the blocks'
// reads and the values' writes; nine threads per pair as in k_pair_sum3.  The
// two cases are walked apart: with the flags' test between them the loads of a
// batch wait for one another (48^3: 144 and 174 us, 116 apart).
__global__ void __launch_bounds__(kPairBlock3) k_closure_sum3(int s0, PairArrays p, const float *__restrict__ K,
                                                              const float *__restrict__ low,
                                                              const unsigned char *__restrict__ flags, uint32_t stride,
                                                              const unsigned long long *__restrict__ fallbacks,
                                                              double *__restrict__ values) {
    const int s = s0 + blockIdx.x;
    const int l = threadIdx.x / 9, en = threadIdx.x - l * 9, i = en / 3, k = en - i * 3;
    const int turned = k * 3 + i;
    const int32_t k0 = p.slice_ptr[s], n = p.slice_ptr[s + 1] - k0;
    const uint4 to = p.slots3[(int64_t)s * 32 + l];
    const uint32_t *cs = p.codes + (int64_t)k0 * 32 + l;
    df64 sum = pair_zero<df64>();
    const auto batch = [&](auto count, auto any) {
        constexpr int N = decltype(count)::value;
        uint32_t c[N];
        df64 v[N];
#pragma unroll
        for (int j = 0; j < N; ++j) c[j] = __ldg(cs + 32 * j);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            v[j] = pair_zero<df64>();
            const int64_t pos = (int64_t)(c[j] & ~kPairTurned) * 9 + (c[j] & kPairTurned ? turned : en);
            if (c[j] != kPairNone) v[j].hi = __ldg(K + pos);
            if (decltype(any)::value && c[j] != kPairNone && flags[(c[j] & ~kPairTurned) % stride])
                v[j].lo = __ldg(low + pos);
        }
#pragma unroll
        for (int j = 0; j < N; ++j) pair_add(sum, v[j]);
        cs += 32 * N;
    };
    const auto walk = [&](auto any) {
        for (int f = n >> 2; f > 0; --f) batch(std::integral_constant<int, 4>{}, any);
        if (n & 2) batch(std::integral_constant<int, 2>{}, any);
        if (n & 1) batch(std::integral_constant<int, 1>{}, any);
    };
    if (*fallbacks == 0) walk(std::false_type{});
    else walk(std::true_type{});
    if (to.x == kPairNone) return;
    const double r = closure_value(sum);
    values[to.x + i * to.y + k] = r;
    if (to.z != kPairNone) values[to.z + k * to.w + i] = r;
}

// The same sums by pairs of DOFs that are not numbered node by node (see
// has_block_plan): one lane per pair, `s1` past the last slice.  Learned law at 48^3
// with such a numbering, the whole call: 0.68 ms (3.66 with full element matrices
// from the network on the CUDA cores; 0.54 numbered node by node).
__global__ void __launch_bounds__(256) k_closure_entries(int s0, int s1, PairArrays p, const float *__restrict__ K,
                                                         const float *__restrict__ low,
                                                         const unsigned char *__restrict__ flags, uint32_t stride,
                                                         const unsigned long long *__restrict__ fallbacks,
                                                         double *__restrict__ values) {
    const int s = s0 + blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (s >= s1) return;
    const bool any = *fallbacks != 0;
    const uint2 to = p.slots[(int64_t)s * 32 + lane];
    df64 sum = pair_zero<df64>();
    for (int32_t k = p.slice_ptr[s]; k < p.slice_ptr[s + 1]; ++k) {
        const uint32_t c = __ldg(p.codes + (int64_t)k * 32 + lane);
        if (c == kPairNone) continue;
        pair_add(sum, df64{__ldg(K + c), any && flags[c / 9u % stride] ? __ldg(low + c) : -0.f});
    }
    const double r = closure_value(sum);
    if (to.x != kPairNone) values[to.x] = r;
    if (to.y != kPairNone) values[to.y] = r;
}

// Residual of the learned law, likewise (element entries (E, 12)).
__global__ void k_closure_gather(int64_t n_rows, const int32_t *__restrict__ inc_ptr, const int32_t *__restrict__ inc,
                                 const float *__restrict__ re, const float *__restrict__ low,
                                 const unsigned char *__restrict__ flags,
                                 const unsigned long long *__restrict__ fallbacks, double *__restrict__ out) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    const bool any = *fallbacks != 0;
    df64 acc{0.f, 0.f};
    for (int32_t it = inc_ptr[r]; it < inc_ptr[r + 1]; ++it) {
        const int32_t q = inc[it];
        pair_add(acc, df64{re[q], any && flags[q / 12] ? low[q] : 0.f});
    }
    out[r] = closure_value(acc);
}

}  // namespace

void closure_sums(const skg_pattern *pat, int s0, int s1, const ClosureBlocks &b, double *values, cudaStream_t s) {
    if (s1 <= s0) return;
    if (pat->pairs.block == 1) {
        k_closure_entries<<<grid_for(s1 - s0, 8), 256, 0, s>>>(s0, s1, pair_arrays(pat->pairs), b.K, b.K_low, b.flags,
                                                              (uint32_t)block_stride(pat->n_elements), b.fallbacks,
                                                              values);
        SKG_LAUNCH_CHECK("closure_entries");
        return;
    }
    k_closure_sum3<<<(unsigned)(s1 - s0), kPairBlock3, 0, s>>>(s0, pair_arrays(pat->pairs), b.K, b.K_low, b.flags,
                                                               (uint32_t)block_stride(pat->n_elements), b.fallbacks,
                                                               values);
    SKG_LAUNCH_CHECK("closure_sum3");
}

void closure_residual(const skg_pattern *pat, const ClosureBlocks &b, double *residual, cudaStream_t s) {
    if (!pat->n_rows) return;
    k_closure_gather<<<grid_for(pat->n_rows, 128), 128, 0, s>>>(pat->n_rows, pat->inc_ptr.get(), pat->inc.get(), b.r,
                                                               b.r_low, b.flags, b.fallbacks, residual);
    SKG_LAUNCH_CHECK("closure_gather");
}

// Whole-array copies of the results to the host.
void nh_download(const skg_pattern *pat, const double *d_residual, const double *d_values, double *h_residual,
                 double *h_values, cudaStream_t s) {
    if (h_values && d_values && pat->nnz)
        SKG_CUDA(cudaMemcpyAsync(h_values, d_values, (size_t)pat->nnz * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (h_residual && d_residual && pat->n_rows)
        SKG_CUDA(cudaMemcpyAsync(h_residual, d_residual, (size_t)pat->n_rows * sizeof(double),
                                 cudaMemcpyDeviceToHost, s));
}

void nh_gather(const skg_pattern *pat, const double *Ke, const double *re, double *d_residual, double *d_values,
               cudaStream_t s) {
    if (d_values && Ke) gather_element_matrices(pat, Ke, d_values, s);
    if (d_residual && re && pat->n_rows) {
        k_vector_gather<<<grid_for(pat->n_rows, 128), 128, 0, s>>>(pat->n_rows, pat->inc_ptr.get(), pat->inc.get(),
                                                                  re, d_residual);
        SKG_LAUNCH_CHECK("nh_residual_gather");
    }
}

void residual_to_host(const skg_pattern *pat, const double *d_residual, double *h_residual, cudaStream_t s,
                      cudaStream_t cs) {
    if (!h_residual || !d_residual) return;
    EventSet ev;
    if (cs != s) ev.order(s, cs);
    nh_download(pat, d_residual, nullptr, h_residual, nullptr, cs);
}

}  // namespace skg

using namespace skg;

namespace skg {
namespace {

// Plain-law residual and tangent; with h_values / h_residual (page-locked
// host) the results also go there, chunk by chunk on the fused path.
void nh_assemble(const skg_pattern *pat, const double *d_p, int64_t npts, const int32_t *d_t, int64_t ne,
                 const double *d_u, double mu, double lmbda, double wsum, double *d_residual, double *d_values,
                 double *h_residual, double *h_values, cudaStream_t s) {
    require(pat != nullptr, "pattern is NULL");
    require(pat->row_local == 12 && pat->n_elements == ne, "neo-Hookean assembly needs the vector P1 pattern");
    require(!d_values || pat->col_local == 12, "tangent output needs a pattern with CSR columns");
    require(ne == 0 || (d_p && d_t && d_u), "mesh or displacement arrays are NULL");
    DevBuf<double> u_stage;
    d_u = device_resident(d_u, pat->n_rows, u_stage, s);
    const int64_t stride = block_stride(ne);
    DevBuf<double> Ke(d_values ? (size_t)stride * 90 : 0, s), re(d_residual ? (size_t)ne * 12 : 0, s);
    auto elem = [&](int64_t e0, int64_t e1) {
        k_nh_packed<<<grid_for(e1 - e0, kNhBlock), kNhBlock, 0, s>>>(ne, e0, e1, stride, d_p, npts, d_t,
                                                                    pat->row_dofs.get(), d_u, mu, lmbda, wsum,
                                                                    Ke.get(), re.get());
        SKG_LAUNCH_CHECK("nh_packed");
    };
    const auto residual = [&](cudaStream_t cs) {  // per-DOF sums, and their copy on cs
        nh_gather(pat, nullptr, re.get(), d_residual, nullptr, s);
        residual_to_host(pat, d_residual, h_residual, s, cs);
    };
    if (d_values && has_block_plan(pat, 4)) {
        run_pair_passes(
            pat, ne, d_values, h_values, s, elem,
            [&](int s0, int s1, cudaStream_t st) { block_sums(pat->pairs, s0, s1, Ke.get(), d_values, st); }, residual);
        return;
    }
    if (ne) elem(0, ne);
    if (d_values) {
        DevBuf<double> full((size_t)ne * 144, s);
        expand_blocks(ne, 4, Ke.get(), full.get(), s);
        gather_element_matrices(pat, full.get(), d_values, s);
    }
    residual(s);
    nh_download(pat, nullptr, d_values, nullptr, h_values, s);
}

}  // namespace
}  // namespace skg

extern "C" int skg_nh_assemble(const skg_pattern *pat, const double *d_p, int64_t npts, const int32_t *d_t,
                               int64_t ne, const double *d_u, double mu, double lmbda, double wsum,
                               double *d_residual, double *d_values, void *stream) {
    return guarded([&] {
        nh_assemble(pat, d_p, npts, d_t, ne, d_u, mu, lmbda, wsum, d_residual, d_values, nullptr, nullptr,
                    as_stream(stream));
    });
}

extern "C" int skg_nh_assemble_host(const skg_pattern *pat, const double *d_p, int64_t npts, const int32_t *d_t,
                                    int64_t ne, const double *d_u, double mu, double lmbda, double wsum,
                                    double *d_residual, double *d_values, double *h_residual, double *h_values,
                                    void *stream) {
    return guarded([&] {
        require(d_residual && d_values && h_residual && h_values, "device staging or host output is NULL");
        nh_assemble(pat, d_p, npts, d_t, ne, d_u, mu, lmbda, wsum, d_residual, d_values, h_residual, h_values,
                    as_stream(stream));
    });
}
