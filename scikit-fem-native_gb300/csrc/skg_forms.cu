// Nodal H1 forms (value, gradient, symmetric gradient, divergence;
// bilinear_form_assembler.cpp:79-105) with coefficients constant on each
// element, P1 or P2, scalar or vector, on affine tetrahedra.
//
// With B_k the adjugate rows (det J times the barycentric gradients, B_0 =
// -(B_1 + B_2 + B_3)) the barycentric blocks
//   H_kl[c][d] = ( s/2 (B_k,d B_l,c + d_cd B_k.B_l) + dv B_k,c B_l,d + d_cd g B_k.B_l ) / |det J|
// carry geometry and coefficients, and the element matrix is
//   K_(a,c),(b,d) = sum_kl T^kl_ab H_kl[c][d] + d_cd v |det J| M_ab
// with the rule's tables T^kl_ab = sum_q w_q c^k_a c^l_b (grad N_a = sum_k c^k_a
// grad lambda_k, nonzero on the one or two support vertices of a only) and
// M_ab = sum_q w_q N_a N_b.  Every kind gives a symmetric matrix (H_lk =
// H_kl^T), so only the blocks a <= b are evaluated, and the pair sums
// (skg_pairs.cuh) write both places.  No point data is read or tabulated.
//
// Bound by the FP64 pipe: about 230 FP64 instructions per vector P1 element,
// 1,160 to 1,870 per vector P2 element (142 terms of 9 products and the 10 blocks
// H_kl; fewer for exact rules and without a value coefficient).
#include <algorithm>
#include <cmath>
#include <vector>

#include "skg_common.cuh"
#include "skg_fp64.cuh"
#include "skg_pairs.cuh"

namespace skg {

void gather_element_matrices(const skg_pattern *pat, const double *Ke, double *values, cudaStream_t s);

namespace {

constexpr int kFormBlock = 64;

__host__ __device__ constexpr int lo_of(int b) {
    return b < 4 ? b : (b == 4 ? 0 : b == 5 ? 1 : b == 6 ? 2 : b == 7 ? 0 : b == 8 ? 1 : 2);
}
__host__ __device__ constexpr int hi_of(int b) { return b < 4 ? b : (b == 4 ? 1 : b == 5 ? 2 : b == 6 ? 0 : 3); }

// Rule tables on the device: P1 {weight sum, M (10 packed)}; P2 {T (55 packed
// pairs x 4: supports (lo, lo), (lo, hi), (hi, lo), (hi, hi)), M (55)}.
constexpr int kP1Table = 11, kP2Table = 55 * 5;

struct FormCoefs {
    const double *arr[4];  // value, gradient, symmetric gradient, divergence: per element, or NULL
    double cst[4];
};

struct Element {
    double B[4][3], ad;  // adjugate rows, |det J|
    double vm, hs, dv, dg;  // value x |det J|; the others over |det J|; dg includes the trace part hs
};

__device__ __forceinline__ Element load_element(int64_t ne, int64_t e, const double *__restrict__ p, int64_t npts,
                                                const int32_t *__restrict__ t, const FormCoefs &fc, const Fp64 &F) {
    Element el;
    int32_t v[4];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = t[k * ne + e];
        ok = ok && v[k] >= 0 && v[k] < npts;
    }
    if (!ok) v[0] = v[1] = v[2] = v[3] = 0;
    double J[9];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double x0 = p[i * npts + v[0]];
#pragma unroll
        for (int r = 0; r < 3; ++r) J[i * 3 + r] = F.sub(p[i * npts + v[r + 1]], x0);
    }
    double (*B)[3] = el.B;
    el.ad = fabs(F.adjugate(J, B));
#pragma unroll
    for (int i = 0; i < 3; ++i) B[0][i] = -F.add3(B[1][i], B[2][i], B[3][i]);
    const auto coef = [&](int k) { return fc.arr[k] ? fc.arr[k][e] : fc.cst[k]; };
    const double inv = ok ? 1.0 / el.ad : __longlong_as_double(0x7ff8000000000000LL);
    el.vm = F.mul(coef(0), el.ad);
    el.hs = F.mul(0.5 * coef(2), inv);
    el.dv = F.mul(coef(3), inv);
    el.dg = fma(coef(1), inv, el.hs);
    return el;
}

// Gram products dg B_k . B_l: dot products for k, l >= 1, the rest from the
// zero row sums.
__device__ __forceinline__ void gram(const Element &el, double G[4][4], const Fp64 &F) {
#pragma unroll
    for (int k = 1; k < 4; ++k)
#pragma unroll
        for (int l = k; l < 4; ++l) {
            G[k][l] = F.mul(el.dg, F.dot(el.B[k], el.B[l]));
            G[l][k] = G[k][l];
        }
#pragma unroll
    for (int l = 1; l < 4; ++l) {
        G[0][l] = -F.add3(G[1][l], G[2][l], G[3][l]);
        G[l][0] = G[0][l];
    }
    G[0][0] = -F.add3(G[0][1], G[0][2], G[0][3]);
}

// Vector block (k, l), k <= l: H[c][d] = pk_d B_l,c + qk_c B_l,d (c != d),
// tk_c B_l,c + diag (c == d), with pk = hs B_k, qk = dv B_k, tk = pk + qk.
__device__ __forceinline__ void vector_block(const double pk[3], const double qk[3], const double tk[3],
                                             const double Bl[3], bool same, double diag, double H[9], const Fp64 &F) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (c == d) {
                H[c * 3 + d] = fma(tk[c], Bl[c], diag);
            } else if (!same) {
                H[c * 3 + d] = fma(pk[d], Bl[c], F.mul(qk[c], Bl[d]));
            } else if (d > c) {
                const double x = F.mul(tk[d], Bl[c]);  // diagonal block: symmetric
                H[c * 3 + d] = x;
                H[d * 3 + c] = x;
            }
        }
}

// Vector P1: blocks (np, stride, 3, 3), see skg_pairs.cuh.  MASS: there is a
// value coefficient.
template <bool MASS>
__global__ void __launch_bounds__(kFormBlock) k_form_p1v(int64_t ne, int64_t e_begin, int64_t e_end, int64_t stride,
                                                        const double *__restrict__ p, int64_t npts,
                                                        const int32_t *__restrict__ t, FormCoefs fc,
                                                        const double *__restrict__ tab, double *__restrict__ Ke) {
    __shared__ __align__(16) double stages[kFormBlock / 32 * 2 * WarpStore::kStage];
    const int lane = threadIdx.x & 31;
    const int64_t e0 = e_begin + (int64_t)blockIdx.x * kFormBlock + (threadIdx.x & ~31);
    const int n = (int)(e_end - e0 < 32 ? e_end - e0 : 32);
    if (n <= 0) return;
    WarpStore out{stages + (threadIdx.x >> 5) * 2 * WarpStore::kStage};
    const Fp64 F = Fp64::load();
    Element el = load_element(ne, lane < n ? e0 + lane : e0, p, npts, t, fc, F);  // lanes past the end: unwritten
    const double sw = __ldg(tab);
    el.hs *= sw;
    el.dv *= sw;
    el.dg *= sw;
    const double ht = F.add(el.hs, el.dv);
    double G[4][4];
    gram(el, G, F);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        double pk[3], qk[3], tk[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            pk[c] = F.mul(el.hs, el.B[a][c]);
            qk[c] = F.mul(el.dv, el.B[a][c]);
            tk[c] = F.mul(ht, el.B[a][c]);
        }
#pragma unroll
        for (int b = a; b < 4; ++b) {
            double H[9];
            vector_block(pk, qk, tk, el.B[b], a == b,
                         MASS ? fma(el.vm, __ldg(tab + 1 + tri_index(4, a, b)), G[a][b]) : G[a][b], H, F);
            double *st = out.next() + 9 * lane;
#pragma unroll
            for (int x = 0; x < 9; ++x) st[x] = H[x];
            out.store(Ke + (tri_index(4, a, b) * stride + e0) * 9, n, 9);
        }
    }
    out.finish();
}

// Coefficients of an exact rule, in units of -1/30: term (k, l) of the entry
// (a, b), with k, l among the support vertices of a, b.  The gradient of vertex
// shape a is (4 lambda_a - 1) B_a, that of edge shape (i, j) is 4 (lambda_j B_i +
// lambda_i B_j), and the integrals of lambda_m lambda_n are (1 + [m = n]) / 120.
__host__ __device__ constexpr int other_of(int b, int k) { return lo_of(b) == k ? hi_of(b) : lo_of(b); }
__host__ __device__ constexpr int exact_term(int a, int k, int b, int l) {
    const bool same = (a < 4 ? a : other_of(a, k)) == (b < 4 ? b : other_of(b, l));
    return a < 4 || b < 4 ? (same ? -3 : 1) : (same ? -8 : -4);
}

// Vector P2: the 10 blocks H_kl in registers, the 55 blocks from the rule's
// table, or for a rule exact on quadratics (EXACT) as small multiples of H / -30
// (of -4 times that between edges): 1 to 3 operations per entry instead of 1 to
// 4, and none for the blocks between vertices.  Bound by the FP64 pipe: about
// 1870 instructions per element from the table with the mass term, 1160 EXACT
// without (MASS: there is a value coefficient); 19x17x18 cells 110 -> 80 us.
template <bool EXACT, bool MASS>
__global__ void __launch_bounds__(kFormBlock, 4) k_form_p2v(int64_t ne, int64_t e_begin, int64_t e_end,
                                                           int64_t stride, const double *__restrict__ p, int64_t npts,
                                                           const int32_t *__restrict__ t, FormCoefs fc,
                                                           const double *__restrict__ tab, double *__restrict__ Ke) {
    __shared__ __align__(16) double stages[kFormBlock / 32 * 2 * WarpStore::kStage];
    __shared__ double Ts[EXACT && !MASS ? 1 : kP2Table];
    if (!EXACT || MASS) {
        for (int i = threadIdx.x; i < kP2Table; i += kFormBlock) Ts[i] = tab[i];
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const int64_t e0 = e_begin + (int64_t)blockIdx.x * kFormBlock + (threadIdx.x & ~31);
    const int n = (int)(e_end - e0 < 32 ? e_end - e0 : 32);
    if (n <= 0) return;
    WarpStore out{stages + (threadIdx.x >> 5) * 2 * WarpStore::kStage};
    const Fp64 F = Fp64::load();
    const double two = F.add(F.one, F.one), four = F.add(two, two);  // in registers
    double H[10][9], vm;
    {
        Element el = load_element(ne, lane < n ? e0 + lane : e0, p, npts, t, fc, F);
        vm = el.vm;
        if (EXACT) {
            el.hs *= -1.0 / 30.0;
            el.dv *= -1.0 / 30.0;
            el.dg *= -1.0 / 30.0;
        }
        const double ht = F.add(el.hs, el.dv);
        double G[4][4];
        gram(el, G, F);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            double pk[3], qk[3], tk[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                pk[c] = F.mul(el.hs, el.B[k][c]);
                qk[c] = F.mul(el.dv, el.B[k][c]);
                tk[c] = F.mul(ht, el.B[k][c]);
            }
#pragma unroll
            for (int l = k; l < 4; ++l)
                vector_block(pk, qk, tk, el.B[l], k == l, G[k][l], H[tri_index(4, k, l)], F);
        }
    }
#pragma unroll
    for (int a = 0; a < 10; ++a) {
        if (EXACT && a == 4) {  // from here on between edges only
#pragma unroll
            for (int q = 0; q < 10; ++q)
#pragma unroll
                for (int x = 0; x < 9; ++x) H[q][x] = F.mul(-four, H[q][x]);
        }
#pragma unroll
        for (int b = a; b < 10; ++b) {
            constexpr int kSup = 4;
            const int t4 = tri_index(10, a, b);
            const int ka[2] = {lo_of(a), hi_of(a)}, kb[2] = {lo_of(b), hi_of(b)};
            double v[9];
            bool first = true;
#pragma unroll
            for (int u = 0; u < kSup; ++u) {
                if ((u & 2 && a < 4) || (u & 1 && b < 4)) continue;  // one support vertex
                const int k = ka[u >> 1], l = kb[u & 1];
                const double T = EXACT ? 0.0 : Ts[EXACT ? 0 : t4 * 4 + u];
                const int times = a < 4 ? exact_term(a, k, b, l) : exact_term(a, k, b, l) / -4;  // -3, 1 or 2
                const double *h = H[k <= l ? tri_index(4, k, l) : tri_index(4, l, k)];
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        if (a == b && d < c) continue;  // diagonal block: symmetric
                        const double x = h[k <= l ? c * 3 + d : d * 3 + c];
                        double &r = v[c * 3 + d];
                        if (!EXACT) r = first ? F.mul(T, x) : fma(T, x, r);
                        else if (times == 1) r = first ? x : F.add(x, r);
                        else if (times == 2) r = first ? F.mul(two, x) : fma(two, x, r);
                        else r = first ? F.mul(-F.three_, x) : fma(-F.three_, x, r);
                    }
                first = false;
            }
            const double m = MASS ? F.mul(vm, Ts[MASS ? 220 + t4 : 0]) : 0.0;
            double *st = out.next() + 9 * lane;
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const double x = a == b && d < c ? v[d * 3 + c] : v[c * 3 + d];
                    st[c * 3 + d] = MASS && c == d ? F.add(x, m) : x;
                }
            out.store(Ke + ((int64_t)t4 * stride + e0) * 9, n, 9);
        }
    }
    out.finish();
}

// Scalar P1 / P2: packed upper triangles (np, stride).
template <int NN>
__global__ void __launch_bounds__(kTile) k_form_scalar(int64_t ne, int64_t e_begin, int64_t e_end, int64_t stride,
                                                       const double *__restrict__ p, int64_t npts,
                                                       const int32_t *__restrict__ t, FormCoefs fc,
                                                       const double *__restrict__ tab, double *__restrict__ Ke) {
    const int64_t e = e_begin + (int64_t)blockIdx.x * kTile + threadIdx.x;
    if (e < e_end) {
        const Fp64 F = Fp64::load();
        const Element el = load_element(ne, e, p, npts, t, fc, F);
        double G[4][4];
        gram(el, G, F);
        const double x = el.hs + el.dv;  // the one component's symmetric-gradient and divergence terms
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int l = k; l < 4; ++l) {
                G[k][l] = fma(x * el.B[k][0], el.B[l][0], G[k][l]);
                G[l][k] = G[k][l];
            }
#pragma unroll
        for (int a = 0; a < NN; ++a)
#pragma unroll
            for (int b = a; b < NN; ++b) {
                const int q = tri_index(NN, a, b);
                if constexpr (NN == 4) {
                    Ke[q * stride + e] = fma(el.vm, __ldg(tab + 1 + q), F.mul(__ldg(tab), G[a][b]));
                } else {
                    double v = F.mul(el.vm, __ldg(tab + 220 + q));
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if ((u & 2 && a < 4) || (u & 1 && b < 4)) continue;
                        v = fma(__ldg(tab + q * 4 + u), G[u & 2 ? hi_of(a) : lo_of(a)][u & 1 ? hi_of(b) : lo_of(b)], v);
                    }
                    Ke[q * stride + e] = v;
                }
            }
    }
}

std::vector<double> form_table(int nodes, int nq, const double *X, const double *W) {
    const int np = nodes * (nodes + 1) / 2;
    std::vector<double> T(nodes == 4 ? kP1Table : kP2Table, 0.0);
    for (int q = 0; q < nq; ++q) {
        const double lam[4] = {1.0 - X[q] - X[nq + q] - X[2 * nq + q], X[q], X[nq + q], X[2 * nq + q]};
        double N[10], c[10][2];  // shapes; coefficients of the support vertices' barycentric gradients
        for (int a = 0; a < nodes; ++a) {
            const int i = lo_of(a), j = hi_of(a);
            if (nodes == 4) {
                N[a] = lam[a];
                c[a][0] = 1.0;
            } else if (a < 4) {
                N[a] = lam[a] * (2.0 * lam[a] - 1.0);
                c[a][0] = 4.0 * lam[a] - 1.0;
            } else {
                N[a] = 4.0 * lam[i] * lam[j];
                c[a][0] = 4.0 * lam[j];
                c[a][1] = 4.0 * lam[i];
            }
        }
        if (nodes == 4) T[0] += W[q];
        for (int a = 0; a < nodes; ++a)
            for (int b = a; b < nodes; ++b) {
                const int k = tri_index(nodes, a, b);
                T[(nodes == 4 ? 1 : 4 * np) + k] += W[q] * N[a] * N[b];
                for (int u = 0; nodes == 10 && u < 4; ++u) {
                    if ((u & 2 && a < 4) || (u & 1 && b < 4)) continue;
                    T[k * 4 + u] += W[q] * c[a][u >> 1] * c[b][u & 1];
                }
            }
    }
    return T;
}

// True when the rule's table of gradient products is that of exact integration,
// to the rounding of its sums (at most 5e-16 for the rules of up to 343 points that
// are exact; the entries are at least 1/30).  A rule further off keeps its own
// table: the results follow the caller's rule.
bool p2_form_is_exact(const std::vector<double> &T) {
    for (int a = 0; a < 10; ++a)
        for (int b = a; b < 10; ++b)
            for (int u = 0; u < 4; ++u) {
                if ((u & 2 && a < 4) || (u & 1 && b < 4)) continue;
                const int k = u & 2 ? hi_of(a) : lo_of(a), l = u & 1 ? hi_of(b) : lo_of(b);
                if (!(std::fabs(T[tri_index(10, a, b) * 4 + u] + exact_term(a, k, b, l) / 30.0) <= 1e-15)) return false;
            }
    return true;
}

}  // namespace

void affine_forms_assemble(const skg_pattern *pat, const double *d_p, int64_t npts, const int32_t *d_t, int nodes,
                           int64_t ne, int comp, int nq, const double *h_X, const double *h_W,
                           const double *const coef[4], const double cst[4], double *d_values, double *h_values,
                           cudaStream_t s) {
    require(pat != nullptr, "pattern is NULL");
    require(nodes == 4 || nodes == 10, "affine forms take P1 (4) or P2 (10) tetrahedra");
    require(comp == 1 || comp == 3, "affine forms take 1 or 3 components");
    const int L = nodes * comp, np = nodes * (nodes + 1) / 2;
    require(ne == pat->n_elements && pat->row_local == L && pat->col_local == L, "mesh does not match the pattern");
    require(nq > 0 && h_X && h_W, "quadrature rule is empty");
    require(ne == 0 || (d_p && d_t), "mesh arrays are NULL");
    require(pat->nnz == 0 || d_values, "output is NULL");
    if (ne == 0) {
        if (pat->nnz) SKG_CUDA(cudaMemsetAsync(d_values, 0, (size_t)pat->nnz * sizeof(double), s));
        if (h_values && pat->nnz)
            SKG_CUDA(cudaMemcpyAsync(h_values, d_values, (size_t)pat->nnz * sizeof(double), cudaMemcpyDeviceToHost, s));
        return;
    }
    const std::vector<double> T = form_table(nodes, nq, h_X, h_W);
    const double *tab = device_table(T.data(), T.size(), s);
    FormCoefs fc;
    for (int k = 0; k < 4; ++k) {
        fc.arr[k] = coef[k];
        fc.cst[k] = coef[k] ? 0.0 : cst[k];
    }
    const int64_t stride = block_stride(ne);
    DevBuf<double> Ke((size_t)stride * np * (comp == 3 ? 9 : 1), s);
    const bool mass = fc.arr[0] || fc.cst[0] != 0.0;
    const bool exact = comp == 3 && nodes == 10 && p2_form_is_exact(T);
    const auto vector_form = nodes == 4 ? (mass ? k_form_p1v<true> : k_form_p1v<false>)
                             : exact    ? (mass ? k_form_p2v<true, true> : k_form_p2v<true, false>)
                                        : (mass ? k_form_p2v<false, true> : k_form_p2v<false, false>);
    auto elem = [&](int64_t e0, int64_t e1) {
        if (comp == 3)
            vector_form<<<grid_for(e1 - e0, kFormBlock), kFormBlock, 0, s>>>(ne, e0, e1, stride, d_p, npts, d_t, fc, tab,
                                                                            Ke.get());
        else if (nodes == 4)
            k_form_scalar<4><<<grid_for(e1 - e0, kTile), kTile, 0, s>>>(ne, e0, e1, stride, d_p, npts, d_t, fc, tab, Ke.get());
        else
            k_form_scalar<10><<<grid_for(e1 - e0, kTile), kTile, 0, s>>>(ne, e0, e1, stride, d_p, npts, d_t, fc, tab, Ke.get());
        SKG_LAUNCH_CHECK("form");
    };
    if (comp == 3 ? has_block_plan(pat, nodes) : pat->pairs.block == 1 && pat->pairs.nodes == nodes) {
        run_pair_passes(pat, ne, d_values, h_values, s, elem, [&](int s0, int s1, cudaStream_t st) {
            block_sums(pat->pairs, s0, s1, Ke.get(), d_values, st);
        });
        return;
    }
    elem(0, ne);
    DevBuf<double> full((size_t)ne * L * L, s);
    if (comp == 3) {
        expand_blocks(ne, nodes, Ke.get(), full.get(), s);
    } else {
        expand_packed(ne, nodes, Ke.get(), full.get(), s);
    }
    gather_element_matrices(pat, full.get(), d_values, s);
    if (h_values && pat->nnz)
        SKG_CUDA(cudaMemcpyAsync(h_values, d_values, (size_t)pat->nnz * sizeof(double), cudaMemcpyDeviceToHost, s));
}

}  // namespace skg

using namespace skg;

extern "C" int skg_h1_assemble_affine_forms(const skg_pattern *pat, const double *d_p, int64_t npts,
                                            const int32_t *d_t, int32_t nodes, int64_t ne, int32_t comp, int32_t nq,
                                            const double *h_X, const double *h_W, const double *d_value,
                                            const double *d_gradient, const double *d_symgrad, const double *d_div,
                                            double c_value, double c_gradient, double c_symgrad, double c_div,
                                            double *d_values, double *h_values, void *stream) {
    return guarded([&] {
        const double *coef[4] = {d_value, d_gradient, d_symgrad, d_div};
        const double cst[4] = {c_value, c_gradient, c_symgrad, c_div};
        affine_forms_assemble(pat, d_p, npts, d_t, nodes, ne, comp, nq, h_X, h_W, coef, cst, d_values, h_values,
                              as_stream(stream));
    });
}

extern "C" int skg_p1_assemble_affine_forms(const skg_pattern *pat, const double *d_p, int64_t npts,
                                            const int32_t *d_t, int64_t ne, int32_t comp, int32_t nq,
                                            const double *h_X, const double *h_W, const double *d_value,
                                            const double *d_gradient, const double *d_symgrad,
                                            const double *d_div, double c_value, double c_gradient,
                                            double c_symgrad, double c_div, double *d_values, double *h_values,
                                            void *stream) {
    return skg_h1_assemble_affine_forms(pat, d_p, npts, d_t, 4, ne, comp, nq, h_X, h_W, d_value, d_gradient, d_symgrad,
                                        d_div, c_value, c_gradient, c_symgrad, c_div, d_values, h_values, stream);
}
