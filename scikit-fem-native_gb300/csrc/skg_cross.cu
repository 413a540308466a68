// Test x trial forms between two nodal bases of one affine mesh and rule with a
// coefficient constant on each element (NativeCrossBilinearForm.assemble,
// python/skfemntv/bilinear_form.py:180-242): value, gradient, row divergence
// (vector test, scalar trial) and column divergence (scalar test, vector
// trial), straight from coordinates.
//
// The point sums collapse to tables of the rule: with B_k the adjugate rows and
// grad N_a = sum_k c^k_a B_k / det J on the support vertices of a,
//   value      |det J| sum_q w N_a N_b                       (per component)
//   gradient   sum_kl T^kl_ab B_k.B_l / |det J|              (per component)
//   column div sign(det J) sum_l R^l_ab B_l,c, R = sum_q w N_a c^l_b
//   row div    the same with the roles of a and b changed
// No contraction tensor (nine values per point for a divergence) and no
// tabulated point data is made, uploaded or read.
#include <vector>

#include "skg_common.cuh"
#include "skg_pairs.cuh"

namespace skg {

void gather_element_matrices(const skg_pattern *pat, const double *Ke, double *values, cudaStream_t s);

namespace {

enum CrossKind { kValue = 0, kGradient = 1, kRowDiv = 2, kColumnDiv = 3 };

__host__ __device__ constexpr int sup0(int b) {
    return b < 4 ? b : (b == 4 ? 0 : b == 5 ? 1 : b == 6 ? 2 : b == 7 ? 0 : b == 8 ? 1 : 2);
}
__host__ __device__ constexpr int sup1(int b) { return b < 4 ? b : (b == 4 ? 1 : b == 5 ? 2 : b == 6 ? 0 : 3); }

// Thread per (element, test node a): the Ct rows (a, r) of the element matrix
// (E, nt Ct, nc Cc).  tab (nt, nc, 4): value tables in entry 0; gradient T^kl
// over the supports; divergences R^l over the differentiated function's
// supports.
__global__ void __launch_bounds__(128, 4) k_cross_affine(int64_t ne, const double *__restrict__ p, int64_t npts,
                                                      const int32_t *__restrict__ t, int kind, int nt, int Ct, int nc,
                                                      int Cc, const double *__restrict__ tab,
                                                      const double *__restrict__ coef, double cst,
                                                      double *__restrict__ Ke) {
    extern __shared__ double Ts[];
    for (int i = threadIdx.x; i < nt * nc * 4; i += blockDim.x) Ts[i] = tab[i];
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ne * nt) return;
    const int64_t e = i / nt;
    const int a = (int)(i - e * nt), Lc = nc * Cc;
    int32_t v[4];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = t[k * ne + e];
        ok = ok && v[k] >= 0 && v[k] < npts;
    }
    if (!ok) v[0] = v[1] = v[2] = v[3] = 0;
    double J[9], B[4][3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double x0 = p[d * npts + v[0]];
#pragma unroll
        for (int r = 0; r < 3; ++r) J[d * 3 + r] = p[d * npts + v[r + 1]] - x0;
    }
    B[1][0] = J[4] * J[8] - J[5] * J[7];
    B[1][1] = J[2] * J[7] - J[1] * J[8];
    B[1][2] = J[1] * J[5] - J[2] * J[4];
    B[2][0] = J[5] * J[6] - J[3] * J[8];
    B[2][1] = J[0] * J[8] - J[2] * J[6];
    B[2][2] = J[2] * J[3] - J[0] * J[5];
    B[3][0] = J[3] * J[7] - J[4] * J[6];
    B[3][1] = J[1] * J[6] - J[0] * J[7];
    B[3][2] = J[0] * J[4] - J[1] * J[3];
    const double det = J[0] * B[1][0] + J[1] * B[2][0] + J[2] * B[3][0];
#pragma unroll
    for (int d = 0; d < 3; ++d) B[0][d] = -(B[1][d] + B[2][d] + B[3][d]);
    double c = coef ? coef[e] : cst;
    if (!ok) c = __longlong_as_double(0x7ff8000000000000LL);
    const double *T = Ts + a * nc * 4;
    const double ci = kind == kGradient ? c / fabs(det) : 0.0;
    double *row = Ke + (e * nt + a) * (int64_t)Ct * Lc;
    const auto comp = [&](int k, int d) { return d == 0 ? B[k][0] : d == 1 ? B[k][1] : B[k][2]; };
    const auto pick = [&](int k, int d) { return k == 0 ? comp(0, d) : k == 1 ? comp(1, d) : k == 2 ? comp(2, d) : comp(3, d); };
    const int a0 = sup0(a), a1 = sup1(a);
    for (int b = 0; b < nc; ++b) {
        const int b0 = sup0(b), b1 = sup1(b);
        const double *q = T + b * 4;
        if (kind == kValue || kind == kGradient) {
            double x;
            if (kind == kValue) {
                x = c * fabs(det) * q[0];
            } else {
                const auto dot = [&](int k, int l) {
                    return pick(k, 0) * pick(l, 0) + pick(k, 1) * pick(l, 1) + pick(k, 2) * pick(l, 2);
                };
                x = q[0] * dot(a0, b0);
                if (b1 != b0) x += q[1] * dot(a0, b1);
                if (a1 != a0) {
                    x += q[2] * dot(a1, b0);
                    if (b1 != b0) x += q[3] * dot(a1, b1);
                }
                x *= ci;
            }
            for (int r = 0; r < Ct; ++r)
                for (int s = 0; s < Cc; ++s) row[r * Lc + b * Cc + s] = r == s ? x : 0.0;
        } else {
            const int f0 = kind == kColumnDiv ? b0 : a0, f1 = kind == kColumnDiv ? b1 : a1;
            const double cs = det < 0.0 ? -c : c;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                double x = q[0] * pick(f0, d);
                if (f1 != f0) x += q[1] * pick(f1, d);
                row[kind == kColumnDiv ? b * 3 + d : d * Lc + b] = cs * x;
            }
        }
    }
}

// Shapes and the coefficients of the support vertices' barycentric gradients.
void shapes(int nodes, const double lam[4], double N[10], double c[10][2]) {
    for (int a = 0; a < nodes; ++a) {
        const int i = sup0(a), j = sup1(a);
        c[a][1] = 0.0;
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
}

}  // namespace
}  // namespace skg

using namespace skg;

extern "C" int skg_cross_assemble_affine(const skg_pattern *pat, const double *d_p, int64_t npts, const int32_t *d_t,
                                         int64_t ne, int32_t nq, const double *h_X, const double *h_W, int32_t kind,
                                         int32_t nt, int32_t Ct, int32_t nc, int32_t Cc, const double *d_coef,
                                         double c_coef, double *d_values, void *stream) {
    return guarded([&] {
        require(pat != nullptr, "pattern is NULL");
        require((nt == 4 || nt == 10) && (nc == 4 || nc == 10) && Ct > 0 && Cc > 0, "invalid local sizes");
        require(ne == pat->n_elements && pat->row_local == nt * Ct && pat->col_local == nc * Cc,
                "mesh does not match the pattern");
        require(kind >= kValue && kind <= kColumnDiv, "invalid cross kind");
        require(kind != kRowDiv || (Ct == 3 && Cc == 1), "row divergence requires vector test and scalar trial");
        require(kind != kColumnDiv || (Cc == 3 && Ct == 1), "column divergence requires scalar test and vector trial");
        require(kind == kRowDiv || kind == kColumnDiv || Ct == Cc,
                "value and gradient contractions require matching component counts");
        require(nq > 0 && h_X && h_W, "quadrature rule is empty");
        if (ne == 0) return;  // no elements: no CSR entries
        require(d_p && d_t && d_values, "mesh or output arrays are NULL");
        cudaStream_t s = as_stream(stream);
        std::vector<double> T((size_t)nt * nc * 4, 0.0);
        for (int q = 0; q < nq; ++q) {
            const double lam[4] = {1.0 - h_X[q] - h_X[nq + q] - h_X[2 * nq + q], h_X[q], h_X[nq + q], h_X[2 * nq + q]};
            double Na[10], ca[10][2], Nb[10], cb[10][2];
            shapes(nt, lam, Na, ca);
            shapes(nc, lam, Nb, cb);
            for (int a = 0; a < nt; ++a)
                for (int b = 0; b < nc; ++b) {
                    double *x = T.data() + (a * nc + b) * 4;
                    for (int u = 0; u < 4; ++u) {
                        if (kind == kValue) x[u] += u == 0 ? h_W[q] * Na[a] * Nb[b] : 0.0;
                        else if (kind == kGradient) x[u] += h_W[q] * ca[a][u >> 1] * cb[b][u & 1];
                        else if (u < 2) x[u] += h_W[q] * (kind == kColumnDiv ? Na[a] * cb[b][u] : Nb[b] * ca[a][u]);
                    }
                }
        }
        const double *tab = device_table(T.data(), T.size(), s);
        DevBuf<double> Ke((size_t)ne * nt * Ct * nc * Cc, s);
        k_cross_affine<<<grid_for(ne * nt, 128), 128, (size_t)nt * nc * 4 * 8, s>>>(ne, d_p, npts, d_t, kind, nt, Ct, nc,
                                                                                   Cc, tab, d_coef, c_coef, Ke.get());
        SKG_LAUNCH_CHECK("cross_affine");
        gather_element_matrices(pat, Ke.get(), d_values, s);
    });
}
