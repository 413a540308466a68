// Linear-form (load / residual vector) assembly: the GPU counterpart of
// LinearFormAssembler (cpp/src/assembly/linear_form_assembler.cpp:41-154),
//   r[dof(a, c)] += sum_q w (f_c N_a + G_cj dN_a/dx_j).
// One thread per DOF walks the DOF's incidence list (element, local dof) in
// ascending element order, so the sum per DOF is made in a fixed order
// without atomics.
//
// On affine meshes the element vectors come straight from coordinates and the
// rule (k_linear_affine): the shapes and barycentric derivatives are the same
// on every element, so nothing tabulated is read, and the coefficients are read
// by strides in the layout the caller has.
#include <vector>

#include "skg_common.cuh"
#include "skg_pairs.cuh"

namespace skg {
namespace {

__global__ void k_linear_rows(int64_t n_rows, const int32_t *__restrict__ inc_ptr, const int32_t *__restrict__ inc,
                              int n, int C, int nq, const double *__restrict__ shape, const double *__restrict__ grad,
                              const double *__restrict__ w, const double *__restrict__ value,
                              const double *__restrict__ gradient, double *__restrict__ out) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    const int L = n * C;
    double acc = 0.;
    for (int32_t t = inc_ptr[r]; t < inc_ptr[r + 1]; ++t) {
        const int32_t item = inc[t];
        const int64_t e = item / L;
        const int i = item - (int)(e * L);
        const int a = i / C, c = i % C;
        double local = 0.;
        for (int q = 0; q < nq; ++q) {
            const int64_t eq = e * nq + q;
            double contrib = 0.;
            if (value) contrib += shape[eq * n + a] * value[eq * C + c];
            if (gradient) {
                const double *g = grad + (eq * n + a) * 3;
                const double *G = gradient + (eq * C + c) * 3;
                contrib += g[0] * G[0] + g[1] * G[1] + g[2] * G[2];
            }
            local += w[eq] * contrib;
        }
        acc += local;
    }
    out[r] = acc;
}

// Element strides of a coefficient: element, point, component (, direction).
struct LoadStrides {
    int64_t e, q, c, d;
};

__host__ __device__ constexpr int end0(int b) {
    return b < 4 ? b : (b == 4 ? 0 : b == 5 ? 1 : b == 6 ? 2 : b == 7 ? 0 : b == 8 ? 1 : 2);
}
__host__ __device__ constexpr int end1(int b) { return b < 4 ? b : (b == 4 ? 1 : b == 5 ? 2 : b == 6 ? 0 : 3); }

constexpr int kLoadBlock = 64;
constexpr size_t kSharedBytes = 227 * 1024;  // of one block

// Thread per element: its vector (E, NN CC) of f.v + G:grad v, the sums of all
// entries in registers, one pass over the points.  tab: per point the weight,
// NN shapes, NN x 2 coefficients of the support vertices' gradients.  Bound by
// the FP64 pipe (33 instructions per point for a P2 vector load; 20^3 43 -> 37 us
// in blocks of 64 instead of 128 elements, the values read one point ahead) and the
// read of the coefficients.
template <int NN, int CC>
__global__ void __launch_bounds__(kLoadBlock) k_linear_affine(int64_t ne, const double *__restrict__ p, int64_t npts,
                                                         const int32_t *__restrict__ t, int nq,
                                                         const double *__restrict__ tab, int n_tab,
                                                         const double *__restrict__ value, LoadStrides vs,
                                                         const double *__restrict__ gradient, LoadStrides gs,
                                                         double *__restrict__ le) {
    constexpr int L = NN * CC, kRow = 1 + 3 * NN;
    __shared__ __align__(16) double stage[kLoadBlock * L];
    extern __shared__ double Ts[];
    for (int i = threadIdx.x; i < n_tab; i += kLoadBlock) Ts[i] = tab[i];
    __syncthreads();
    const int64_t e0 = (int64_t)blockIdx.x * kLoadBlock, e = e0 + threadIdx.x;
    if (e < ne) {
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
        const double ad = ok ? fabs(det) : __longlong_as_double(0x7ff8000000000000LL);
        const double sg = det < 0.0 ? -1.0 : 1.0;  // |det J| / det J
        double acc[L];
#pragma unroll
        for (int i = 0; i < L; ++i) acc[i] = 0.0;
        double next[CC];  // values one point ahead
#pragma unroll
        for (int c = 0; c < CC; ++c) next[c] = value ? __ldg(value + e * vs.e + c * vs.c) : 0.0;
        for (int q = 0; q < nq; ++q) {
            const double *T = Ts + q * kRow;
            if (value) {
                const double w = T[0] * ad;
                double now[CC];
#pragma unroll
                for (int c = 0; c < CC; ++c) {
                    now[c] = next[c];
                    if (q + 1 < nq) next[c] = __ldg(value + e * vs.e + (q + 1) * vs.q + c * vs.c);
                }
#pragma unroll
                for (int c = 0; c < CC; ++c) {
                    const double f = w * now[c];
#pragma unroll
                    for (int a = 0; a < NN; ++a) acc[a * CC + c] = fma(T[1 + a], f, acc[a * CC + c]);
                }
            }
            if (gradient) {
                const double w = ok ? T[0] * sg : ad;
#pragma unroll
                for (int c = 0; c < CC; ++c) {
                    const double *g = gradient + e * gs.e + q * gs.q + c * gs.c;
                    const double g0 = w * __ldg(g), g1 = w * __ldg(g + gs.d), g2 = w * __ldg(g + 2 * gs.d);
                    double h[4];  // B_k . G_c
#pragma unroll
                    for (int k = 1; k < 4; ++k) h[k] = B[k][0] * g0 + B[k][1] * g1 + B[k][2] * g2;
                    h[0] = -(h[1] + h[2] + h[3]);
#pragma unroll
                    for (int a = 0; a < NN; ++a) {
                        acc[a * CC + c] = fma(T[1 + NN + 2 * a], h[end0(a)], acc[a * CC + c]);
                        if (a >= 4) acc[a * CC + c] = fma(T[2 + NN + 2 * a], h[end1(a)], acc[a * CC + c]);
                    }
                }
            }
        }
        double *st = stage + threadIdx.x * L;
#pragma unroll
        for (int i = 0; i < L; ++i) st[i] = acc[i];
    }
    store_tile(stage, le + e0 * L, (int)(ne - e0 < kLoadBlock ? ne - e0 : kLoadBlock) * L * 8);
}

// Rule tables, per point: weight, shapes, gradient coefficients.
std::vector<double> load_table(int nodes, int nq, const double *X, const double *W) {
    std::vector<double> T;
    for (int q = 0; q < nq; ++q) {
        const double lam[4] = {1.0 - X[q] - X[nq + q] - X[2 * nq + q], X[q], X[nq + q], X[2 * nq + q]};
        T.push_back(W[q]);
        for (int a = 0; a < nodes; ++a)
            T.push_back(nodes == 4 ? lam[a] : a < 4 ? lam[a] * (2.0 * lam[a] - 1.0) : 4.0 * lam[end0(a)] * lam[end1(a)]);
        for (int a = 0; a < nodes; ++a) {
            T.push_back(nodes == 4 ? 1.0 : a < 4 ? 4.0 * lam[a] - 1.0 : 4.0 * lam[end1(a)]);
            T.push_back(a < 4 ? 0.0 : 4.0 * lam[end0(a)]);
        }
    }
    return T;
}

}  // namespace

void gather_element_vectors(const skg_pattern *pat, const double *le, double *out, cudaStream_t s);

}  // namespace skg

using namespace skg;

extern "C" int skg_linear_assemble_affine(const skg_pattern *pat, const double *d_p, int64_t npts, const int32_t *d_t,
                                          int32_t nodes, int64_t ne, int32_t comp, int32_t nq, const double *h_X,
                                          const double *h_W, const double *d_value, int64_t ve, int64_t vq, int64_t vc,
                                          const double *d_gradient, int64_t ge, int64_t gq, int64_t gc, int64_t gd,
                                          double *d_out, void *stream) {
    return guarded([&] {
        require(pat != nullptr, "pattern is NULL");
        require((nodes == 4 || nodes == 10) && (comp == 1 || comp == 3), "unsupported element");
        require(ne == pat->n_elements && pat->row_local == nodes * comp, "mesh does not match the pattern");
        require(nq > 0 && h_X && h_W, "quadrature rule is empty");
        require(d_value || d_gradient, "at least one coefficient is required");
        require(d_out && (ne == 0 || (d_p && d_t)), "mesh or output arrays are NULL");
        cudaStream_t s = as_stream(stream);
        if (!pat->n_rows) return;
        const std::vector<double> T = load_table(nodes, nq, h_X, h_W);
        const double *tab = device_table(T.data(), T.size(), s);
        DevBuf<double> le((size_t)ne * nodes * comp, s);
        const LoadStrides vs{ve, vq, vc, 0}, gs{ge, gq, gc, gd};
        if (ne) {
            const size_t smem = T.size() * sizeof(double);
            // The limit belongs to the kernel, not to the launch: it is always set to the
            // same value, or a thread with a smaller rule would lower it between another's
            // two calls.
            const size_t limit = kSharedBytes - kLoadBlock * nodes * comp * sizeof(double);
            require(smem <= limit, "quadrature tables exceed shared memory");
            const auto launch = [&](auto kernel) {
                if (smem > 16 * 1024)
                    SKG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
                kernel<<<grid_for(ne, kLoadBlock), kLoadBlock, smem, s>>>(ne, d_p, npts, d_t, nq, tab, (int)T.size(), d_value, vs,
                                                               d_gradient, gs, le.get());
                SKG_LAUNCH_CHECK("linear_affine");
            };
            if (nodes == 4 && comp == 1) launch(k_linear_affine<4, 1>);
            else if (nodes == 4) launch(k_linear_affine<4, 3>);
            else if (comp == 1) launch(k_linear_affine<10, 1>);
            else launch(k_linear_affine<10, 3>);
        }
        gather_element_vectors(pat, le.get(), d_out, s);
    });
}

extern "C" int skg_linear_assemble_tabulated(const skg_pattern *pat, const int32_t *d_dofs, int64_t ne,
                                             int32_t nodes, int32_t comp, int32_t nq, const double *d_shape,
                                             const double *d_grad, const double *d_w, const double *d_value,
                                             const double *d_gradient, double *d_out, void *stream) {
    return guarded([&] {
        require(pat != nullptr, "pattern is NULL");
        require(ne == pat->n_elements && pat->row_local == nodes * comp, "tabulated arrays do not match the pattern");
        (void)d_dofs;
        cudaStream_t s = as_stream(stream);
        if (!pat->n_rows) return;
        if (ne == 0) {  // no elements: a zero vector
            require(d_out != nullptr, "output is NULL");
            SKG_CUDA(cudaMemsetAsync(d_out, 0, (size_t)pat->n_rows * sizeof(double), s));
            return;
        }
        require(d_value || d_gradient, "at least one coefficient is required");
        require(d_w && (!d_value || d_shape) && (!d_gradient || d_grad), "tabulated geometry arrays are NULL");
        k_linear_rows<<<grid_for(pat->n_rows, 128), 128, 0, s>>>(pat->n_rows, pat->inc_ptr.get(), pat->inc.get(), nodes,
                                                                 comp, nq, d_shape, d_grad, d_w, d_value, d_gradient,
                                                                 d_out);
        SKG_LAUNCH_CHECK("linear_rows");
    });
}
