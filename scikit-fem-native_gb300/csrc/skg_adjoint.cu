// Matrix-free energy J = u^T K(kappa) v of P1 diffusion and its adjoint.
//
// K(kappa) is the matrix `asm(w.kappa * ddot(grad u, grad v), basis)` builds
// for a P1 basis with per-element kappa (python/skfemntv/forms.py:276-374,
// bilinear_form_assembler.cpp:79-105); the reference has no adjoint, so the
// gradients below are checked against central finite differences through the
// assembled matrix and against exact directional derivatives of it.
//
// Per element (affine map with Jacobian J, columns x_k - x_0):
//   V   = |det J| * wsum                 (wsum = sum of the rule's weights)
//   a   = grad u_e = J^-T gu,  b = grad v_e = J^-T gv,
//         gu = (u1-u0, u2-u0, u3-u0), gv likewise
//   J_e = kappa_e V (a . b)
//   dJ/dkappa_e = V (a . b)
//   dJ/dJ       = kappa_e V ((a . b) J^-T - a c^T - b d^T),  c = J^-1 b, d = J^-1 a
//   dJ/dx_k     = column k-1 of dJ/dJ (k = 1..3),  dJ/dx_0 = -(sum of the columns)
//   dJ/du_m     = kappa_e V (grad lambda_m . b),  dJ/dv_m = kappa_e V (grad lambda_m . a)
// The backward pass recomputes the geometry (nothing is stored by the
// forward pass).  Element contributions to vertex / DOF gradients are summed
// by one thread per vertex / DOF over its incidence list in element order
// (fixed order, no atomics); the energy is reduced in a fixed tree order.
#include <vector>

#include "skg_common.cuh"
#include "skg_fp64.cuh"

namespace skg {
namespace {

// Geometry of element e: J and its cofactor matrix C = det J * J^-1 (row k of
// C is det J times the gradient of lambda_{k+1}); the kernels apply the
// powers of 1 / det J to a few scalars instead of forming J^-1.
struct ElemAdj {
    double C[4][3], id, aid;  // rows 1..3; id = 1 / det J, aid = 1 / |det J|
};

__device__ __forceinline__ void elem_geom(const double *__restrict__ p, int64_t npts, const int32_t *__restrict__ t,
                                          int64_t ne, int64_t e, const Fp64 &F, ElemAdj &g) {
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
    g.id = 1.0 / F.adjugate(J, g.C);
    g.aid = fabs(g.id);
}

// The element's differences of u and v, and a~ = det J grad u_e, b~ = det J grad v_e.
__device__ __forceinline__ void elem_fields(const ElemAdj &g, const int32_t *__restrict__ dofs,
                                            const double *__restrict__ u, const double *__restrict__ v, int64_t e,
                                            const Fp64 &F, double a[3], double b[3]) {
    const int32_t d0 = dofs[e * 4], d1 = dofs[e * 4 + 1], d2 = dofs[e * 4 + 2], d3 = dofs[e * 4 + 3];
    const double u0 = u[d0], v0 = v[d0];
    const double gu[3] = {F.sub(u[d1], u0), F.sub(u[d2], u0), F.sub(u[d3], u0)};
    const double gv[3] = {F.sub(v[d1], v0), F.sub(v[d2], v0), F.sub(v[d3], v0)};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        a[j] = fma(g.C[3][j], gu[2], fma(g.C[2][j], gu[1], F.mul(g.C[1][j], gu[0])));
        b[j] = fma(g.C[3][j], gv[2], fma(g.C[2][j], gv[1], F.mul(g.C[1][j], gv[0])));
    }
}

// 32-byte accesses: one full sector per thread.
__device__ __forceinline__ void store4(double *p, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}
__device__ __forceinline__ void load4(const double *p, double x[4]) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3]) : "l"(p));
}

constexpr int kRed = 256;

// One element's energy, the same expression in both passes (identical bits).
__device__ __forceinline__ double elem_energy(double k, double wsum, double aid, double phi, const Fp64 &F) {
    return F.mul(F.mul(F.mul(k, wsum), aid), phi);
}

// Forward: per-element energies reduced per block (fixed tree order).
__global__ void __launch_bounds__(kRed) k_energy(int64_t ne, const double *__restrict__ p, int64_t npts,
                                                 const int32_t *__restrict__ t, const int32_t *__restrict__ dofs,
                                                 const double *__restrict__ kappa, const double *__restrict__ u,
                                                 const double *__restrict__ v, double wsum,
                                                 double *__restrict__ block_sums) {
    __shared__ double red[kRed];
    const int64_t e = (int64_t)blockIdx.x * kRed + threadIdx.x;
    double f = 0.0;
    if (e < ne) {
        const Fp64 F = Fp64::load();
        ElemAdj g;
        elem_geom(p, npts, t, ne, e, F, g);
        double a[3], b[3];
        elem_fields(g, dofs, u, v, e, F, a, b);
        // kappa |det J| wsum (grad u_e . grad v_e) = kappa wsum (a~ . b~) / |det J|
        f = elem_energy(kappa ? kappa[e] : 1.0, wsum, g.aid, F.dot(a, b), F);
    }
    red[threadIdx.x] = f;
    __syncthreads();
    for (int off = kRed / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) block_sums[blockIdx.x] = red[0];
}

// One block, fixed order: thread i sums the block sums i, i + 1024, ... in
// turn, then the threads are combined by a fixed tree.
__global__ void __launch_bounds__(1024) k_sum_blocks(const double *__restrict__ in, int64_t n,
                                                     double *__restrict__ out) {
    __shared__ double red[1024];
    double s = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += 1024) s += in[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int off = 512; off > 0; off >>= 1) {
        if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

// Element e's adjoint contributions (see k_energy_grad_elem); returns its energy.
__device__ __forceinline__ double elem_adjoint(int64_t ne, const double *__restrict__ p, int64_t npts,
                                               const int32_t *__restrict__ t, const int32_t *__restrict__ dofs,
                                               const double *__restrict__ kappa, const double *__restrict__ u,
                                               const double *__restrict__ v, double wsum, double gout,
                                               double *__restrict__ gkappa, double *__restrict__ cx,
                                               double *__restrict__ cv, int64_t e) {
    const Fp64 F = Fp64::load();
    ElemAdj g;
    elem_geom(p, npts, t, ne, e, F, g);
    // with tildes for the scaled quantities:  a = a~ / det, b = b~ / det,
    // c = J^-1 b = c~ / det^2, d = J^-1 a = d~ / det^2, phi = a . b = phi~ / det^2
    double a[3], b[3], c[3], d[3];
    elem_fields(g, dofs, u, v, e, F, a, b);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        c[k] = F.dot(g.C[k + 1], b);
        d[k] = F.dot(g.C[k + 1], a);
    }
    const double phi = F.dot(a, b);
    const double k = kappa ? kappa[e] : 1.0;
    if (gkappa) gkappa[e] = gout * wsum * g.aid * phi;  // V phi = wsum phi~ / |det|
    const double s2 = F.mul(F.mul(F.mul(gout, k), wsum), g.aid);  // s / det^2 with s = gout kappa V
    const double s3 = F.mul(s2, g.id);                            // s / det^3
    // dJ/du_m = s grad lambda_m . b = s c_{m-1} (m = 1..3), dJ/dv_m = s d_{m-1};
    // lambda_0's gradient is minus the sum of the others
    double du[4] = {0.0, 0.0, 0.0, 0.0};
    if (cv) {
        double dv[4];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            du[m + 1] = F.mul(s2, c[m]);
            dv[m + 1] = F.mul(s2, d[m]);
        }
        du[0] = -F.add3(du[1], du[2], du[3]);
        dv[0] = -F.add3(dv[1], dv[2], dv[3]);
        store4(cv + e * 4, dv[0], dv[1], dv[2], dv[3]);
    }
    // dJ/dJ_ij = s (phi Ji[j][i] - a_i c_j - b_i d_j) = s / det^3 (phi~ C[j][i] - a~_i c~_j - b~_i d~_j)
    const double ph = F.mul(s3, phi);
    double as[3], bs[3], sum[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        as[i] = F.mul(s3, a[i]);
        bs[i] = F.mul(s3, b[i]);
    }
    double *out = cx + e * 16;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        double gJ[3];  // vertex j + 1
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            gJ[i] = fma(-bs[i], d[j], fma(-as[i], c[j], F.mul(ph, g.C[j + 1][i])));
            sum[i] = j == 0 ? gJ[i] : F.add(sum[i], gJ[i]);
        }
        store4(out + (j + 1) * 4, gJ[0], gJ[1], gJ[2], du[j + 1]);
    }
    store4(out, -sum[0], -sum[1], -sum[2], du[0]);
    return elem_energy(k, wsum, g.aid, phi, F);  // as k_energy forms it
}

// Backward, element pass: dJ/dkappa and the per-element vertex / DOF
// contributions (scaled by the upstream gradient).  cx: per element and vertex
// one 32-byte record (dx, dy, dz, du), stored and loaded as whole sectors; cv
// (only when dJ/du or dJ/dv is wanted): 4 dv per element.
// WITH_J: the element energies are also reduced per block exactly as
// k_energy does (same expression, same tree), so that one pass gives J and
// its gradients.
template <bool WITH_J>
__global__ void __launch_bounds__(kRed) k_energy_grad_elem(int64_t ne, const double *__restrict__ p, int64_t npts,
                                                           const int32_t *__restrict__ t,
                                                           const int32_t *__restrict__ dofs,
                                                           const double *__restrict__ kappa,
                                                           const double *__restrict__ u,
                                                           const double *__restrict__ v, double wsum, double gout,
                                                           double *__restrict__ gkappa, double *__restrict__ cx,
                                                           double *__restrict__ cv,
                                                           double *__restrict__ block_sums) {
    const int64_t e = (int64_t)blockIdx.x * kRed + threadIdx.x;
    double f = 0.0;
    if (e < ne) f = elem_adjoint(ne, p, npts, t, dofs, kappa, u, v, wsum, gout, gkappa, cx, cv, e);
    if constexpr (WITH_J) {
        __shared__ double red[kRed];
        red[threadIdx.x] = f;
        __syncthreads();
        for (int off = kRed / 2; off > 0; off >>= 1) {
            if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
            __syncthreads();
        }
        if (threadIdx.x == 0) block_sums[blockIdx.x] = red[0];
    }
}

// Backward, gather pass: one thread per row of an incidence list (vertex or
// DOF), summing the element contributions in element order.
//   coordinates (out_x, (3, n_rows), component-major like mesh.p) and / or
//   u / v DOFs (out_u, out_v (n_rows)); both in one walk when the vertex and
//   DOF incidence lists coincide (scalar P1 with every vertex a DOF).
__global__ void __launch_bounds__(128, 4) k_energy_grad_gather(int64_t n_rows, const int32_t *__restrict__ inc_ptr,
                                                            const int32_t *__restrict__ inc,
                                                            const double *__restrict__ cx,
                                                            const double *__restrict__ cv,
                                                            double *__restrict__ out_x, double *__restrict__ out_u,
                                                            double *__restrict__ out_v) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    double s[4] = {0.0, 0.0, 0.0, 0.0}, sv = 0.0;
    const int32_t end = inc_ptr[r + 1];
    for (int32_t it = inc_ptr[r]; it < end; it += 4) {  // four records in flight
        double x[4][4], y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int32_t item = it + j < end ? inc[it + j] : -1;  // element * 4 + vertex
            y[j] = -0.0;  // leaves the sums unchanged
#pragma unroll
            for (int i = 0; i < 4; ++i) x[j][i] = -0.0;
            if (item >= 0) {
                load4(cx + (int64_t)item * 4, x[j]);
                if (cv) y[j] = __ldg(cv + item);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i] += x[j][i];
            sv += y[j];
        }
    }
    if (out_x) {
        out_x[r] = s[0];
        out_x[n_rows + r] = s[1];
        out_x[2 * n_rows + r] = s[2];
    }
    if (out_u) out_u[r] = s[3];
    if (out_v) out_v[r] = sv;
}

}  // namespace
}  // namespace skg

using namespace skg;

extern "C" int skg_p1_energy(const double *d_p, int64_t npts, const int32_t *d_t, int64_t ne, const int32_t *d_dofs,
                             const double *d_kappa, const double *d_u, const double *d_v, double wsum, double *d_out,
                             void *stream) {
    return guarded([&] {
        require(ne >= 0 && d_out && (ne == 0 || (d_p && d_t && d_dofs && d_u && d_v)), "invalid energy arguments");
        cudaStream_t s = as_stream(stream);
        const int64_t nb = ne ? (ne + kRed - 1) / kRed : 1;
        DevBuf<double> partial(nb, s);
        if (ne) {
            k_energy<<<(unsigned)nb, kRed, 0, s>>>(ne, d_p, npts, d_t, d_dofs, d_kappa, d_u, d_v, wsum, partial.get());
            SKG_LAUNCH_CHECK("energy");
        } else {
            SKG_CUDA(cudaMemsetAsync(partial.get(), 0, 8, s));
        }
        k_sum_blocks<<<1, 1024, 0, s>>>(partial.get(), nb, d_out);
        SKG_LAUNCH_CHECK("energy_sum");
    });
}

namespace {
void energy_grad(const skg_pattern *vertex_inc, const skg_pattern *dof_inc, const double *d_p, int64_t npts,
                 const int32_t *d_t, int64_t ne, const int32_t *d_dofs, const double *d_kappa, const double *d_u,
                 const double *d_v, double wsum, double grad_out, double *d_energy, double *d_gkappa, double *d_gp,
                 double *d_gu, double *d_gv, cudaStream_t s) {
    {
        require(ne >= 0 && (ne == 0 || (d_p && d_t && d_dofs && d_u && d_v)), "invalid energy arguments");
        require(!d_gp || (vertex_inc && vertex_inc->row_local == 4 && vertex_inc->n_elements == ne &&
                          vertex_inc->n_rows == npts),
                "coordinate gradients need the vertex incidence handle of this mesh");
        require((!d_gu && !d_gv) || (dof_inc && dof_inc->row_local == 4 && dof_inc->n_elements == ne),
                "DOF gradients need the DOF incidence handle of this basis");
        const bool fields = d_gu || d_gv;
        DevBuf<double> cx((size_t)(ne ? ne : 1) * 16, s), cv(fields ? (size_t)(ne ? ne : 1) * 4 : 0, s);
        const int64_t nb = ne ? (ne + kRed - 1) / kRed : 1;
        DevBuf<double> partial(d_energy ? nb : 0, s);
        if (ne) {
            if (d_energy)
                k_energy_grad_elem<true><<<(unsigned)nb, kRed, 0, s>>>(ne, d_p, npts, d_t, d_dofs, d_kappa, d_u, d_v,
                                                                       wsum, grad_out, d_gkappa, cx.get(), cv.get(),
                                                                       partial.get());
            else
                k_energy_grad_elem<false><<<(unsigned)nb, kRed, 0, s>>>(ne, d_p, npts, d_t, d_dofs, d_kappa, d_u,
                                                                        d_v, wsum, grad_out, d_gkappa, cx.get(),
                                                                        cv.get(), nullptr);
            SKG_LAUNCH_CHECK("energy_grad_elem");
        } else if (d_energy) {
            SKG_CUDA(cudaMemsetAsync(partial.get(), 0, 8, s));
        }
        if (d_energy) {
            k_sum_blocks<<<1, 1024, 0, s>>>(partial.get(), nb, d_energy);
            SKG_LAUNCH_CHECK("energy_sum");
        }
        const bool shared = vertex_inc == dof_inc;  // one incidence structure for both
        if (d_gp && shared) {
            k_energy_grad_gather<<<grid_for(npts, 128), 128, 0, s>>>(npts, vertex_inc->inc_ptr.get(),
                                                                     vertex_inc->inc.get(), cx.get(), cv.get(), d_gp,
                                                                     d_gu, d_gv);
            SKG_LAUNCH_CHECK("energy_grad_xuv");
            return;
        }
        if (d_gp) {
            k_energy_grad_gather<<<grid_for(npts, 128), 128, 0, s>>>(npts, vertex_inc->inc_ptr.get(),
                                                                     vertex_inc->inc.get(), cx.get(), nullptr, d_gp,
                                                                     nullptr, nullptr);
            SKG_LAUNCH_CHECK("energy_grad_x");
        }
        if (d_gu || d_gv) {
            k_energy_grad_gather<<<grid_for(dof_inc->n_rows, 128), 128, 0, s>>>(
                dof_inc->n_rows, dof_inc->inc_ptr.get(), dof_inc->inc.get(), cx.get(), cv.get(), nullptr, d_gu, d_gv);
            SKG_LAUNCH_CHECK("energy_grad_uv");
        }
    }
}
}  // namespace

extern "C" int skg_p1_energy_grad(const skg_pattern *vertex_inc, const skg_pattern *dof_inc, const double *d_p,
                                  int64_t npts, const int32_t *d_t, int64_t ne, const int32_t *d_dofs,
                                  const double *d_kappa, const double *d_u, const double *d_v, double wsum,
                                  double grad_out, double *d_gkappa, double *d_gp, double *d_gu, double *d_gv,
                                  void *stream) {
    return guarded([&] {
        energy_grad(vertex_inc, dof_inc, d_p, npts, d_t, ne, d_dofs, d_kappa, d_u, d_v, wsum, grad_out, nullptr,
                    d_gkappa, d_gp, d_gu, d_gv, as_stream(stream));
    });
}

extern "C" int skg_p1_energy_value_and_grad(const skg_pattern *vertex_inc, const skg_pattern *dof_inc,
                                            const double *d_p, int64_t npts, const int32_t *d_t, int64_t ne,
                                            const int32_t *d_dofs, const double *d_kappa, const double *d_u,
                                            const double *d_v, double wsum, double grad_out, double *d_energy,
                                            double *d_gkappa, double *d_gp, double *d_gu, double *d_gv,
                                            void *stream) {
    return guarded([&] {
        require(d_energy != nullptr, "energy output is NULL");
        energy_grad(vertex_inc, dof_inc, d_p, npts, d_t, ne, d_dofs, d_kappa, d_u, d_v, wsum, grad_out, d_energy,
                    d_gkappa, d_gp, d_gu, d_gv, as_stream(stream));
    });
}
