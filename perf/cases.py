"""Workloads of the assembly library, called through its public entry points.

A case is one repeated call of a finite-element program on one mesh: the unit
cube (or a box) cut into hexahedra of six tetrahedra each, interior vertices
jittered by up to a fifth of the cell size.  The program keeps its basis and
its assembler between calls, as the library's users do, and calls again with
the coefficients, displacements or fields of the next step.

Families (``kind``), each with the sizes it is used at:

  laplace     scalar P1 stiffness with one conductivity per element or with the
              coefficient 1; through ``asm`` (host matrix: the drop-in call) or
              device values (GPU solvers)
  aniso       scalar P2 diffusion with a symmetric positive tensor per element,
              device values, in each of the three precision modes
  elasticity  vector P1 or P2 linear elasticity, constant Lame parameters
  stokes      divergence coupling of P2 velocity and P1 pressure, through
              ``asm`` on two bases
  load        P2 vector load of a body force given at the quadrature points,
              through ``asm``
  maxwell     Nedelec N1 curl-curl and mass, one permeability per element
  neohooke    neo-Hookean residual and tangent at a displacement (one Newton
              iteration)
  adjoint     energy of P1 diffusion and its gradients by conductivity and node
              coordinates: forward and backward of one optimisation step
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "scikit-fem-native_gb300")
if _PKG not in sys.path:
    sys.path.insert(1, _PKG)

_EDGES = ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))
_HEX = ((0, 1, 3, 7), (0, 3, 2, 7), (0, 2, 6, 7), (0, 6, 4, 7), (0, 4, 5, 7), (0, 5, 1, 7))
_MU, _LAMBDA = 1.0, 10.0        # neo-Hookean law
_LAME = (0.8, 1.3)              # shear modulus and first Lame parameter


def listed():
    return [
        # the smallest drop-in call: a 1,296-tet matrix handed back as scipy CSR
        dict(name="laplace_p1_6_asm", kind="laplace", nx=6, ny=6, nz=6, call="asm", kappa=True),
        # plain P1 Laplace at the size of the 32^3 configuration, coefficient 1
        dict(name="laplace_p1_32", kind="laplace", nx=32, ny=32, nz=32, call="device", kappa=False),
        # the headline: P2 anisotropic diffusion, 1,572,864 tets, FP64
        dict(name="aniso_p2_64", kind="aniso", nx=64, ny=64, nz=64, precision="fp64"),
        # the FP64-accurate mode on the FP32 pipes, a box with odd counts
        dict(name="aniso_p2_37x29x31_emulated", kind="aniso", nx=37, ny=29, nz=31, precision="fp64_emulated"),
        # the mixed-precision mode (1e-7 class)
        dict(name="aniso_p2_48_split", kind="aniso", nx=48, ny=48, nz=48, precision="split_fp32"),
        # structural mechanics with linear elements
        dict(name="elasticity_p1_48", kind="elasticity", nx=48, ny=48, nz=48, order=1),
        # structural mechanics with quadratic elements, the default 11-point rule
        dict(name="elasticity_p2_19x17x18", kind="elasticity", nx=19, ny=17, nz=18, order=2),
        # Taylor-Hood coupling block of a flow solver
        dict(name="stokes_p2p1_14", kind="stokes", nx=14, ny=14, nz=14),
        # right-hand side of the same solver
        dict(name="load_p2_20", kind="load", nx=20, ny=20, nz=20),
        # Maxwell curl-curl + mass at the size of the 48^3 configuration, relabelled vertices
        dict(name="maxwell_n1_48", kind="maxwell", nx=48, ny=48, nz=48, precision="fp64"),
        # one Newton iteration of the hyperelastic configuration, 823,875 DOFs
        dict(name="neohooke_64", kind="neohooke", nx=64, ny=64, nz=64),
        # forward and backward of the differentiable energy, 1,572,864 tets
        dict(name="adjoint_64", kind="adjoint", nx=64, ny=64, nz=64),
    ]


# cells per axis, smallest and largest (geometric means of the three axes)
_RANGE = {"laplace": (2, 64), "aniso": (2, 64), "elasticity1": (2, 48), "elasticity2": (2, 18), "stokes": (2, 14),
          "load": (2, 20), "maxwell": (2, 48), "neohooke": (2, 64), "adjoint": (2, 64)}


def draw(rng):
    kind = rng.choice(["laplace", "aniso", "aniso", "elasticity", "stokes", "load", "maxwell", "neohooke", "adjoint"])
    case = dict(kind=kind)
    family = kind
    if kind == "laplace":
        case["kappa"] = rng.random() < 0.5
        case["call"] = rng.choice(["asm", "device"])
    elif kind == "aniso":
        case["precision"] = rng.choice(["fp64", "fp64_emulated", "split_fp32"])
    elif kind == "elasticity":
        case["order"] = rng.choice([1, 2])
        family = "elasticity%d" % case["order"]
    elif kind == "maxwell":
        case["precision"] = rng.choice(["fp64", "fp64", "split_fp32"])
    lo, hi = _RANGE[family]
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    cells = [max(1, round(n * math.exp(rng.uniform(-0.25, 0.25)))) for _ in range(3)]
    while math.prod(cells) > hi ** 3:
        cells = [max(1, c - 1) for c in cells]
    case["nx"], case["ny"], case["nz"] = cells
    return case


# ------------------------------------------------------------------- inputs


def _cells(case):
    return case["nx"], case["ny"], case["nz"]


def _mesh(cells, seed):
    """Vertices (3, n) float64 and tetrahedra (4, E) int64 of the jittered box."""
    nx, ny, nz = cells
    z, y, x = np.meshgrid(np.linspace(0.0, 1.0, nz + 1), np.linspace(0.0, 1.0, ny + 1), np.linspace(0.0, 1.0, nx + 1),
                          indexing="ij")
    p = np.stack((x.ravel(), y.ravel(), z.ravel()))
    rng = np.random.default_rng([seed, 11])
    inner = np.all((p > 1e-12) & (p < 1 - 1e-12), axis=0)
    h = np.array([1.0 / nx, 1.0 / ny, 1.0 / nz])[:, None]
    p[:, inner] += rng.uniform(-0.2, 0.2, size=(3, int(inner.sum()))) * h
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    n0 = (i + (nx + 1) * (j + (ny + 1) * k)).ravel()
    dx, dy, dz = 1, nx + 1, (nx + 1) * (ny + 1)
    cube = np.stack([n0, n0 + dx, n0 + dy, n0 + dx + dy, n0 + dz, n0 + dx + dz, n0 + dy + dz, n0 + dx + dy + dz])
    t = np.stack([cube[list(pattern)] for pattern in _HEX], axis=1)  # (4, 6, cubes)
    return p, np.ascontiguousarray(t.transpose(0, 2, 1).reshape(4, -1).astype(np.int64))


def _relabelled(p, t, seed):
    """The same mesh with its vertices numbered at random (the edges' orientations follow)."""
    perm = np.random.default_rng([seed, 12]).permutation(p.shape[1])
    q = np.empty_like(p)
    q[:, perm] = p
    return q, perm[t]


def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + stream)


def _normal(shape, seed, stream):
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=_generator(seed, stream))


def _spd(E, seed):
    """A = Q diag(exp(N(0, 0.5^2))) Q^T with Q a random rotation (unit quaternions): (E, 3, 3)."""
    w, x, y, z = torch.nn.functional.normalize(_normal((E, 4), seed, 1), dim=1).unbind(1)
    Q = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], dim=1).view(E, 3, 3)
    lam = torch.exp(0.5 * _normal((E, 3), seed, 2))
    A = (Q * lam[:, None, :]) @ Q.transpose(1, 2)
    return 0.5 * (A + A.transpose(1, 2))


def _kappa(E, seed, sigma):
    return torch.exp(sigma * _normal((E,), seed, 3))


def _displacement(p, seed):
    """Sum of 8 sine modes of amplitude 0.05 with axis wavevectors, node-major (3 n,)."""
    rng = np.random.default_rng([seed, 13])
    u = np.zeros_like(p)
    for _ in range(8):
        d = rng.standard_normal(3)
        d /= np.linalg.norm(d)
        axis, phase = int(rng.integers(3)), rng.uniform(0.0, 2.0 * np.pi)
        u += 0.05 * d[:, None] * np.sin(np.pi * p[axis] + phase)[None]
    return u.T.ravel()


_A4, _B4 = 0.5854101966249685, 0.1381966011250105
_RULE4 = (np.array([[_A4, _B4, _B4, _B4], [_B4, _A4, _B4, _B4], [_B4, _B4, _A4, _B4]]), np.full(4, 1.0 / 24.0))
_RULE1 = (np.full((3, 1), 0.25), np.array([1.0 / 6.0]))


def _force(E, Q, seed):
    """Body force at the quadrature points, component-first (3, E, Q), in host memory."""
    return np.random.default_rng([seed, 14]).standard_normal((3, E, Q))


def prepare(case, seed):
    import skfemntv_gb300 as sk
    from skfemntv_gb300.assembly import NativeTensorForm

    kind = case["kind"]
    p, t = _mesh(_cells(case), seed)
    if kind == "maxwell":
        p, t = _relabelled(p, t, seed)
    E = t.shape[1]
    mesh = sk.MeshTet(p, t)
    p1 = lambda dim: sk.ElementVector(sk.ElementTetP1(), dim=dim)  # noqa: E731
    p2 = lambda dim: sk.ElementVector(sk.ElementTetP2(), dim=dim)  # noqa: E731
    state = dict(kind=kind, case=case, sk=sk)
    if kind == "laplace":
        basis = sk.Basis(mesh, p1(1), quadrature=_RULE1)
        state["kappa"] = _kappa(E, seed, 1.0).cpu().numpy()[:, None] if case["kappa"] else 1.0
        if case["call"] == "asm":
            state.update(basis=basis, form=sk.BilinearForm(lambda u, v, w: w.kappa * sk.ddot(sk.grad(u), sk.grad(v))))
        else:
            state["form"] = sk.NativeBilinearForm(basis)
    elif kind == "aniso":
        basis = sk.Basis(sk.MeshTet2.from_mesh(mesh), p2(1), quadrature=_RULE4)
        state["form"] = NativeTensorForm(basis)
        state["A"] = _spd(E, seed).permute(1, 2, 0).contiguous()  # component-first (3, 3, E)
    elif kind == "elasticity":
        if case["order"] == 1:
            basis = sk.Basis(mesh, p1(3))
        else:
            basis = sk.Basis(sk.MeshTet2.from_mesh(mesh), p2(3))
        state["form"] = sk.NativeBilinearForm(basis)
    elif kind == "stokes":
        mesh2 = sk.MeshTet2.from_mesh(mesh)
        state["velocity"] = sk.Basis(mesh2, p2(3))
        state["pressure"] = sk.Basis(mesh2, p1(1), quadrature=state["velocity"].quadrature)
        state["form"] = sk.BilinearForm(lambda u, q, w: -(sk.div(u) * q))
    elif kind == "load":
        state["basis"] = sk.Basis(sk.MeshTet2.from_mesh(mesh), p2(3))
        state["f"] = _force(E, len(state["basis"].W), seed)
        state["form"] = sk.LinearForm(lambda v, w: sk.dot(w.f, v))
    elif kind == "maxwell":
        state["form"] = sk.TetN1Assembler(sk.AffineTetN1Basis(mesh))
        state["nu"] = (1.0 / _kappa(E, seed, 0.3)).cpu().numpy()[:, None]
    elif kind == "neohooke":
        state["form"] = sk.NeoHookean(sk.Basis(mesh, p1(3), quadrature=_RULE1), mu=_MU, lmbda=_LAMBDA)
        state["u"] = torch.as_tensor(_displacement(p, seed), device="cuda")
    else:
        basis = sk.Basis(mesh, p1(1), quadrature=_RULE1)
        state["op"] = sk.P1Energy(basis)
        state["kappa"] = _kappa(E, seed, 1.0)
        state["x"] = torch.as_tensor(p, device="cuda").contiguous()
        state["u"], state["v"] = _normal((basis.N,), seed, 4), _normal((basis.N,), seed, 5)
    return state


def run(state):
    kind, case, sk = state["kind"], state["case"], state["sk"]
    if kind == "laplace":
        if case["call"] == "asm":
            K = sk.asm(state["form"], state["basis"], kappa=state["kappa"])
            return K.indptr, K.indices, K.data
        return state["form"].assemble_device(gradient=state["kappa"])
    if kind == "aniso":
        return state["form"].assemble_device(None, precision=case["precision"], tensor_device=state["A"],
                                             tensor_kind=2)
    if kind == "elasticity":
        return state["form"].assemble_device(symmetric_gradient=2.0 * _LAME[0], divergence=_LAME[1])
    if kind == "stokes":
        K = sk.asm(state["form"], state["velocity"], state["pressure"])
        return K.indptr, K.indices, K.data
    if kind == "load":
        return sk.asm(state["form"], state["basis"], f=state["f"])
    if kind == "maxwell":
        return state["form"].assemble_device(mass_coefficient=1.0, curl_coefficient=state["nu"],
                                             precision=case["precision"])
    if kind == "neohooke":
        return state["form"].assemble_device(state["u"])
    kappa = state["kappa"].detach().requires_grad_(True)
    x = state["x"].detach().requires_grad_(True)
    J = state["op"](kappa, x, state["u"], state["v"])
    J.backward()
    return J.detach(), kappa.grad, x.grad


# --------------------------------------------------------------------- work


def _counts(cells):
    """Vertices, edges, faces and tetrahedra of the box."""
    x, y, z = cells
    V = (x + 1) * (y + 1) * (z + 1)
    axis = x * (y + 1) * (z + 1) + (x + 1) * y * (z + 1) + (x + 1) * (y + 1) * z
    diagonal = x * y * (z + 1) + x * (y + 1) * z + (x + 1) * y * z
    edges, T = axis + diagonal + x * y * z, 6 * x * y * z
    return V, edges, 1 - V + edges + T, T


def work(case):
    """Inputs read once (coordinates, connectivity, coefficients), outputs written
    once; the operations of the closed form of the element matrices and of the
    sums of the entries that meet in one nonzero."""
    V, S, F, T = _counts(_cells(case))
    kind = case["kind"]
    mesh1, mesh2 = 24 * V + 16 * T, 24 * V + 40 * T
    nnz1, nnz2, nnzn = V + 2 * S, V + 7 * S + 12 * F + 6 * T, S + 6 * F + 6 * T
    if kind == "laplace":
        return dict(bytes=mesh1 + 8 * nnz1 + (8 * T if case["kappa"] else 0), flops=95 * T + 16 * T - nnz1)
    if kind == "aniso":
        return dict(bytes=mesh2 + 72 * T + 8 * nnz2, flops=250 * T + 100 * T - nnz2)
    if kind == "elasticity":
        if case["order"] == 1:
            return dict(bytes=mesh1 + 72 * nnz1, flops=430 * T + 144 * T - 9 * nnz1)
        return dict(bytes=mesh2 + 72 * nnz2, flops=2500 * T + 900 * T - 9 * nnz2)
    if kind == "stokes":
        nnz = 3 * (V + 4 * S + 3 * F)
        return dict(bytes=mesh2 + 12 * nnz, flops=300 * T + 120 * T - nnz)
    if kind == "load":
        return dict(bytes=mesh2 + 24 * 11 * T + 24 * (V + S), flops=(60 + 660 + 33) * T + 30 * T)
    if kind == "maxwell":
        return dict(bytes=mesh1 + 32 * T + 8 * T + 8 * nnzn, flops=350 * T + 36 * T - nnzn)
    if kind == "neohooke":
        return dict(bytes=mesh1 + 24 * V + 24 * V + 72 * nnz1, flops=800 * T + 156 * T - 9 * nnz1)
    return dict(bytes=mesh1 + 16 * V + 8 * T + 8 * T + 24 * V, flops=250 * T + 12 * T)


# -------------------------------------------------------------------- exact


def _geometry(p, t):
    """Barycentric gradients (E, 4, 3) and |det J| (E,) in float64 on the GPU."""
    v = p[:, t[:4]].permute(2, 1, 0)  # (E, 4, 3)
    J = (v[:, 1:] - v[:, :1]).transpose(1, 2)
    c = torch.stack([torch.linalg.cross(J[:, :, 1], J[:, :, 2]), torch.linalg.cross(J[:, :, 2], J[:, :, 0]),
                     torch.linalg.cross(J[:, :, 0], J[:, :, 1])], dim=1)
    det = (c[:, 0] * J[:, :, 0]).sum(1)
    g = c / det[:, None, None]
    return torch.cat((-g.sum(1, keepdim=True), g), dim=1), det.abs()


def _edges(t, n):
    """First-seen edge ids (6, E) and the directed local edges' signs (6, E)."""
    a = torch.stack([t[i] for i, _ in _EDGES], dim=1)
    b = torch.stack([t[j] for _, j in _EDGES], dim=1)
    key = (torch.minimum(a, b) * n + torch.maximum(a, b)).reshape(-1)
    unique, inverse = torch.unique(key, return_inverse=True)
    first = torch.full(unique.shape, key.numel(), dtype=torch.int64, device=key.device)
    first.scatter_reduce_(0, inverse, torch.arange(key.numel(), device=key.device), "amin")
    rank = torch.empty_like(first)
    rank[torch.argsort(first)] = torch.arange(first.numel(), device=key.device)
    return rank[inverse].view(-1, 6).T, torch.where(a < b, 1.0, -1.0).double().T


def _csr(rows, cols, K, n_cols):
    """CSR values of the element blocks K (E, R, C) at dofs rows (E, R) x cols (E, C)."""
    key = (rows[:, :, None] * n_cols + cols[:, None, :]).reshape(-1)
    unique, inverse = torch.unique(key, return_inverse=True)
    del key
    return torch.zeros(unique.shape, dtype=torch.float64, device=K.device).index_add_(0, inverse, K.reshape(-1))


def _shapes(X, order):
    """Values (Q, n) and derivatives by the barycentric coordinates (Q, n, 4)."""
    X = torch.as_tensor(X, device="cuda")
    lam = torch.cat((1.0 - X.sum(0, keepdim=True), X)).T
    one = torch.eye(4, dtype=torch.float64, device="cuda")
    if order == 1:
        return lam, one.expand(lam.shape[0], 4, 4)
    val = [lam[:, i] * (2 * lam[:, i] - 1) for i in range(4)] + [4 * lam[:, i] * lam[:, j] for i, j in _EDGES]
    der = [(4 * lam[:, i] - 1)[:, None] * one[i] for i in range(4)]
    der += [4 * (lam[:, j][:, None] * one[i] + lam[:, i][:, None] * one[j]) for i, j in _EDGES]
    return torch.stack(val, 1), torch.stack(der, 1)


def _keast():
    a, b, c, d, e = .25, .7857142857142857, .0714285714285714, .1005964238332008, .3994035761667992
    X = np.array([[a, b, c, c, c, d, e, e, e, d, d], [a, c, c, c, b, e, d, e, d, e, d],
                  [a, c, c, b, c, e, e, d, d, d, e]])
    return X, np.array([-.01315555555555555] + [.00762222222222222] * 4 + [.02488888888888888] * 6)


def _vector(dofs):
    return (3 * dofs[:, :, None] + torch.arange(3, device=dofs.device)).flatten(1)


def exact(case, seed):
    kind = case["kind"]
    p0, t0 = _mesh(_cells(case), seed)
    if kind == "maxwell":
        p0, t0 = _relabelled(p0, t0, seed)
    p, t = torch.as_tensor(p0, device="cuda"), torch.as_tensor(t0, device="cuda")
    E, n = t.shape[1], p.shape[1]
    g, det = _geometry(p, t)
    verts = t.T
    with_edges = kind in ("aniso", "stokes", "load", "maxwell") or case.get("order") == 2
    if with_edges:
        ee, sign = _edges(t, n)
        n_edges = int(ee.max()) + 1
        quad = torch.cat((verts, ee.T + n), dim=1)  # (E, 10)
    if kind == "laplace":
        kappa = _kappa(E, seed, 1.0) if case["kappa"] else torch.ones_like(det)
        K = (g @ g.transpose(1, 2)) * (kappa * det / 6.0)[:, None, None]
        values = _csr(verts, verts, K, n)
        return (None, None, values.cpu().numpy()) if case["call"] == "asm" else values
    if kind == "aniso":
        _, D = _shapes(_RULE4[0], 2)
        G = (g @ _spd(E, seed) @ g.transpose(1, 2)) * det[:, None, None]
        T = torch.einsum("q,qak,qbl->klab", torch.as_tensor(_RULE4[1], device="cuda"), D, D)
        return _csr(quad, quad, (G.view(E, 16) @ T.reshape(16, 100)).view(E, 10, 10), n + n_edges)
    if kind == "elasticity":
        mu, lam = _LAME
        X, W = _RULE4 if case["order"] == 1 else _keast()
        _, D = _shapes(X, case["order"])
        nodes, N = (verts, n) if case["order"] == 1 else (quad, n + n_edges)
        m = nodes.shape[1]
        K = torch.zeros((E, m, 3, m, 3), dtype=torch.float64, device="cuda")
        for q in range(len(W)):
            d = D[q] @ g  # (E, m, 3)
            o = torch.einsum("eac,ebd->eacbd", d, d) * (det * W[q])[:, None, None, None, None]
            K += lam * o + mu * o.transpose(2, 4)
            tr = torch.einsum("eacbc->eab", o)
            for c in range(3):
                K[:, :, c, :, c] += mu * tr
        dofs = _vector(nodes)
        return _csr(dofs, dofs, K.view(E, 3 * m, 3 * m), 3 * N)
    if kind == "stokes":
        X, W = _keast()
        _, D = _shapes(X, 2)
        psi, _ = _shapes(X, 1)
        R = torch.einsum("q,qi,qak->iak", torch.as_tensor(W, device="cuda"), psi, D)
        K = -torch.einsum("iak,ekc,e->eiac", R, g, det).reshape(E, 4, 30)
        return None, None, _csr(verts, _vector(quad), K, 3 * (n + n_edges)).cpu().numpy()
    if kind == "load":
        X, W = _keast()
        phi, _ = _shapes(X, 2)
        f = torch.as_tensor(_force(E, len(W), seed), device="cuda")
        local = torch.einsum("q,qa,ceq,e->eac", torch.as_tensor(W, device="cuda"), phi, f, det).reshape(E, 30)
        out = torch.zeros(3 * (n + n_edges), dtype=torch.float64, device="cuda")
        return out.index_add_(0, _vector(quad).reshape(-1), local.reshape(-1)).cpu().numpy()
    if kind == "maxwell":
        # phi_a = lambda_i g_j - lambda_j g_i, int lambda_i lambda_j = det (1 + delta_ij) / 120
        nu = 1.0 / _kappa(E, seed, 0.3)
        i, j = (torch.tensor(list(k), device="cuda") for k in zip(*_EDGES))
        gg = (g @ g.transpose(1, 2)) * (det / 120.0)[:, None, None]
        d = torch.eye(4, dtype=torch.float64, device="cuda")
        pair = lambda a, b: 1.0 + d[a][:, b]  # noqa: E731
        M = (pair(i, i) * gg[:, j][:, :, j] - pair(i, j) * gg[:, j][:, :, i] - pair(j, i) * gg[:, i][:, :, j]
             + pair(j, j) * gg[:, i][:, :, i])
        curl = 2.0 * torch.linalg.cross(g[:, i], g[:, j])
        K = M + (curl @ curl.transpose(1, 2)) * (nu * det / 6.0)[:, None, None]
        K = K * sign.T[:, :, None] * sign.T[:, None, :]
        return _csr(ee.T, ee.T, K, n_edges)
    if kind == "neohooke":
        u = torch.as_tensor(_displacement(p0, seed), device="cuda").view(n, 3)
        F = torch.einsum("eac,eaj->ecj", u[verts], g) + torch.eye(3, dtype=torch.float64, device="cuda")
        Fi = torch.linalg.inv(F)
        lnJ = torch.log(torch.linalg.det(F))
        vol = det / 6.0
        FiT = Fi.transpose(1, 2)
        P = _MU * (F - FiT) + _LAMBDA * lnJ[:, None, None] * FiT
        dofs = _vector(verts)
        r = torch.zeros(3 * n, dtype=torch.float64, device="cuda")
        r.index_add_(0, dofs.reshape(-1), (torch.einsum("ecj,eaj->eac", P, g) * vol[:, None, None]).reshape(-1))
        h = torch.einsum("eij,eaj->eai", FiT, g)
        K = torch.einsum("eak,ebi->eaibk", h, h) * (_MU - _LAMBDA * lnJ)[:, None, None, None, None]
        K += _LAMBDA * torch.einsum("eai,ebk->eaibk", h, h)
        gg = _MU * (g @ g.transpose(1, 2))
        for c in range(3):
            K[:, :, c, :, c] += gg
        K *= vol[:, None, None, None, None]
        return r, _csr(dofs, dofs, K.reshape(E, 12, 12), 3 * n)
    kappa = _kappa(E, seed, 1.0)
    x = p.clone().requires_grad_(True)
    u, v = _normal((n,), seed, 4), _normal((n,), seed, 5)
    g, det = _geometry(x, t)
    energy = (torch.einsum("ea,eaj->ej", u[verts], g) * torch.einsum("ea,eaj->ej", v[verts], g)).sum(1) * det / 6.0
    J = (kappa * energy).sum()
    J.backward()
    return J.detach(), energy.detach(), x.grad
