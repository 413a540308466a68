"""Pair sums against the oracle where tiles, windows and slices end: one cell, a tile of 64 elements
and two more, whole tiles, an odd box; scalar, symmetric and partly nonsymmetric coefficients.

Tolerances (largest error over the largest entry): an FP64 entry is at most 24 contributions of about 60
roundings each, 2^-53 apiece relative to the contributions: 1e-12 holds with margin; double-float 1e-12 and
split FP32 1e-7 are the modes' own bounds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sk = pytest.importorskip("skfemntv_gb300")
import oracle as O  # noqa: E402
from skfemntv_gb300.assembly import NativeTensorForm  # noqa: E402

BOUND = {"fp64": 1e-12, "fp64_emulated": 1e-12, "split_fp32": 1e-7}


def _mesh(cells, seed=3):
    m = sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, n + 1) for n in cells))
    rng = np.random.default_rng(seed)
    p = m.p + rng.uniform(-0.15, 0.15, m.p.shape) / np.array(cells)[:, None]
    return sk.MeshTet(p, m.t)


def _tensors(E, kind):
    rng = np.random.default_rng(7)
    B = rng.standard_normal((E, 3, 3))
    A = np.einsum("eij,ekj->eik", B, B) + 2 * np.eye(3)
    if kind == "mixed":  # the last element of the first tile and the mesh's last one
        for e in {min(63, E - 1), E - 1}:
            A[e, 0, 2] += 0.7
            A[e, 2, 1] -= 0.4
    return A


@pytest.mark.parametrize("kind", ["symmetric", "mixed"])
@pytest.mark.parametrize("cells", [(1, 1, 1), (11, 1, 1), (4, 4, 4), (7, 5, 3)])
@pytest.mark.parametrize("precision", sorted(BOUND))
@pytest.mark.parametrize("order", [1, 2])
def test_tensor_form(order, precision, cells, kind):
    m = _mesh(cells)
    if order == 2:
        m = sk.MeshTet2.from_mesh(m)
    elem = sk.ElementTetP2() if order == 2 else sk.ElementTetP1()
    basis = sk.Basis(m, sk.ElementVector(elem, dim=1))
    E, Q = basis._coefficient_shape
    A = np.broadcast_to(np.moveaxis(_tensors(E, kind), 0, -1)[..., None], (3, 3, E, Q))
    K = NativeTensorForm(basis).assemble(A, precision)
    ob = O.make_basis(m.p, m.t, order == 2, quadrature=(basis.X, basis.W))
    data, indptr, indices = O.cross_gradient_tensor_assemble(ob, O.anisotropic_tensor(A, ob.dx.shape))
    assert np.array_equal(K.indptr, indptr) and np.array_equal(K.indices, indices)
    assert np.max(np.abs(K.data - data)) <= BOUND[precision] * np.max(np.abs(data))


X1, W1 = np.full((3, 1), 0.25), np.array([1.0 / 6.0])
KINDS = ("value", "gradient", "symmetric_gradient", "divergence")


@pytest.mark.parametrize("one_point", [False, True])
@pytest.mark.parametrize("cells", [(1, 1, 1), (11, 1, 1), (4, 4, 4), (7, 5, 3)])
@pytest.mark.parametrize("order,comp", [(1, 1), (1, 3), (2, 1), (2, 3)])
def test_affine_forms(order, comp, cells, one_point):
    """Every kind at once, per element and constant, on the default rules and on one that is not exact on
    quadratics; bound as above (an entry of the vector P2 matrix takes about 60 roundings as well)."""
    m = _mesh(cells)
    if order == 2:
        m = sk.MeshTet2.from_mesh(m)
    elem = sk.ElementTetP2() if order == 2 else sk.ElementTetP1()
    quadrature = (X1, W1) if one_point else None
    basis = sk.Basis(m, sk.ElementVector(elem, dim=comp), quadrature=quadrature)
    ob = O.make_basis(m.p, m.t, order == 2, comp=comp, quadrature=quadrature)
    form = sk.NativeBilinearForm(basis)
    rng = np.random.default_rng(1)
    E, Q = basis._coefficient_shape
    for co in ({k: rng.uniform(0.5, 2.0, (E, 1)) for k in KINDS}, dict(zip(KINDS, (0.5, 0.8, 1.6, 1.3)))):
        K = form.assemble(**co)
        assert basis._tab is None  # no tabulated point data
        full = {k: np.broadcast_to(c, (E, Q)) for k, c in co.items()}
        data, indptr, indices = O.bilinear_assemble(ob, **full)
        assert np.array_equal(K.indptr, indptr) and np.array_equal(K.indices, indices)
        assert np.max(np.abs(K.data - data)) <= 1e-12 * np.max(np.abs(data))


@pytest.mark.parametrize("one_point", [False, True])
@pytest.mark.parametrize("cells", [(1, 1, 1), (11, 1, 1), (7, 5, 3)])
@pytest.mark.parametrize("order", [1, 2])
def test_vector_forms_without_a_value_term(order, cells, one_point):
    """As above, without the mass term."""
    m = _mesh(cells)
    if order == 2:
        m = sk.MeshTet2.from_mesh(m)
    quadrature = (X1, W1) if one_point else None
    basis = sk.Basis(m, sk.ElementVector(sk.ElementTetP2() if order == 2 else sk.ElementTetP1(), dim=3),
                     quadrature=quadrature)
    ob = O.make_basis(m.p, m.t, order == 2, comp=3, quadrature=quadrature)
    E, Q = basis._coefficient_shape
    rng = np.random.default_rng(4)
    co = {"gradient": 0.8, "symmetric_gradient": rng.uniform(0.5, 2.0, (E, 1)), "divergence": 1.3}
    K = sk.NativeBilinearForm(basis).assemble(**co)
    data, _, _ = O.bilinear_assemble(ob, **{k: np.broadcast_to(c, (E, Q)) for k, c in co.items()})
    assert np.max(np.abs(K.data - data)) <= 1e-12 * np.max(np.abs(data))


def _affine_pair(cells, orders, comps):
    m = sk.MeshTet2.from_mesh(_mesh(cells))
    elem = {1: sk.ElementTetP1(), 2: sk.ElementTetP2()}
    return [sk.Basis(m, sk.ElementVector(elem[o], dim=c), quadrature=O.tet_quadrature_p2()) for o, c in zip(orders, comps)]


@pytest.mark.parametrize("cells", [(1, 1, 1), (11, 1, 1), (7, 5, 3)])
@pytest.mark.parametrize("kind,orders,comps", [("column_divergence", (1, 2), (1, 3)), ("row_divergence", (2, 1), (3, 1)),
                                               ("value", (2, 1), (1, 1)), ("gradient", (1, 2), (3, 3)),
                                               ("gradient", (2, 2), (1, 1)), ("value", (2, 2), (3, 3))])
def test_cross_kinds_from_coordinates(kind, orders, comps, cells):
    """Coefficients constant per element go through the fused cross kernel; the same coefficients with one
    point off by one unit in the last place go through the tabulated tensor path, and agree to 1e-12 of the
    largest entry (both sum the same products; the perturbation is 2^-52)."""
    test, trial = _affine_pair(cells, orders, comps)
    form = sk.NativeCrossBilinearForm(test, trial)
    E, Q = form.coefficient_shape
    for c in (np.full((E, 1), 1.7) + np.arange(E)[:, None] / E, 0.6):
        fused = form.assemble(kind, c)
        per_point = np.array(np.broadcast_to(c, (E, Q)))
        per_point[0, 0] = np.nextafter(per_point[0, 0], 9.0)
        general = form.assemble(kind, per_point)
        assert np.array_equal(fused.indptr, general.indptr) and np.array_equal(fused.indices, general.indices)
        assert np.max(np.abs(fused.data - general.data)) <= 1e-12 * np.max(np.abs(general.data))


@pytest.mark.parametrize("cells", [(1, 1, 1), (11, 1, 1), (4, 4, 4), (7, 5, 3)])
@pytest.mark.parametrize("order,comp", [(1, 1), (1, 3), (2, 1), (2, 3)])
def test_affine_loads_in_every_layout(order, comp, cells):
    """Constant, per-element, per-point, component-first, transposed and reversed coefficients against the
    oracle; at most 24 elements of 11 points with about 10 roundings each: 1e-12 of the largest entry."""
    m = _mesh(cells)
    if order == 2:
        m = sk.MeshTet2.from_mesh(m)
    basis = sk.Basis(m, sk.ElementVector(sk.ElementTetP2() if order == 2 else sk.ElementTetP1(), dim=comp))
    ob = O.make_basis(m.p, m.t, order == 2, comp=comp, quadrature=(basis.X, basis.W))
    form = sk.NativeLinearForm(basis)
    E, Q = basis._coefficient_shape
    rng = np.random.default_rng(2)
    shape = (E, Q, comp)
    cases = [(rng.standard_normal(comp), rng.standard_normal((comp, 3))), (rng.standard_normal((E, 1, comp)), None),
             (np.moveaxis(rng.standard_normal((comp, E, Q)), 0, -1), rng.standard_normal(shape + (3,))),
             (rng.standard_normal((Q, E, comp)).transpose(1, 0, 2), np.moveaxis(rng.standard_normal((comp, 3, E, Q)), (0, 1), (-2, -1))),
             (None, np.broadcast_to(rng.standard_normal((E, 1, 1, 3)), shape + (3,))), (rng.standard_normal(shape)[::-1], None)]
    for value, gradient in cases:
        got, _ = form.assemble(value=value, gradient=gradient)
        assert basis._tab is None
        full = [None if c is None else np.ascontiguousarray(np.broadcast_to(c, shape + tail))
                for c, tail in ((value, ()), (gradient, (3,)))]
        want = O.linear_assemble(ob, value=full[0], gradient=full[1])
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("terms", ["both", "mass", "curl"])
@pytest.mark.parametrize("cells", [(1, 1, 1), (11, 1, 1), (4, 4, 4), (7, 5, 3)])
@pytest.mark.parametrize("intorder", [1, 2, 4])
def test_n1_rules(intorder, cells, terms):
    """Coefficients per element on a rule that is not exact for the mass term and on two that are; about 24
    contributions of 60 roundings: 1e-12 of the largest entry."""
    m = _mesh(cells)
    rng = np.random.default_rng(5)
    mass, curl = rng.uniform(0.5, 2.0, (2, m.t.shape[1], 1)) * np.array([terms != "curl", terms != "mass"])[:, None, None]
    K = sk.TetN1Assembler(sk.AffineTetN1Basis(m, intorder=intorder)).assemble_maxwell(mass_coefficient=mass,
                                                                                      curl_coefficient=curl)
    data, indptr, indices = O.n1_assemble_maxwell(O.make_n1_basis(m.p, m.t, intorder), mass, curl)
    assert np.array_equal(K.indptr, indptr) and np.array_equal(K.indices, indices)
    assert np.max(np.abs(K.data - data)) <= 1e-12 * np.max(np.abs(data))


@pytest.mark.parametrize("law", ["plain", "learned", "learned, all elements by the plain law"])
@pytest.mark.parametrize("cells", [(1, 1, 1), (11, 1, 1), (4, 4, 4), (7, 5, 3)])
def test_neo_hookean(cells, law, surrogate):
    """Residual and tangent.  FP64 entries, and FP64 entries carried in two FP32 parts (2^-48 apiece), as above;
    the learned law's own error is 1e-4 at this deformation, 1e-3 holds with margin."""
    m = _mesh(cells)
    b = sk.Basis(m, sk.ElementVector(sk.ElementTetP1(), dim=3), quadrature=(X1, W1))
    rng = np.random.default_rng(11)
    G = rng.uniform(-0.08, 0.08, (3, 3))
    u = (G @ m.p + 0.01 * np.sin(np.pi * m.p[::-1]) / max(cells)).T.ravel()
    r, K = sk.NeoHookean(b, 1.0, 10.0).assemble(
        u, **({} if law == "plain" else dict(surrogate=surrogate, tol=1e-2 if law == "learned" else -1.0)))
    x = m.p[:, m.t]
    J = np.moveaxis(x[:, 1:] - x[:, :1], -1, 0)
    g = np.linalg.inv(J)
    g = np.concatenate([-g.sum(axis=1, keepdims=True), g], axis=1)  # (E, 4, 3)
    V = np.abs(np.linalg.det(J)) / 6.0
    Gu = np.einsum("eac,eaj->ecj", u.reshape(-1, 3)[m.t.T], g)
    re = np.einsum("e,ecj,eaj->eac", V, O.nh_first_piola(Gu, 1.0, 10.0), g).reshape(len(V), 12)
    Ke = np.einsum("e,ericj,eai,ebj->earbc", V, O.nh_tangent(Gu, 1.0, 10.0), g, g).reshape(len(V), 12, 12)
    dofs = (3 * m.t.T[:, :, None] + np.arange(3)).reshape(len(V), 12)
    res, tan = np.zeros(b.N), np.zeros((b.N, b.N))
    np.add.at(res, dofs, re)
    np.add.at(tan, (dofs[:, :, None], dofs[:, None, :]), Ke)
    bound = 1e-3 if law == "learned" else 1e-12
    assert np.max(np.abs(r - res)) <= bound * np.max(np.abs(res))
    assert np.max(np.abs(K.toarray() - tan)) <= bound * np.max(np.abs(tan))
