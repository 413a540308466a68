"""Neo-Hookean residual and tangent at small strains and on stretched elements, against the law in extended
precision (numpy's long double, 113 bits on the Arm hosts of this GPU), formed from the displacement gradient H without the identity:

    F - F^-T = ((tr cof H + det H) I + J H + H^T - cof H) / J,   J - 1 = tr H + tr cof H + det H.

Tolerance, relative to the largest entry: an entry is a sum of at most 24 elements' entries of 7 products each;
each product is at most (aspect ratio) times the largest entry and carries about 20 roundings of 2^-53, and at
most two thirds of 24 x 7 x 20 add up: 2000 x 2^-53 x aspect ratio.  Nothing in it depends on the strain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sk = pytest.importorskip("skfemntv_gb300")

X1, W1 = np.full((3, 1), 0.25), np.array([1.0 / 6.0])
MU, LAMBDA = 1.0, 10.0
LD = np.longdouble


def _cross(a, b):
    return np.stack([a[..., i] * b[..., j] - a[..., j] * b[..., i] for i, j in ((1, 2), (2, 0), (0, 1))], axis=-1)


def _cofactors(M):  # of the rows
    return np.stack([_cross(M[:, 1], M[:, 2]), _cross(M[:, 2], M[:, 0]), _cross(M[:, 0], M[:, 1])], axis=1)


def _dot(a, b):
    return (a * b).sum(axis=-1)


def _law(p, t, u):
    """Element residuals (E, 4, 3) and tangents (E, 4, 3, 4, 3) in long double."""
    x, u = p.astype(LD)[:, t].transpose(2, 1, 0), u.astype(LD).reshape(-1, 3)[t.T]
    e, d = x[:, 1:] - x[:, :1], u[:, 1:] - u[:, :1]
    c = _cofactors(e)
    det = _dot(e[:, 0], c[:, 0])
    g = c / det[:, None, None]
    g = np.concatenate([-g.sum(axis=1, keepdims=True), g], axis=1)
    V = abs(det) / LD(6)
    H = (d[:, :, :, None] * g[:, 1:, None, :]).sum(axis=1)
    C = _cofactors(H)
    diagonal = np.eye(3, dtype=LD)
    trace = lambda M: M[:, 0, 0] + M[:, 1, 1] + M[:, 2, 2]  # noqa: E731
    second = trace(C) + _dot(H[:, 0], C[:, 0])
    J1 = trace(H) + second
    J = (1 + J1)[:, None, None]
    HT = H.transpose(0, 2, 1)
    S = (second[:, None, None] * diagonal + J * H + HT - C) / J  # F - F^-T
    FiT = ((1 + trace(H))[:, None, None] * diagonal - HT + C) / J
    lnJ = np.log1p(J1)
    P = MU * S + LAMBDA * lnJ[:, None, None] * FiT
    r = V[:, None, None] * (P[:, None] * g[:, :, None, :]).sum(axis=-1)
    h = (FiT[:, None] * g[:, :, None, :]).sum(axis=-1)
    gg = (g[:, :, None] * g[:, None]).sum(axis=-1)
    K = ((MU - LAMBDA * lnJ)[:, None, None, None, None] * h[:, :, None, None, :] * h[:, None, :, :, None].transpose(0, 1, 3, 2, 4)
         + LAMBDA * h[:, :, :, None, None] * h[:, None, None, :, :]
         + MU * gg[:, :, None, :, None] * diagonal[None, None, :, None, :])
    return r, V[:, None, None, None, None] * K


def _mesh(aspect):
    m = sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, 4),) * 3)
    p = m.p + np.random.default_rng(3).uniform(-0.03, 0.03, m.p.shape)
    p[2] /= aspect
    return sk.MeshTet(p, m.t)


def _form(m):
    return sk.NeoHookean(sk.Basis(m, sk.ElementVector(sk.ElementTetP1(), dim=3), quadrature=(X1, W1)), MU, LAMBDA)


@pytest.mark.parametrize("strain", [1e-12, 1e-8, 1e-6, 1e-3, 0.1])
@pytest.mark.parametrize("aspect", [1.0, 1e2, 1e4])
def test_residual_and_tangent(aspect, strain):
    m = _mesh(aspect)
    rng = np.random.default_rng(5)
    x = m.p.copy()
    H = strain * rng.uniform(-1.0, 1.0, (3, 3))
    # a strain of that size in every direction: a part linear in the coordinates and a bent one (whose
    # interpolation error across the thin direction has to stay below that size too)
    u = (H @ x + 0.3 * strain / aspect * np.stack([x[0] * x[1], x[1] * x[1], x[2] * x[0]])).T.ravel()
    r, K = _form(m).assemble(u)
    t = m.t
    re, Ke = _law(m.p, t, u)
    dofs = (3 * t.T[:, :, None] + np.arange(3)).reshape(-1, 12)
    res, tan = np.zeros(len(u), LD), np.zeros((len(u),) * 2, LD)
    np.add.at(res, dofs, re.reshape(-1, 12))
    np.add.at(tan, (dofs[:, :, None], dofs[:, None, :]), Ke.reshape(-1, 12, 12))
    bound = 2000 * 2.0 ** -53 * aspect
    assert np.max(abs(r - res)) <= bound * np.max(abs(res))
    assert np.max(abs(K.toarray() - tan)) <= bound * np.max(abs(tan))


def test_strong_compression():
    """Every edge shortened to 1e-4 of its length: the differences of the displaced edges' ends lose that
    factor, nothing more (ln J included, det F being 1e-12)."""
    m = _mesh(1.0)
    u = (-(1.0 - 1e-4) * m.p).T.ravel()
    r, K = _form(m).assemble(u)
    re, Ke = _law(m.p, m.t, u)
    dofs = (3 * m.t.T[:, :, None] + np.arange(3)).reshape(-1, 12)
    res, tan = np.zeros(len(u), LD), np.zeros((len(u),) * 2, LD)
    np.add.at(res, dofs, re.reshape(-1, 12))
    np.add.at(tan, (dofs[:, :, None], dofs[:, None, :]), Ke.reshape(-1, 12, 12))
    bound = 2000 * 2.0 ** -53 * 1e4
    assert np.max(abs(r - res)) <= bound * np.max(abs(res))
    assert np.max(abs(K.toarray() - tan)) <= bound * np.max(abs(tan))


@pytest.mark.parametrize("aspect", [1.0, 1e4])
@pytest.mark.parametrize("shift", [0.0, 0.5])
def test_no_residual_without_deformation(aspect, shift):
    """The undeformed state and a translation: exactly zero."""
    m = _mesh(aspect)
    r, _ = _form(m).assemble(np.full(3 * m.p.shape[1], shift))
    assert not r.any()
