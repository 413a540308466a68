"""A coefficient that is not finite on one element gives the fused cross forms what it gives the general path (the
contraction with the kind's tensor, whose zeros multiply it too), and leaves the other entries alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sk = pytest.importorskip("skfemntv_gb300")
import oracle as O  # noqa: E402


def _tensor(kind, Ct, Cc):
    """(row kind, column kind, contraction tensor) of a kind of NativeCrossBilinearForm.assemble."""
    if kind == "value":
        return "value", "value", np.eye(Ct)
    if kind == "gradient":
        return "gradient", "gradient", np.einsum("rc,ij->ricj", np.eye(Ct), np.eye(3))
    if kind == "row_divergence":
        return "gradient", "value", np.eye(3)[:, :, None]
    return "value", "gradient", np.eye(3)[None]


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("special", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("kind,orders,comps", [("value", (2, 1), (3, 3)), ("value", (1, 2), (1, 1)),
                                               ("gradient", (1, 2), (3, 3)), ("gradient", (2, 2), (1, 1)),
                                               ("row_divergence", (2, 1), (3, 1)), ("column_divergence", (1, 2), (1, 3))])
def test_non_finite_coefficient(kind, orders, comps, special):
    m = sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, n + 1) for n in (3, 2, 2)))
    p = m.p + np.random.default_rng(3).uniform(-0.05, 0.05, m.p.shape)
    m = sk.MeshTet2.from_mesh(sk.MeshTet(p, m.t))
    elem = {1: sk.ElementTetP1(), 2: sk.ElementTetP2()}
    test, trial = (sk.Basis(m, sk.ElementVector(elem[o], dim=c), quadrature=O.tet_quadrature_p2())
                   for o, c in zip(orders, comps))
    form = sk.NativeCrossBilinearForm(test, trial)
    c = np.random.default_rng(1).uniform(0.5, 2.0, (m.nelements, 1))
    c[7] = special
    got = form.assemble(kind, c).data.copy()
    row, column, T = _tensor(kind, *comps)
    with np.errstate(invalid="ignore"):
        full = np.broadcast_to(c, form.coefficient_shape)[(...,) + (None,) * T.ndim] * T
    want = form.assemble_tensor(row, column, full).data
    finite = np.isfinite(want)
    assert finite.any() and not finite.all()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[~finite & ~np.isnan(want)], want[~finite & ~np.isnan(want)])
    # both sum the same products
    assert np.max(np.abs(got[finite] - want[finite])) <= 1e-12 * np.max(np.abs(want[finite]))
