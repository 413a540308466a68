"""Results follow the caller's quadrature rule, also one that is exact but for its last digits.

Tolerance: an entry sums at most 24 contributions of about 60 roundings of 2^-53, whose absolute sum is at most 8
times the largest entry: 60 x 2^-53 x 8, a sixth of what the perturbed weights change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sk = pytest.importorskip("skfemntv_gb300")
import oracle as O  # noqa: E402


@pytest.mark.parametrize("value", [False, True])
def test_p2_vector_rule_with_perturbed_weights(value):
    """Weights 3e-13 too large (relative): so is every entry."""
    m = sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, 4),) * 3)
    p = m.p + np.random.default_rng(3).uniform(-0.04, 0.04, m.p.shape)
    m = sk.MeshTet2.from_mesh(sk.MeshTet(p, m.t))
    X, W = O.tet_quadrature_p1()
    rule = (X, W * (1.0 + 3e-13))
    basis = sk.Basis(m, sk.ElementVector(sk.ElementTetP2(), dim=3), quadrature=rule)
    ob = O.make_basis(m.p, m.t, True, comp=3, quadrature=rule)
    co = {"symmetric_gradient": 1.6, "divergence": 1.3}
    if value:
        co["value"] = 0.7
    K = sk.NativeBilinearForm(basis).assemble(**co)
    data, indptr, indices = O.bilinear_assemble(ob, **{k: np.broadcast_to(np.float64(c), basis._coefficient_shape)
                                                       for k, c in co.items()})
    assert np.array_equal(K.indptr, indptr) and np.array_equal(K.indices, indices)
    assert np.max(np.abs(K.data - data)) <= 60 * 2.0 ** -53 * 8 * np.max(np.abs(data))
