"""Whether a ten-node mesh is affine does not depend on points that no element uses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sk = pytest.importorskip("skfemntv_gb300")


@pytest.mark.parametrize("unused", [0.25, 1e6, np.nan])
@pytest.mark.parametrize("curved", [False, True])
def test_unused_points(curved, unused):
    m = sk.MeshTet2.from_mesh(sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, 3),) * 3))
    p = m.p.copy()
    if curved:
        p[:, m.t[4:]] += np.random.default_rng(0).uniform(-0.02, 0.02, (3, *m.t[4:].shape))
    with_unused = np.concatenate((p, np.full((3, 1), unused)), axis=1)
    scalar = sk.ElementVector(sk.ElementTetP2(), dim=1)
    plain, other = (sk.Basis(sk.MeshTet2(q, m.t), scalar) for q in (p, with_unused))
    assert plain.is_affine is other.is_affine is (not curved)
    K, L = (sk.NativeBilinearForm(b).assemble(gradient=1.0) for b in (plain, other))
    assert np.array_equal(K.data, L.data)
