"""Vector P1 matrices whose DOFs are not numbered node by node (component after component, and at random): the same
sums in the same order as the node by node numbering, so the same values bit for bit, from the packed blocks alone
(no full element matrices: 90 doubles per element, 90 floats in two parts for the learned law).  With a host result,
by chunks (more than 2^22 values at 32^3) and whole."""
import numpy as np
import pytest
from test_gpu_pair_memory import _peak

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
sk = pytest.importorskip("skfemntv_gb300")

X1, W1 = np.full((3, 1), 0.25), np.array([1.0 / 6.0])


def _bases(cells, numbering):
    """A basis numbered node by node, the same basis renumbered on the device, and the new DOF of each DOF."""
    m = sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, n + 1) for n in cells))
    p = m.p + np.random.default_rng(3).uniform(-0.1, 0.1, m.p.shape) / np.array(cells)[:, None]
    m = sk.MeshTet(p, m.t)
    plain, other = (sk.Basis(m, sk.ElementVector(sk.ElementTetP1(), dim=3), quadrature=(X1, W1)) for _ in range(2))
    dofs = np.arange(plain.N)
    new = dofs % 3 * (plain.N // 3) + dofs // 3 if numbering == "components" else np.random.default_rng(1).permutation(dofs)
    other._dofs_dev = torch.as_tensor(new.astype(np.int32), device="cuda")[plain._dev_dofs().long()].contiguous()
    return plain, other, new


def _same(K, L, new):
    """L renumbered back is K, bit for bit."""
    back = L.tocoo()
    old = np.empty_like(new)
    old[new] = np.arange(len(new))
    row, col = old[back.row], old[back.col]
    order = np.lexsort((col, row))
    return np.array_equal(K.indices, col[order]) and np.array_equal(K.data, back.data[order])


@pytest.mark.parametrize("numbering", ["components", "random"])
@pytest.mark.parametrize("cells", [(1, 1, 1), (7, 5, 3), (32, 32, 32)])
def test_elasticity(cells, numbering):
    plain, other, new = _bases(cells, numbering)
    co = dict(value=0.5, symmetric_gradient=1.6, divergence=1.3)
    forms = [sk.NativeBilinearForm(b) for b in (plain, other)]
    K, L = (f.assemble(**co) for f in forms)
    assert _same(K, L, new)
    stride = -(-plain.mesh.nelements // 128) * 128
    for f in forms:
        assert _peak(lambda: f.assemble_device(**co)) <= 720 * stride + (1 << 16)


@pytest.mark.parametrize("law", ["plain", "learned", "learned, all elements by the plain law"])
@pytest.mark.parametrize("numbering", ["components", "random"])
@pytest.mark.parametrize("cells", [(1, 1, 1), (7, 5, 3), (32, 32, 32)])
def test_neo_hookean(cells, numbering, law, surrogate):
    plain, other, new = _bases(cells, numbering)
    m = plain.mesh
    G = np.random.default_rng(11).uniform(-0.08, 0.08, (3, 3))
    u = (G @ m.p + 0.01 * np.sin(np.pi * m.p[::-1]) / max(cells)).T.ravel()
    v = np.empty_like(u)
    v[new] = u
    kw = {} if law == "plain" else dict(surrogate=surrogate, tol=1e-2 if law == "learned" else -1.0)
    r, K = sk.NeoHookean(plain, 1.0, 10.0).assemble(u, **kw)
    s, L = sk.NeoHookean(other, 1.0, 10.0).assemble(v, **kw)
    assert np.array_equal(r, s[new])
    assert _same(K, L, new)
