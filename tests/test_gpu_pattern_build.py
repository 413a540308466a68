"""Row groups of patterns built one after another while the host reuses its memory: the groups that the device
holds are the ones that were made (P1 in the FP32-pair modes is summed by row groups; a wrong range of rows would
leave values unwritten or written twice).

Tolerance: FP64 against double-float sums of at most 24 contributions, 1e-12 of the largest entry as everywhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
sk = pytest.importorskip("skfemntv_gb300")


@pytest.mark.parametrize("cells", [(1, 1, 1), (5, 4, 3), (16, 9, 11), (30, 28, 25)])
def test_row_groups_of_consecutive_patterns(cells):
    m = sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, n + 1) for n in cells))
    basis = sk.Basis(m, sk.ElementVector(sk.ElementTetP1(), dim=1))
    kappa = np.random.default_rng(2).uniform(0.5, 2.0, (m.nelements, 1))
    stream = torch.cuda.Stream()
    forms = []
    with torch.cuda.stream(stream):
        for _ in range(6):
            forms.append(sk.NativeBilinearForm(basis))
            np.full(1 << 16, 0x7f7f7f7f, dtype=np.int32)  # host memory of the size of the groups, reused
    for form in forms:
        want = form.assemble(gradient=kappa).data.copy()
        got = form.assemble(gradient=kappa, precision="fp64_emulated").data
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


def _values(basis, rows, cols, coef):
    """Anisotropic P2 stiffness by skg_h1_assemble_affine on a pattern of the given DOF arrays: CSR matrix."""
    from scipy.sparse import csr_matrix
    from skfemntv_gb300 import _device as dev
    from skfemntv_gb300._native import SKG_FP64, call
    from skfemntv_gb300.assembly import Pattern

    m, (E, Q) = basis.mesh, basis._coefficient_shape
    pattern = Pattern(rows, cols, E, basis._nodes, basis._nodes, basis.N, basis.N)
    values = torch.empty(pattern.nnz, dtype=torch.float64, device="cuda")
    call("skg_h1_assemble_affine", pattern.h, dev.ptr(m._dev("p")), m.p.shape[1], dev.ptr(m._dev("t")), basis._nodes,
         E, Q, dev.hptr(basis.X), dev.hptr(basis.W), 1, dev.ptr(coef), SKG_FP64, dev.ptr(values), dev.stream_ptr())
    indptr, indices = pattern.host_csr()
    return csr_matrix((values.cpu().numpy(), indices, indptr), shape=(basis.N, basis.N))


@pytest.mark.parametrize("order", [1, 2])
def test_row_and_column_dofs_in_two_arrays(order):
    """Two arrays of the same content are the same pattern as one array, bit for bit; columns numbered in another
    way are another pattern, with the same entries (sums of the same terms in another order: 1e-12)."""
    m = sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, n + 1) for n in (7, 5, 3)))
    p = m.p + np.random.default_rng(3).uniform(-0.02, 0.02, m.p.shape)
    m = sk.MeshTet(p, m.t)
    if order == 2:
        m = sk.MeshTet2.from_mesh(m)
    basis = sk.Basis(m, sk.ElementVector(sk.ElementTetP2() if order == 2 else sk.ElementTetP1(), dim=1))
    B = np.random.default_rng(7).standard_normal((m.nelements, 3, 3))
    coef = torch.as_tensor(np.einsum("eij,ekj->eik", B, B) + 2 * np.eye(3), device="cuda").contiguous()
    dofs = basis._dev_dofs()
    one, two = (_values(basis, dofs, cols, coef) for cols in (dofs, dofs.clone()))
    assert np.array_equal(one.indices, two.indices) and np.array_equal(one.data, two.data)
    perm = np.random.default_rng(1).permutation(basis.N)
    other = _values(basis, dofs, torch.as_tensor(perm.astype(np.int32), device="cuda")[dofs.long()].contiguous(), coef)
    difference = abs(other[:, perm] - one)
    assert difference.max() <= 1e-12 * np.max(np.abs(one.data))
