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
