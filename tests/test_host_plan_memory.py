"""The memory estimate counts the plan of the sums: node pairs of a vector basis, every CSR entry of two bases."""
import numpy as np
import pytest

sk = pytest.importorskip("skfemntv_gb300")


class _Mesh:
    def __init__(self, E):
        self.nelements = E


class _Basis:
    def __init__(self, E, Q, nodes, comp, N):
        self.mesh, self.W, self._nodes, self._comp, self.N = _Mesh(E), np.full(Q, 1.0 / Q), nodes, comp, N
        self.element_dofs = np.zeros((nodes * comp, E), dtype=np.int64)
        self._tab = None


E, Q = 12_000, 4


def _without_plan(E, Lr, rows):
    return 20 * E * Lr + 4 * (rows + 1) + 16 * rows


@pytest.mark.parametrize("nodes,comp,per_node", [(4, 1, 0.18), (10, 1, 1.4), (4, 3, 0.18), (10, 3, 1.4)])
def test_same_basis_counts_node_pairs(nodes, comp, per_node):
    """Positions: 4 bytes for each of the n (n + 1) / 2 blocks of an element, at most doubled by padding; targets
    8 (scalar) or 16 bytes for each of the at most (nnz / comp^2 + nodes) / 2 pairs."""
    N = comp * int(E * per_node)
    est = sk.estimate_bilinear_memory(_Basis(E, Q, nodes, comp, N))
    plan = est.coloring_bytes_upper_bound - _without_plan(E, nodes * comp, N)
    positions = 4 * E * nodes * (nodes + 1) // 2
    targets = (8 if comp == 1 else 16) * (est.nnz_upper_bound // comp ** 2 + N // comp) // 2
    assert positions + targets <= plan <= 2.25 * positions + 1.1 * targets + 20_000


@pytest.mark.parametrize("test,trial", [((10, 3), (4, 1)), ((4, 1), (10, 3)), ((10, 3), (10, 3)), ((4, 1), (4, 1))])
def test_two_bases_count_every_entry(test, trial):
    """4 bytes for each entry of the element matrices, at most doubled by padding, 8 for each CSR entry."""
    a, b = (_Basis(E, Q, n, c, c * E) for n, c in (test, trial))
    est = sk.estimate_bilinear_memory(a, b)
    Lr, Lc = test[0] * test[1], trial[0] * trial[1]
    plan = est.coloring_bytes_upper_bound - _without_plan(E, Lr, a.N)
    positions, targets = 4 * E * Lr * Lc, 8 * est.nnz_upper_bound
    assert positions + targets <= plan <= 2.25 * positions + 1.1 * targets + 20_000
