"""The element passes and pair sums where their tiles end (128 elements; warps of 32 and blocks of 64 for vector
forms and loads), and the FP64 passes that take over when a value leaves the FP32 range, on meshes large enough for
their blocks to walk several tiles and windows (more than 304 tiles and 608 windows; 608 tiles for N1).

Tolerances: those of test_gpu_pairs.py against the oracle (1e-12 of the largest entry, 1e-7 split).  The FP64 passes
behind an FP32-pair call run the kernels of the FP64 call on the same data: bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
sk = pytest.importorskip("skfemntv_gb300")
import oracle as O  # noqa: E402
from skfemntv_gb300.assembly import NativeTensorForm  # noqa: E402

BOUND = {"fp64": 1e-12, "fp64_emulated": 1e-12, "split_fp32": 1e-7}


def _mesh(E, quadratic):
    """The first E elements of a jittered box, without the vertices they do not use."""
    m = sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, n + 1) for n in (5, 4, 3)))
    p = m.p + np.random.default_rng(3).uniform(-0.03, 0.03, m.p.shape)
    used, t = np.unique(m.t[:, :E], return_inverse=True)
    m = sk.MeshTet(p[:, used], t.reshape(4, E))
    return sk.MeshTet2.from_mesh(m) if quadratic else m


def _tensors(E, nonsymmetric):
    rng = np.random.default_rng(7)
    B = rng.standard_normal((E, 3, 3))
    A = np.einsum("eij,ekj->eik", B, B) + 2 * np.eye(3)
    for e in nonsymmetric:
        if e < E:
            A[e, 0, 2] += 0.7
            A[e, 2, 1] -= 0.4
    return A


@pytest.mark.parametrize("nonsymmetric", [(), (127,), (128,), (127, 128)])
@pytest.mark.parametrize("E", [127, 128, 129, 256, 257])
@pytest.mark.parametrize("precision", sorted(BOUND))
@pytest.mark.parametrize("order", [1, 2])
def test_tensor_form_at_tile_ends(order, precision, E, nonsymmetric):
    m = _mesh(E, order == 2)
    elem = sk.ElementTetP2() if order == 2 else sk.ElementTetP1()
    basis = sk.Basis(m, sk.ElementVector(elem, dim=1))
    Q = len(basis.W)
    A = np.broadcast_to(np.moveaxis(_tensors(E, nonsymmetric), 0, -1)[..., None], (3, 3, E, Q))
    K = NativeTensorForm(basis).assemble(A, precision)
    ob = O.make_basis(m.p, m.t, order == 2, quadrature=(basis.X, basis.W))
    data, indptr, indices = O.cross_gradient_tensor_assemble(ob, O.anisotropic_tensor(A, ob.dx.shape))
    assert np.array_equal(K.indptr, indptr) and np.array_equal(K.indices, indices)
    assert np.max(np.abs(K.data - data)) <= BOUND[precision] * np.max(np.abs(data))


@pytest.mark.parametrize("E", [31, 32, 33, 63, 64, 65, 127, 128, 129])
@pytest.mark.parametrize("order,comp", [(1, 1), (1, 3), (2, 1), (2, 3)])
def test_forms_and_loads_at_block_ends(order, comp, E):
    m = _mesh(E, order == 2)
    elem = sk.ElementTetP2() if order == 2 else sk.ElementTetP1()
    basis = sk.Basis(m, sk.ElementVector(elem, dim=comp))
    ob = O.make_basis(m.p, m.t, order == 2, comp=comp, quadrature=(basis.X, basis.W))
    rng = np.random.default_rng(1)
    Q = len(basis.W)
    co = {k: rng.uniform(0.5, 2.0, (E, 1)) for k in ("value", "gradient", "symmetric_gradient", "divergence")}
    K = sk.NativeBilinearForm(basis).assemble(**co)
    data, indptr, indices = O.bilinear_assemble(ob, **{k: np.broadcast_to(c, (E, Q)) for k, c in co.items()})
    assert np.array_equal(K.indptr, indptr) and np.array_equal(K.indices, indices)
    assert np.max(np.abs(K.data - data)) <= 1e-12 * np.max(np.abs(data))
    value, gradient = rng.standard_normal((E, Q, comp)), rng.standard_normal((E, Q, comp, 3))
    got, _ = sk.NativeLinearForm(basis).assemble(value=value, gradient=gradient)
    want = O.linear_assemble(ob, value=value, gradient=gradient)
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("precision", ["fp64", "split_fp32"])
@pytest.mark.parametrize("E", [127, 128, 129, 256, 257])
def test_n1_at_tile_ends(E, precision):
    m = _mesh(E, False)
    rng = np.random.default_rng(5)
    mass, curl = rng.uniform(0.5, 2.0, (2, E, 1))
    K = sk.TetN1Assembler(sk.AffineTetN1Basis(m)).assemble_maxwell(mass_coefficient=mass, curl_coefficient=curl,
                                                                  precision=precision)
    data, indptr, indices = O.n1_assemble_maxwell(O.make_n1_basis(m.p, m.t, 2), mass, curl)
    assert np.array_equal(K.indptr, indptr) and np.array_equal(K.indices, indices)
    assert np.max(np.abs(K.data - data)) <= BOUND[precision] * np.max(np.abs(data))


@pytest.fixture(scope="module")
def large():
    """27^3 x 6 = 118,098 P2 elements: 923 tiles, more than 2,000 windows, more than 2^22 values (a host result is
    copied chunk by chunk); FP64 values of a coefficient far outside the FP32 range."""
    m = sk.MeshTet2.from_mesh(sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, 28),) * 3))
    basis = sk.Basis(m, sk.ElementVector(sk.ElementTetP2(), dim=1), quadrature=O.tet_quadrature_p1())
    E, Q = basis._coefficient_shape
    A = _tensors(E, (127, 128, E // 2, E - 1))
    form = NativeTensorForm(basis)
    assert form.pattern.nnz >= 1 << 22
    values = {}
    for scale in (1.0, 1e40):
        pub = np.broadcast_to(np.moveaxis(scale * A, 0, -1)[..., None], (3, 3, E, Q))
        values[scale] = pub, form.assemble(pub, copy=False).data.copy()
    return form, values


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("precision", ["fp64_emulated", "split_fp32"])
def test_fp64_takes_over_out_of_range(large, precision, host):
    form, values = large
    for scale in (1e40, 1.0, 1e40):  # the range flag of one call does not reach the next
        pub, want = values[scale]
        if host:
            got = form.assemble(pub, precision, copy=False).data
        else:
            got = form.assemble_device(pub, precision).cpu().numpy()[: form.pattern.nnz]
        if scale == 1.0:
            assert not np.array_equal(got, want)  # the FP32-pair passes
            assert np.max(np.abs(got - want)) <= BOUND[precision] * np.max(np.abs(want))
        else:
            assert np.array_equal(got, want)


def test_n1_fp64_takes_over_out_of_range():
    m = sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, 25),) * 3)  # 82,944 elements, 648 tiles
    form = sk.TetN1Assembler(sk.AffineTetN1Basis(m))
    nu = np.exp(np.random.default_rng(4).normal(0.0, 0.3, m.nelements))[:, None]
    for scale in (1e40, 1.0, 1e40):
        co = dict(mass_coefficient=scale, curl_coefficient=scale * nu)
        want = form.assemble_maxwell(**co).data.copy()
        got = form.assemble_maxwell(**co, precision="split_fp32").data
        if scale == 1.0:
            assert not np.array_equal(got, want)
            assert np.max(np.abs(got - want)) <= 1e-7 * np.max(np.abs(want))
        else:
            assert np.array_equal(got, want)
