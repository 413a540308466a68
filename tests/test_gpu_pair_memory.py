"""Scratch of the precision modes: the FP32-pair calls hold no more device memory than the FP64 call, whose
matrices they need as well when a value leaves the FP32 range.

Measured as the high watermark of the stream-ordered allocations (the process's default memory pool) over one
call.  Tolerance: 64 KiB, for the scale exponent and the range flag and the pool's rounding of small blocks."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
sk = pytest.importorskip("skfemntv_gb300")
from skfemntv_gb300.assembly import NativeTensorForm  # noqa: E402

USED_CURRENT, USED_HIGH = 7, 8  # cudaMemPoolAttrUsedMemCurrent, cudaMemPoolAttrUsedMemHigh


def _pool():
    rt = ctypes.CDLL("libcudart.so.13")
    pool = ctypes.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), torch.cuda.current_device()) == 0
    return rt, pool


def _attribute(rt, pool, which):
    v = ctypes.c_uint64()
    assert rt.cudaMemPoolGetAttribute(pool, which, ctypes.byref(v)) == 0
    return v.value


def _peak(call):
    rt, pool = _pool()
    torch.cuda.synchronize()
    zero = ctypes.c_uint64(0)
    assert rt.cudaMemPoolSetAttribute(pool, USED_HIGH, ctypes.byref(zero)) == 0
    before = _attribute(rt, pool, USED_CURRENT)
    call()
    torch.cuda.synchronize()
    return _attribute(rt, pool, USED_HIGH) - before


@pytest.mark.parametrize("tensor", [False, True])
def test_fp32_pairs_take_no_more_scratch_than_fp64(tensor):
    m = sk.MeshTet2.from_mesh(sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, 13),) * 3))
    b = sk.Basis(m, sk.ElementVector(sk.ElementTetP2(), dim=1))
    E = m.nelements
    A = torch.eye(3, dtype=torch.float64, device="cuda")[:, :, None].expand(3, 3, E).contiguous()
    if tensor:
        form = NativeTensorForm(b)
        call = lambda p: form.assemble_device(None, precision=p, tensor_device=A)  # noqa: E731
    else:
        form = sk.NativeBilinearForm(b)
        call = lambda p: form.assemble_device(gradient=np.ones((E, 1)), precision=p)  # noqa: E731
    for p in ("fp64", "fp64_emulated", "split_fp32"):
        call(p)  # tables
    peak = {p: _peak(lambda: call(p)) for p in ("fp64", "fp64_emulated", "split_fp32")}
    triangles = 55 * 8 * E * (2 if tensor else 1)
    assert triangles <= peak["fp64"] <= triangles + 55 * 16 * 128 + (1 << 16) + E // 64
    for p in ("fp64_emulated", "split_fp32"):
        assert peak[p] <= peak["fp64"] + (1 << 16), peak
