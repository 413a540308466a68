"""Loads by rules of different sizes from two threads at once: the shared memory that one thread's rule needs is
not taken from it by the other's.  The results are those of single calls, bit for bit (sums in a fixed order)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sk = pytest.importorskip("skfemntv_gb300")


def test_rules_of_different_sizes_in_two_threads():
    m = sk.MeshTet2.from_mesh(sk.MeshTet.init_tensor(*(np.linspace(0.0, 1.0, 6),) * 3))
    forms = [sk.NativeLinearForm(sk.Basis(m, sk.ElementVector(sk.ElementTetP2(), dim=3), intorder=order))
             for order in (8, 6)]  # 216 and 125 points: tables of 53 and 31 KB
    want = [f.assemble(value=np.ones(3))[0] for f in forms]
    errors = []

    def run(k):
        try:
            for _ in range(300):
                assert np.array_equal(forms[k].assemble(value=np.ones(3))[0], want[k])
        except Exception as error:  # noqa: BLE001 - reported below, from the main thread
            errors.append(error)

    threads = [threading.Thread(target=run, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
