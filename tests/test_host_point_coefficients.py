"""Coefficients given per point are told from coefficients constant on each element without reading them whole,
except where only a few elements make the difference; the answer is that of the full comparison."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytest.importorskip("skfemntv_gb300")
from skfemntv_gb300.assembly import per_element  # noqa: E402

E, Q = 100_003, 11


def test_varying_coefficient_is_not_read_whole(monkeypatch):
    c = np.random.default_rng(0).uniform(0.5, 2.0, (E, Q))
    compared = []
    equal = np.array_equal
    monkeypatch.setattr(np, "array_equal", lambda a, b: compared.append(a.size) or equal(a, b))
    assert per_element(c, E, Q, "value") is None
    assert sum(compared) <= 256 * Q


@pytest.mark.parametrize("where", [0, 1, E // 2, E - 1])
@pytest.mark.parametrize("other", [2.5, np.nan, np.inf])
def test_one_varying_element_is_found(where, other):
    c = np.repeat(np.random.default_rng(1).uniform(0.5, 2.0, (E, 1)), Q, axis=1)
    assert np.array_equal(per_element(c, E, Q, "value"), c[:, 0])
    c[where, Q - 1] = other
    assert per_element(c, E, Q, "value") is None


@pytest.mark.parametrize("shape", [(1, 4), (2, 2), (63, 3), (64, 1), (65, 4), (0, 4)])
def test_small_and_broadcast(shape):
    e, q = shape
    rows = np.arange(e, dtype=float)
    full = np.repeat(rows[:, None], q, axis=1)
    for c in (full, full[::-1][::-1], np.asfortranarray(full), rows[:, None]):
        assert np.array_equal(per_element(c, e, q, "value"), rows)
    assert np.ndim(per_element(1.5, e, q, "value")) == 0
    assert np.array_equal(per_element(np.full((1, q), 2.0), e, q, "value"), np.full(e, 2.0))
    inf = np.full((e, q), np.inf)
    assert np.array_equal(per_element(inf, e, q, "value"), np.full(e, np.inf))
    if e and q > 1:
        assert per_element(np.full((e, q), np.nan), e, q, "value") is None
