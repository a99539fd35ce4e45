"""The point-surface builder's array form against its item-by-item form: the same points and normals bit
for bit, and what the loop refuses stays refused with the same error."""
import numpy as np
import pytest

from srsoriginal_b200.sr import sr

INF, NAN = float("inf"), float("nan")
RNG = np.random.default_rng(2)
LISTS = [
    (RNG.normal(size=(40, 2, 3)).tolist(), [0.1, 0.2, -0.3], [1, 2, 3], True),
    (RNG.normal(size=(3, 2, 3)).astype(np.float32), [0, 0, 1.0], None, False),
    ([[(1, 2, 3), (0, 0, 1)]], None, [0, 0, 1], False),
    ([], None, None, False),
    ([[[1, 2, 3], [0, 0, 0]]], None, None, False),
    ([[[1, 2], [0, 0, 1]]], None, None, False),
    ([[[1, 2, 3]]], None, None, False),
    ([[[1, 2, None], [0, 0, 1]]], None, None, False),
    ([[["1", "2", "3"], [0, 0, 1]]], None, None, False),
    ([[[INF, 0, 0], [0, 0, 1]]], [0.1, 0, 0], None, False),
    ([[[1, 2, 3], [0, NAN, 1]]], None, None, True),
    ([[[10 ** 30, 2, 3], [0, 0, True]]], None, None, False),
]


@pytest.mark.parametrize("case", range(len(LISTS)))
def test_surface_arrays_equal_the_loop(case, monkeypatch):
    def build():
        try:
            return sr._surface_3d(*LISTS[case])
        except Exception as e:  # noqa: BLE001  (compared below)
            return type(e), str(e)

    got = build()
    monkeypatch.setattr(sr, "_surface_arrays", staticmethod(lambda *a: None))
    ref = build()
    if isinstance(ref[0], type):
        assert got == ref
    else:
        for a, b in zip(got, ref):
            assert a.shape == b.shape and a.dtype == b.dtype
            assert np.array_equal(a, b, equal_nan=True) and np.array_equal(np.signbit(a), np.signbit(b))
