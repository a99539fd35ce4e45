"""Point lists whose array form numpy refuses, or would read otherwise than number by number: the loop takes them."""
import numpy as np
import pytest

from srsoriginal_b200.sr import sr


def _tensors():
    import torch

    p = torch.tensor([[1.0, 2.0, 30.0], [0.0, 3.0, 29.0]], dtype=torch.float64, requires_grad=True)
    n = torch.tensor([[0.0, 0.0, 1.0], [0.0, 1.0, 1.0]], dtype=torch.float64)
    return torch.stack([p, n], dim=1), [[p[k], n[k]] for k in range(2)], [[list(p[k]), n[k]] for k in range(2)]


class NoArray(list):
    """A list that numpy cannot take."""

    def __array__(self, *args, **kwargs):
        raise RuntimeError("not an array")


MASKED = np.ma.array([[[1.0, 2.0, 30.0], [0.0, 0.0, 1.0]], [[0.0, 3.0, 29.0], [0.0, 1.0, 1.0]]])
MASKED[1, 0, 0] = np.ma.masked


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("points", [
    lambda: _tensors()[0], lambda: _tensors()[1], lambda: _tensors()[2],
    lambda: NoArray([[[1.0, 2.0, 30.0], [0.0, 0.0, 1.0]]]), lambda: MASKED,
], ids=["tensor", "tensors", "scalars", "no_array", "masked"])
def test_what_the_loop_takes_is_taken(points, monkeypatch):
    got = sr._surface_3d(points(), [0.1, 0.2, -0.3], [1, 2, 3], True)
    monkeypatch.setattr(sr, "_surface_arrays", staticmethod(lambda *a: None))
    ref = sr._surface_3d(points(), [0.1, 0.2, -0.3], [1, 2, 3], True)
    for a, b in zip(got, ref):
        assert a.dtype == b.dtype and np.array_equal(a, b, equal_nan=True)
