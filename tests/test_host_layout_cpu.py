"""Host arrays as the library reads them: (..., 2, N) to C-contiguous (..., N, 2)."""
import numpy as np
import pytest

from fasttools2d_gb300.mex import _interleaved


@pytest.mark.parametrize("shape", [(2, 0), (2, 1), (2, 7), (3, 2, 5), (1, 2, 1)])
@pytest.mark.parametrize("form", ["c", "f", "step", "reversed", "transposed"])
def test_interleaved(shape, form):
    a = np.random.default_rng(1).standard_normal(shape)
    if form == "f":
        a = np.asfortranarray(a)
    elif form == "step":
        a = np.repeat(a, 2, axis=-1)[..., ::2]
    elif form == "reversed":
        a = a[..., ::-1]
    elif form == "transposed":
        a = np.swapaxes(np.ascontiguousarray(np.swapaxes(a, -1, -2)), -1, -2)
    t = _interleaved(a)
    assert t.flags.c_contiguous and t.dtype == np.float64
    assert np.array_equal(t, np.ascontiguousarray(np.swapaxes(a, -1, -2)))
    if form == "transposed" and a.size:
        assert np.shares_memory(t, a)
