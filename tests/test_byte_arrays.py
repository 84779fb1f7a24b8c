"""The bytes handed to the library for a 0/1 array: every dtype and layout gives
the bytes of x != 0, and arrays that hold them already are not copied."""
import numpy as np
import pytest

from cusna_gb300.sim import _u8


@pytest.mark.parametrize("dtype", [np.bool_, np.uint8, np.int8, np.int64, np.float64])
@pytest.mark.parametrize("shape", [(0, 3, 3), (3, 3), (2, 5, 5)])
def test_bytes_of_every_dtype_and_layout(dtype, shape):
    x = (np.arange(np.prod(shape)).reshape(shape) % 3).astype(dtype)
    for v in (x, x.swapaxes(-1, -2), x[..., ::-1], (x != 0).astype(dtype)):
        got = _u8(v)
        assert got.dtype == np.uint8 and got.flags.c_contiguous
        np.testing.assert_array_equal(got, (v != 0).astype(np.uint8))
    for v in ((x != 0).astype(np.uint8), x != 0):
        assert v.size == 0 or np.shares_memory(_u8(v), v)
    assert _u8(None) is None
