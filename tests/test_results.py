"""Arrays for results (mgpicola._result): writable FP32 arrays of the asked shape on either
side of the size from which they have pages of their own, and the exception of
numpy's own arrays when there is no memory."""
import numpy as np
import pytest

import mgpicola as M


@pytest.mark.parametrize("shape", [(0, 3), (5, 3), ((1 << 20) - 1,), (1 << 20,), (400000, 3)])
def test_result_arrays(shape):
    a = M._result(shape)
    assert a.shape == shape and a.dtype == np.float32 and a.flags.writeable and a.flags.c_contiguous
    a[...] = 1.0
    assert a.sum(dtype=np.float64) == a.size


@pytest.mark.parametrize("shape", [(1 << 45, 3), (1 << 62,)])
def test_too_large_result_raises_memory_error(shape):
    with pytest.raises(MemoryError):
        M._result(shape)
