"""The binding's copy of large results by several threads: equal, independent, any length (CPU)."""
import numpy as np
import pytest


@pytest.mark.parametrize("n", [0, 5, (1 << 20) - 1, 3_000_001])
def test_copy(n):
    import fastbc_gpu as fg

    a = np.arange(n, dtype=np.float64)
    b = fg._copy(a)
    assert b.dtype == a.dtype and np.array_equal(a, b) and (n == 0 or not np.shares_memory(a, b))
