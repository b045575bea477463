"""The coordinates of the KL tables: one float32 division gives the float32
rounding of the reference's float64 expression (K/ocean_noise.cu:826)."""
import numpy as np
import pytest


@pytest.mark.parametrize("n", [1, 2, 3, 7, 60, 127, 300, 301, 511, 512, 1500, 4097, 65537, 3 * 2 ** 20 + 1, 2 ** 23 - 1])
def test_float_division_rounds_like_double(n):
    t = np.arange(n + 2) if n < 10 ** 5 else np.unique(np.linspace(0, n + 1, 100003).astype(np.int64))
    double = ((t + 1 + 0.5 - 2) / n).astype(np.float32)
    single = (t.astype(np.float32) - np.float32(0.5)) / np.float32(n)
    assert single.dtype == np.float32 and np.array_equal(single, double)
