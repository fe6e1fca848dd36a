"""Contiguous elementwise runs around the size at which a thread takes four vectors instead of one: bits of NumPy."""

import numpy as np
import pytest

from tests.util import bits

pytestmark = pytest.mark.gpu

LINE = 148 * 1024 * 4


@pytest.mark.parametrize("n", [4, 5, 1023, 1024, 1027, 65536, LINE - 1, LINE, LINE + 3, LINE + 4, LINE + 1029])
def test_runs_around_the_line(nt, n):
    a, b = np.random.default_rng(7).standard_normal((2, n)).astype(np.float32)
    ta, tb = nt.Tensor.from_numpy(a, "cuda"), nt.Tensor.from_numpy(b, "cuda")
    assert np.array_equal(bits((ta + tb).numpy()), bits(a + b))
    assert np.array_equal(bits((ta * tb).numpy()), bits(a * b))
    assert np.array_equal(bits(nt.relu(ta).numpy()), bits(np.maximum(a, 0)))
    ta *= tb
    assert np.array_equal(bits(ta.numpy()), bits(a * b))
