"""Dense matrices against a value per row (every operand order and position), and sums of short rows: extents around the
vectors and warps of the kernels, few and many rows, unaligned and strided rows."""

import numpy as np
import pytest

from tests.util import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 4), (5, 8), (33, 1000), (4097, 12), (3, 4100), (7, 5)], ids=str)
def test_a_value_per_row(nt, shape):
    rng = np.random.default_rng(0)
    a, r = rng.uniform(0.5, 2, shape).astype(np.float32), rng.uniform(0.5, 2, (shape[0], 1)).astype(np.float32)
    g = rng.uniform(0.5, 2, shape).astype(np.float32)
    ta, tr, tg = (nt.Tensor.from_numpy(v, "cuda") for v in (a, r, g))
    for got, want in ((ta - tr, a - r), (tr - ta, r - a), (ta / tr, a / r), (tr / ta, r / a), (tr * ta, r * a)):
        assert np.array_equal(bits(got.numpy()), bits(want))
    er = tr.expand(*shape)
    for x1, x2, n1, n2 in ((ta, er, a, r), (er, ta, r, a), (er, er, r, r)):
        got = nt.Tensor._new_contiguous(nt._C.div_backward_x2(tg._C_view, x1._C_view, x2._C_view), shape)
        assert np.array_equal(bits(got.numpy()), bits(-n1 / (n2 * n2) * g + np.zeros(shape, np.float32)))


@pytest.mark.parametrize("rows", [64, 65, 4096, 18944, 20001])
@pytest.mark.parametrize("length", [1, 3, 4, 127, 128, 260, 1000, 1023])
def test_short_rows(nt, rows, length):
    x = np.random.default_rng(1).standard_normal((rows, length + 3)).astype(np.float32)
    t = nt.Tensor.from_numpy(x, "cuda")
    for view, ref in ((t[:, :length], x[:, :length]), (t[:, 3:], x[:, 3:]), (t, x)):
        if ref.shape[1] >= 1024:
            continue
        want = ref.astype(np.float64).sum(axis=1)
        assert np.abs(view.sum(axis=1).numpy() - want).max() <= 1e-6 * np.abs(ref).astype(np.float64).sum(axis=1).max()
        assert np.array_equal(view.max(axis=1).numpy(), ref.max(axis=1)) and np.array_equal(view.min(axis=1).numpy(), ref.min(axis=1))
