"""Products and quotients with a value per row, and a row maximum whose input has a gradient already: the one-pass kernels'
gradients against double precision; ragged rows, few and many rows, short and long ones."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 5), (7, 3), (8, 128), (9, 1000), (200, 1023), (149, 1028), (160, 4099), (4737, 1024), (3, 50, 1000), (200, 5000), (148, 16384),
          (5, 70000), (149, 255), (512, 256), (513, 256), (2048, 1024), (2049, 1024), (2056, 257), (2057, 257), (4736, 1027), (4737, 1027), (4737, 4096)]


def close(got, want, scale):
    assert got.shape == want.shape
    assert np.all(np.abs(got - want) <= 2e-6 * scale + 1e-30)


@pytest.mark.parametrize("first", [False, True], ids=["second", "first"])
@pytest.mark.parametrize("op", ["mul", "div"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_gradients_with_a_value_per_row(nt, shape, op, first):
    rng = np.random.default_rng(5)
    full, rows = (rng.uniform(0.5, 2, s).astype(np.float32) for s in (shape, shape[:-1] + (1,)))
    target = rng.standard_normal(shape).astype(np.float32)
    a, b = (rows, full) if first else (full, rows)
    for squared in (False, True):  # a gradient that is a factor of another storage, and one that is not
        ta, tb = (nt.Tensor.from_numpy(v, "cuda", requires_grad=True) for v in (a, b))
        t = nt.Tensor.from_numpy(target, "cuda")
        y = ta * tb if op == "mul" else ta / tb
        (((y - t) ** 2).mean() if squared else (y * t).sum()).backward()
        da, db = a.astype(np.float64), b.astype(np.float64)
        y64 = da * db if op == "mul" else da / db
        g = 2.0 * (y64 - target) / y64.size if squared else target.astype(np.float64)
        g1, g2 = (db * g, da * g) if op == "mul" else (g / db, -da / db**2 * g)
        s1, s2 = np.abs(g1) + 1.0 / y64.size, np.abs(g2) + 1.0 / y64.size
        if not squared:
            s1, s2 = np.abs(g1), np.abs(g2)
        if first:
            g1, s1 = g1.sum(-1, keepdims=True), 8 * s1.sum(-1, keepdims=True)
            s2 = 8 * s2
        else:
            g2, s2 = g2.sum(-1, keepdims=True), 8 * s2.sum(-1, keepdims=True)
            s1 = 8 * s1
        close(ta.grad.numpy(), g1, s1)
        close(tb.grad.numpy(), g2, s2)


@pytest.mark.parametrize("shape", [(3, 5), (148, 4), (150, 1000), (4096, 1024), (200, 1028), (160, 16384), (149, 16388), (200, 1001)], ids=str)
def test_row_maximum_adds_to_the_gradient_of_its_input(nt, shape):
    rng = np.random.default_rng(6)
    x = rng.standard_normal(shape).astype(np.float32)
    x[0, :2] = 9.0  # a tie: no gradient there
    w = rng.standard_normal(shape).astype(np.float32)
    t = nt.Tensor.from_numpy(x, "cuda", requires_grad=True)
    ((t - t.max(axis=1, keepdim=True)) * nt.Tensor.from_numpy(w, "cuda")).sum().backward()
    mask = (x == x.max(1, keepdims=True)).astype(np.float64)
    mask[mask.sum(1) != 1] = 0
    scale = np.abs(w) + mask * np.abs(w).sum(1, keepdims=True)
    close(t.grad.numpy(), w - mask * w.astype(np.float64).sum(1, keepdims=True), scale)
