"""Both gradients of a large product or quotient with transposed operands in one launch: same bits as the single-gradient
kernels, at ragged tile edges, with a leading dim, sliced operands, and below the size and alignment it takes."""

import numpy as np
import pytest

from tests.util import bits

pytestmark = pytest.mark.gpu

SHAPES = [(1100, 1004), (64, 16384), (16388, 64), (3, 520, 772), (2048, 1028), (1030, 1026), (100, 68)]


@pytest.mark.parametrize("which", ["x2", "x1", "g", "x1 x2"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_both_gradients_with_transposed_operands(nt, shape, which):
    rng = np.random.default_rng(3)

    def operand(name):
        v = rng.uniform(0.5, 2, shape[:-2] + (shape[-1], shape[-2] + 4)).astype(np.float32)
        if name not in which.split():
            v = np.ascontiguousarray(np.swapaxes(v[..., 4:], -1, -2))
            return nt.Tensor.from_numpy(v, "cuda"), v
        t = nt.Tensor.from_numpy(v, "cuda")[..., 4:]
        return nt.transpose(t, len(shape) - 2, len(shape) - 1), np.swapaxes(v[..., 4:], -1, -2)

    (g, hg), (x1, h1), (x2, h2) = (operand(k) for k in ("g", "x1", "x2"))
    C = nt._C
    for t in (x1, x2):
        t.enable_grad()
    for op in ("mul", "div"):
        got = []
        for on in (True, False):
            C.set_transposed_tile_pipeline(on)
            try:
                y = x1 * x2 if op == "mul" else x1 / x2
                (y * g).sum().backward()  # g itself is the quotient's gradient
                got.append([x1.grad.numpy(), x2.grad.numpy()])
            finally:
                C.set_transposed_tile_pipeline(True)
            x1.zero_grad()
            x2.zero_grad()
        for p, q in zip(*got):
            assert np.array_equal(bits(p), bits(q))
        assert np.array_equal(bits(got[0][0]), bits(h2 * hg if op == "mul" else hg / h2))
        if op == "mul":
            assert np.array_equal(bits(got[0][1]), bits(h1 * hg))
        else:
            assert np.allclose(got[0][1], -h1 / (h2.astype(np.float64) ** 2) * hg, rtol=2e-6)
