"""The exact FP32 kernels at the edges of their tiles, k-slices and splits, in every operand layout."""

import numpy as np
import pytest

from tests.util import bits

pytestmark = pytest.mark.gpu

# (M, K, N): below, at and past the 32 / 64 / 128 x 256 tiles and the 8 / 32-deep k-slices; few and many tiles
SHAPES = [(1, 1, 1), (1, 784, 256), (256, 256, 10), (31, 33, 65), (64, 32, 64), (65, 96, 31), (33, 1000, 7), (128, 8, 256),
          (129, 257, 260), (1024, 40, 1028), (1920, 72, 2570),
          (5, 700, 33), (8, 64, 70), (784, 256, 256)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "strided"])
def test_exact_products_are_sequential_sums(nt, shape, layout):
    M, K, N = shape
    rng = np.random.default_rng(M + K + N)
    a, b = rng.uniform(-1, 1, (M, K)).astype(np.float32), rng.uniform(-1, 1, (K, N)).astype(np.float32)
    if layout == "strided":  # neither dim has unit stride
        ta = nt.Tensor.from_numpy(np.repeat(a, 2, axis=1), "cuda")[:, ::2]
        tb = nt.Tensor.from_numpy(np.repeat(b, 2, axis=1), "cuda")[:, ::2]
    else:
        ta = nt.Tensor.from_numpy(np.ascontiguousarray(a.T), "cuda").T if layout == "tn" else nt.Tensor.from_numpy(a, "cuda")
        tb = nt.Tensor.from_numpy(np.ascontiguousarray(b.T), "cuda").T if layout == "nt" else nt.Tensor.from_numpy(b, "cuda")
    want64 = a.astype(np.float64) @ b.astype(np.float64)
    scale = np.abs(a.astype(np.float64)) @ np.abs(b.astype(np.float64))
    rows = np.unique(rng.integers(0, M, 16))
    chain = np.zeros((len(rows), N), np.float32)  # the reference's CPU loop: a rounded product, then a rounded sum
    for k in range(K):
        chain = chain + a[rows, k:k + 1] * b[k]
    keep = nt._C.get_matmul_tc_min_macs()
    try:
        for mode, min_macs in ((0, 1 << 62), (1, 1 << 62), (2, 1 << 62), (1, 1)):
            nt._C.set_matmul_mode(mode)
            nt._C.set_matmul_tc_min_macs(min_macs)  # the last: by expected time, k-splits among the choices
            got = (ta @ tb).numpy()
            assert np.abs(got - want64).max() <= 2e-6 * scale.max()
            assert np.array_equal(bits(got), bits((ta @ tb).numpy()))
            if mode == 2:
                assert np.array_equal(bits(got[rows]), bits(chain))
            if min_macs == 1:
                continue
            bias = nt.Tensor.from_numpy(rng.standard_normal(N).astype(np.float32), "cuda")
            fused = nt.Tensor._new_contiguous(nt._C.linear(ta._C_view, tb._C_view, bias._C_view), (M, N))
            assert np.array_equal(bits(fused.numpy()), bits((ta @ tb + bias).numpy()))
    finally:
        nt._C.set_matmul_mode(1)
        nt._C.set_matmul_tc_min_macs(keep)
