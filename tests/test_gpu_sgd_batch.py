"""The updates of a list of parameters have the bits of one update at a time: ragged sizes around a CTA's chunk, more
parameters than one launch takes, unaligned and strided ones, the same storage twice, planes kept current."""

import numpy as np
import pytest

from tests.util import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 0.25])
def test_many_updates_in_one_call(nt, scale):
    import nanotorch_b200.nn as nn

    rng = np.random.default_rng(0)
    shapes = [(1,), (3,), (255, 33), (2047,), (2048,), (2049,), (64, 64), (1024, 1025)] + [(17, i) for i in range(1, 24)]
    data = [(rng.standard_normal(s).astype(np.float32), rng.standard_normal(s).astype(np.float32)) for s in shapes]

    def build():
        params = []
        base = nt.Tensor.from_numpy(rng_base.copy(), "cuda")
        for d, g in data:
            p = nt.Tensor.from_numpy(d, "cuda", requires_grad=True)
            p._grad = nt.Tensor.from_numpy(g, "cuda")
            params.append(p)
        for view in (base[1:1025], base[1025:], base.reshape(2, 1024).T):  # unaligned, and the same storage again, strided
            view = view._alias()
            view.enable_grad()
            view._grad = nt.Tensor.from_numpy(np.ones(view.shape, np.float32), "cuda")
            params.append(view)
        return params, base

    rng_base = rng.standard_normal(2048).astype(np.float32)
    x = nt.Tensor.from_numpy(rng.standard_normal((128, 64)).astype(np.float32), "cuda")
    (many, base_m), (single, base_s) = build(), build()
    keep = nt._C.get_matmul_tc_min_macs()
    try:
        nt._C.set_matmul_tc_min_macs(0)  # the 64 x 64 parameter becomes an operand with planes
        before = (x @ many[6]).numpy(), (x @ single[6]).numpy()
        nn.GradientDescent(many, 0.1, scale).step()
        for p in single:
            nt._C.sgd_update(p._C_view, p.grad._C_view, 0.1, scale)
        after = (x @ many[6]).numpy(), (x @ single[6]).numpy()
    finally:
        nt._C.set_matmul_tc_min_macs(keep)
    assert np.array_equal(bits(before[0]), bits(before[1])) and np.array_equal(bits(after[0]), bits(after[1]))
    assert not np.array_equal(bits(before[0]), bits(after[0]))
    for p, q in zip(many, single):
        assert np.array_equal(bits(p.numpy()), bits(q.numpy())) and p.version == q.version
    assert np.array_equal(bits(base_m.numpy()), bits(base_s.numpy()))


@pytest.mark.parametrize("sizes", [(7, 7, 7), (5000, 5000, 5000), (1 << 21, 1 << 21, 1 << 21)], ids=str)
@pytest.mark.parametrize("order", [(0, 1, 2), (1, 0, 2), (2, 1, 0)], ids=str)
def test_gradients_that_are_parameters(nt, sizes, order):
    """Updates happen one after the other where a gradient is another parameter's storage: p1's gradient is p0, p2's is p1."""
    import nanotorch_b200.nn as nn

    n = sizes[0]
    p = [nt.Tensor.from_numpy(np.full(n, 8.0 * (i + 1), np.float32), "cuda", requires_grad=True) for i in range(3)]
    p[0]._grad = nt.Tensor.from_numpy(np.full(n, 2.0, np.float32), "cuda")
    p[1]._grad, p[2]._grad = (nt.Tensor._new_view(p[i].storage, (n,), (1,), 0) for i in (0, 1))
    want = [8.0, 16.0, 24.0]
    for i in order:
        want[i] -= 0.5 * (2.0 if i == 0 else want[i - 1])
    nn.GradientDescent([p[i] for i in order], lr=0.5).step()
    for got, w in zip(p, want):
        assert (got.numpy() == w).all()
