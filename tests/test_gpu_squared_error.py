"""A squared error's mean and gradient: the sums that the square leaves, and gradients kept as a factor of the saved
difference, against NumPy in double precision and against the op-by-op path; sizes around a CTA's chunk."""

import numpy as np
import pytest

from tests.util import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(), (1,), (5,), (3, 7), (1023, 4), (64, 64), (4097,), (129, 513), (1200, 1027)], ids=str)
def test_mean_and_sum_of_squares(nt, shape):
    x = np.asarray(np.random.default_rng(1).standard_normal(shape), np.float32)
    t = nt.Tensor.from_numpy(x, "cuda") if shape else nt.Tensor(float(x)).to("cuda")
    square = t ** 2
    assert np.array_equal(bits(square.numpy()), bits(x * x))
    want = np.square(x.astype(np.float64))
    for _ in range(2):  # the second time they are copies of what the square left
        assert abs(float(nt.mean(square).numpy()) - want.mean()) <= 2e-6 * want.mean()
        assert abs(float(nt.sum(square).numpy()) - want.sum()) <= 2e-6 * want.sum()
    square = t ** 2
    with nt.no_grad():
        square += 1.0  # the sums that came with it are out of date
    assert abs(float(nt.mean(square).numpy()) - (want + 1).mean()) <= 2e-6 * (want + 1).mean()


OPS = {"add": lambda a, b: a + b, "mul": lambda a, b: a * b, "truediv": lambda a, b: a / b, "tanh": lambda a, b: a.tanh(),
       "sigmoid": lambda a, b: a.sigmoid(), "relu": lambda a, b: a.relu(), "exp": lambda a, b: a.exp(), "log": lambda a, b: a.log(),
       "sqrt": lambda a, b: a.sqrt(), "neg": lambda a, b: -a, "pow": lambda a, b: a ** 3.0, "matmul": lambda a, b: a @ b.T,
       "transposed": lambda a, b: a.T * b.T, "sum": lambda a, b: a.sum(axis=0), "max": lambda a, b: a.max(axis=1),
       "reshape": lambda a, b: a.reshape(a.numel), "twice": lambda a, b: a * a + b}


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("shape", [(5, 7), (64, 132), (1024, 1056)], ids=str)
def test_gradients_of_a_squared_error(nt, op, shape):
    rng = np.random.default_rng(2)
    a, b = (rng.uniform(0.5, 2, shape).astype(np.float32) for _ in range(2))
    got = []
    for k in (2, nt.Tensor(2.0).to("cuda")):  # a tensor exponent takes the classes' own path
        ta, tb = (nt.Tensor.from_numpy(v, "cuda", requires_grad=True) for v in (a, b))
        y = OPS[op](ta, tb)
        target = nt.Tensor.from_numpy(np.random.default_rng(3).standard_normal(y.shape).astype(np.float32), "cuda")
        nt.mean((y - target) ** k).backward()
        got.append([t.grad.numpy() for t in (ta, tb) if t.grad is not None])
    assert len(got[0]) == len(got[1])
    for g, h in zip(*got):
        assert np.array_equal(bits(g), bits(h)) if op != "matmul" else np.allclose(g, h, rtol=1e-5, atol=1e-9)


def test_a_leaf_under_the_square(nt):
    x = np.random.default_rng(4).standard_normal((33, 5)).astype(np.float32)
    t = nt.Tensor.from_numpy(x, "cuda", requires_grad=True)
    (t ** 2).mean().backward()
    assert np.array_equal(bits(t.grad.numpy()), bits(np.float32(np.float32(1) / np.float32(x.size) * 2) * x))


def test_the_same_elements_have_the_same_sums(nt):
    square = nt.Tensor.from_numpy(np.random.default_rng(5).standard_normal((1200, 1027)).astype(np.float32), "cuda") ** 2
    for f in (nt.mean, nt.sum):
        first = f(square)
        with nt.no_grad():
            kept = first.numpy().copy()
            first += 1.0  # the caller's own
        assert {float(f(square).numpy()) for _ in range(2)} == {float(kept)}


def put(t, values):
    values = np.ascontiguousarray(values, np.float32)
    t.storage.upload(values.ctypes.data, values.nbytes)


@pytest.mark.parametrize("f", ["mean", "sum"])
@pytest.mark.parametrize("square_inside", [True, False], ids=["square captured", "square before"])
@pytest.mark.parametrize("sum_inside", [True, False], ids=["sum captured", "sum after"])
def test_sums_of_a_square_and_a_graph_capture(nt, square_inside, sum_inside, f):
    """Replays follow new values, and an eager sum taken after one replay keeps its value through the next."""
    reduce = getattr(nt, f)
    a, b = (np.random.default_rng(s).standard_normal((64, 33)).astype(np.float32) for s in (6, 7))
    want = lambda v: np.float32(getattr(v.astype(np.float64), f)())  # noqa: E731
    x = nt.Tensor.from_numpy(a, "cuda")
    reduce(x ** 2), nt.sum(x)  # first-use set-up outside the capture
    square = None if square_inside else x ** 2
    total = None
    graph = nt._C.Graph()
    with graph.capture():
        if square_inside:
            square = x ** 2
        if sum_inside:
            total = reduce(square)
        z = x + 1.0  # a launch in any case
    graph.replay()
    if not sum_inside:
        total = reduce(square)
    assert np.isclose(total.numpy(), want(a * a), rtol=2e-6)
    put(x if square_inside else square, b if square_inside else b * b)
    graph.replay()
    assert np.isclose(total.numpy(), want(b * b if sum_inside else a * a), rtol=2e-6)
    assert np.isclose(reduce(square).numpy(), want(b * b), rtol=2e-6)
    graph.close()
    del z


def test_a_written_gradient_does_not_keep_the_difference(nt):
    n = 1 << 20
    a, b = (nt.Tensor.from_numpy(np.full(n, v, np.float32), "cuda", requires_grad=True) for v in (1, 2))
    target = nt.Tensor.from_numpy(np.zeros(n, np.float32), "cuda")
    before = nt.cuda.memory_stats()["bytes_in_use"]
    nt.mean(((a + b) - target) ** 2).backward()
    assert nt.cuda.memory_stats()["bytes_in_use"] - before <= 4 * n  # one gradient, which both leaves have
    assert (a.grad.numpy() == np.float32(6 / n)).all() and (b.grad.numpy() == np.float32(6 / n)).all()


@pytest.mark.parametrize("kind", ["backward", "hook", "error"])
def test_a_waiting_gradient_survives_python_code(nt, kind):
    """A custom op's backward, or a leaf's hook, overwrites the difference of which a gradient still waiting in the sweep is a
    factor; and a sweep that ends in an exception leaves values behind, not factors."""
    from nanotorch_b200 import autograd

    class Scrub(autograd.Function):
        """A sum whose backward zeroes its input and passes no gradient on."""

        def forward(self, d):
            self.d = d
            return nt.Tensor._new_contiguous(nt._C.sum(d._C_view, (0,), d.dtype), ())

        def backward(self, g):
            scrub(self.d)
            return (None,)

    def scrub(d):
        nt._C.mul_inplace(d._C_view, nt.Tensor.from_numpy(np.zeros(d.shape, np.float32), "cuda")._C_view)
        if kind == "error":
            raise ArithmeticError

    x = np.arange(1, 9, dtype=np.float32)
    kept = 0
    for square_first in (True, False):  # one of the two has the square's gradient waiting when the difference is zeroed
        t, leaf = (nt.Tensor.from_numpy(x, "cuda", requires_grad=True) for _ in range(2))
        d = t - 0.5
        other = (leaf * 1.0).sum() if kind == "hook" else Scrub.apply(d)
        if kind == "hook":
            autograd.leaf_grad_hooks[id(leaf)] = lambda p, d=d: scrub(d)
        square = (d ** 2).sum()
        try:
            (square + other if square_first else other + square).backward()
        except RuntimeError as refused:  # zeroed before the square's backward, which notices
            assert "modified inplace" in str(refused)
            continue
        except ArithmeticError:
            assert kind == "error"
        finally:
            autograd.leaf_grad_hooks.pop(id(leaf), None)
        got = d.grad if kind == "error" else t.grad
        if got is not None:
            assert np.array_equal(got.numpy(), 2 * (x - 0.5))
            kept += 1
    assert kept == 1
