"""The native apply / backward sweep against the Python op classes they restate: same bits, forward and gradients.
A subclass of an op class is not the registered class, so it takes the Python forward and backward."""

import gc

import numpy as np
import pytest

from tests.util import bits

pytestmark = pytest.mark.gpu

CASES = [
    ("AddOp", ((5, 7), (5, 7))), ("AddOp", ((5, 7), (7,))), ("SubOp", ((5, 1), (1, 7))), ("MulOp", ((4, 8), (4, 8))),
    ("MulOp", ((3, 5, 7), (5, 1))), ("TrueDivOp", ((4, 8), (4, 8))), ("TrueDivOp", ((5, 7), (7,))),
    ("MatmulOp", ((9, 17), (17, 5))), ("MatmulOp", ((3, 9, 17), (3, 17, 5))), ("LinearOp", ((9, 17), (17, 5), (5,))),
    *[(name, ((6, 11),)) for name in ("NegOp", "ExpOp", "LogOp", "SqrtOp", "TanhOp", "SigmoidOp", "ReluOp", "SumOp",
                                      "MeanOp", "MaxOp", "MinOp", "TOp")],
    ("PowOp", ((6, 11),), 3), ("PowOp", ((6, 11),), -1.5), ("SumOp", ((6, 11),), (0,), True), ("MeanOp", ((6, 11),), -1),
    ("MaxOp", ((2, 3, 4),), 1, True), ("MinOp", ((6, 11),), 0), ("ReshapeOp", ((6, 4),), 3, 8),
    ("ExpandOp", ((6, 1),), 2, 6, 5), ("TransposeOp", ((2, 3, 4),), 0, -1),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-{'x'.join(map(str, c[1]))}-{c[2:]}")
def test_native_path_has_the_bits_of_the_op_classes(nt, case):
    name, shapes, extra = case[0], case[1], case[2:]
    native = getattr(__import__("nanotorch_b200.autograd", fromlist=[name]), name)
    python = type(name + "Python", (native,), {})
    rng = np.random.default_rng(3)
    data = [rng.uniform(0.5, 2, s).astype(np.float32) for s in shapes]
    got = []
    for cls in (native, python):
        leaves = [nt.Tensor.from_numpy(d, "cuda", requires_grad=True) for d in data]
        y = cls.apply(*leaves, *extra)
        w = nt.Tensor.from_numpy(np.random.default_rng(4).standard_normal(y.shape).astype(np.float32), "cuda")
        assert type(y.grad_fn) is cls and y.grad_fn.needs_input_grad[:len(leaves)] == (True,) * len(leaves)
        (y * w).sum().backward()
        got.append([y.numpy()] + [t.grad.numpy() for t in leaves])
    for a, b in zip(*got):
        assert a.shape == b.shape and np.array_equal(bits(a), bits(b))


@pytest.mark.parametrize("shapes", [((64, 7), (1, 7)), ((128, 64), (128, 1)), ((4, 4096), (4, 1)), ((512, 2048), (1, 2048)),
                                    ((2, 3, 4), (1, 3, 1)), ((6, 4), (4,)), ((2, 4), (2, 4))], ids=str)
def test_gradients_that_cancel_are_the_same_zero(nt, shapes):
    """The subtrahend's gradient is a sum of negated values: +0 where they cancel, on either path."""
    from nanotorch_b200.autograd import SubOp

    w = np.random.default_rng(5).integers(1, 9, shapes[0]).astype(np.float32)
    pad = (1,) * (len(shapes[0]) - len(shapes[1])) + shapes[1]
    for axis in [d for d, n in enumerate(pad) if n == 1 and shapes[0][d] % 2 == 0][:1]:  # w, -w, w, -w ... along a summed axis
        w = np.take(w, np.arange(shapes[0][axis]) // 2 * 2, axis) * np.where(np.arange(shapes[0][axis]) % 2, -1, 1).reshape(
            [-1 if d == axis else 1 for d in range(w.ndim)]).astype(np.float32)
    got = []
    for cls in (SubOp, type("SubOpPython", (SubOp,), {})):
        x1, x2 = (nt.Tensor.from_numpy(np.ones(s, np.float32), "cuda", requires_grad=True) for s in shapes)
        (cls.apply(x1, x2) * nt.Tensor.from_numpy(w, "cuda")).sum().backward()
        got.append(x2.grad.numpy())
    assert got[0].shape == got[1].shape == shapes[1] and np.array_equal(bits(got[0]), bits(got[1]))
    assert shapes[0] == shapes[1] or not got[0].any()


def test_results_are_freed_without_the_cycle_collector(nt):
    """A node that saves its own result must not keep it alive: memory comes back by reference count alone."""
    x = nt.Tensor.from_numpy(np.ones((64, 64), np.float32), "cuda", requires_grad=True)
    nt.tanh(x).max(axis=0).exp().sum().backward()
    x.zero_grad()
    gc.collect()
    gc.disable()
    try:
        before = nt.cuda.memory_stats()["bytes_in_use"]
        for _ in range(3):
            nt.tanh(x).max(axis=0).exp().sum().backward()
            x.zero_grad()
        assert nt.cuda.memory_stats()["bytes_in_use"] == before
    finally:
        gc.enable()


def test_saved_tensor_modified_in_place_is_refused(nt):
    x = nt.Tensor.from_numpy(np.ones((4, 4), np.float32), "cuda", requires_grad=True)
    y = x * 2
    z = y * y
    with nt.no_grad():
        y += 1
    with pytest.raises(RuntimeError, match="modified inplace"):
        z.sum().backward()


@pytest.mark.parametrize("axis", [2 ** 70, -2 ** 70, (0, 2 ** 70)], ids=str)
@pytest.mark.parametrize("op", ["sum", "mean", "max"])
def test_an_axis_beyond_64_bits_is_an_index_error(nt, op, axis):
    x = nt.Tensor.from_numpy(np.ones((2, 3), np.float32), "cuda")
    with pytest.raises(IndexError):
        getattr(x, op)(axis=axis)


@pytest.mark.parametrize("made_of", [3, 3.0, True], ids=str)
def test_a_scalar_written_in_place_is_not_its_first_value(nt, made_of):
    """A tensor made of a Python number takes part with that number only until it is written to, under whatever name."""
    x = nt.Tensor.from_numpy(np.array([1.0, 2.0], np.float32), "cuda", requires_grad=True)
    for write in ("add", "alias", "upload"):
        t = nt.Tensor(made_of, device="cuda")
        assert np.array_equal((x * t).numpy(), [made_of, 2 * made_of]) and np.array_equal((x ** t).numpy(), [1, 2 ** made_of])
        if made_of is True:
            continue
        with nt.no_grad():
            if write == "add":
                nt.add(t, 2, out=t)
            elif write == "alias":
                t._alias().__iadd__(2)
            else:
                new = np.array(t.numpy() + 2, t.numpy().dtype)
                t.storage.upload(new.ctypes.data, new.nbytes)
        y = x * t
        assert np.array_equal(y.numpy(), [5, 10]) and np.array_equal((x ** t).numpy(), [1, 32]) and np.array_equal((t - x).numpy(), [4, 3])
        x.zero_grad()
        y.sum().backward()
        assert np.array_equal(x.grad.numpy(), [5, 5])


def test_a_constant_is_written_before_another_stream_uses_it(nt):
    """An upload on the copy stream into a value that had no memory yet comes after the value's own fill, however busy the
    compute stream is; a leaf's own seed is in memory."""
    import ctypes

    big = nt.Tensor.from_numpy(np.ones((4096, 4096), np.float32), "cuda")
    host = np.array([7.0], np.float32)
    with nt.no_grad():
        big @ big
        nt.cuda.sync()
        for _ in range(5):
            s = nt._C.constant(3.0, nt.float32)
            for _ in range(3):
                big @ big
            nt._C._check(nt._C._lib.nt_storage_upload_async(ctypes.c_void_p(s._h), ctypes.c_void_p(host.ctypes.data), ctypes.c_int64(4)))
            nt._C._check(nt._C._lib.nt_upload_fence())
            assert nt.Tensor._new_contiguous(s, ()).numpy() == 7.0
    leaf = nt.Tensor.from_numpy(np.array([2.0], np.float32), "cuda", requires_grad=True)
    used = nt.cuda.memory_stats()["bytes_in_use"]
    leaf.backward()
    assert nt.cuda.memory_stats()["bytes_in_use"] > used and leaf.grad.numpy() == 1.0


def test_an_uploads_address_is_handed_out_behind_its_copy(nt):
    """A reader on another stream that goes through the storage's address finds the uploaded values while the library's own
    stream is still busy: before the first look at the address, and for uploads after it."""
    torch = pytest.importorskip("torch")

    class Seen:
        def __init__(self, t):
            self.__cuda_array_interface__ = {"shape": t.shape, "typestr": "<f4", "version": 2, "data": (t.storage.data_ptr, False)}

    big = nt.Tensor.from_numpy(np.ones((4096, 4096), np.float32), "cuda")
    side = torch.cuda.Stream()
    nt.Tensor.from_numpy(np.zeros(100, np.float32), "cuda")
    with nt.no_grad():
        big @ big
        nt.cuda.sync()
        for value in (5.0, 6.0):
            for _ in range(20):
                big @ big
            t = nt.Tensor.from_numpy(np.full(100, value, np.float32), "cuda")
            with torch.cuda.stream(side):
                seen = torch.as_tensor(Seen(t), device="cuda")
                assert (seen.clone().cpu() == value).all()
            again = np.full(100, -value, np.float32)
            for _ in range(20):
                big @ big
            t.storage.upload(again.ctypes.data, again.nbytes)
            with torch.cuda.stream(side):
                assert (seen.clone().cpu() == -value).all()


def test_a_wait_that_ran_out_beside_another_threads_sync_is_reported(nt):
    """A kernel launched while another thread is inside a synchronising call is not covered by that call's look at the error
    flag: whichever call comes behind the kernel reports that its wait ran out."""
    import threading
    import time

    big = nt.Tensor.from_numpy(np.ones((4096, 4096), np.float32), "cuda")
    reports = []

    def sync():
        try:
            nt.cuda.sync()
        except RuntimeError as e:
            reports.append(str(e))

    before = nt._C.get_wait_limit_clocks()
    with nt.no_grad():
        big @ big
        nt.cuda.sync()
        for _ in range(60):
            big @ big
        thread = threading.Thread(target=sync)
        thread.start()
        time.sleep(0.005)
        nt._C.set_wait_limit_clocks(500_000_000)  # a quarter of a second
        try:
            nt._C.wait_probe()
        finally:
            nt._C.set_wait_limit_clocks(before)
        thread.join()
        sync()
    assert len(reports) == 1 and "code 5" in reports[0]
    sync()
    assert len(reports) == 1


def test_captures_begin_while_another_thread_makes_constants(nt):
    """The start of a capture gives the constants there are their memory, while another thread makes and drops some."""
    import threading

    x = nt.Tensor.from_numpy(np.ones(8, np.float32), "cuda")
    stop = False

    def churn():
        held = []
        while not stop:
            held.append(nt._C.constant(2.0, nt.float32))
            if len(held) > 5:
                held.clear()

    thread = threading.Thread(target=churn)
    thread.start()
    try:
        mine = nt._C.constant(3.0, nt.float32)
        for _ in range(100):
            graph = nt._C.Graph()
            with graph.capture():
                y = x * 2.0
            graph.replay()
            assert (y.numpy() == 2.0).all()
            graph.close()
    finally:
        stop = True
        thread.join()
    assert nt.Tensor._new_contiguous(mine, ()).numpy() == 3.0


def test_other_threads_run_while_a_launch_waits(nt):
    """With the stream's launch queue full a launch waits for the GPU, without the interpreter lock: another thread gets all
    of the processor that it asks for (half of it when the lock is held)."""
    import threading
    import time

    a, b = (nt.Tensor.from_numpy(np.ones(s, np.float32), "cuda") for s in ((8192, 1024), (1024, 4096)))
    used, stop = [], False

    def busy():
        start = time.thread_time()
        while not stop:
            pass
        used.append(time.thread_time() - start)

    nt._C.set_matmul_mode(nt._C.MATMUL_EXACT_FP32)  # 1.3 ms each
    try:
        with nt.no_grad():
            a @ b
            nt.cuda.sync()
            for _ in range(1030):  # the queue takes 1024
                a @ b
            thread = threading.Thread(target=busy)
            start = time.perf_counter()
            thread.start()
            while time.perf_counter() - start < 0.5:
                a @ b
            stop = True
            thread.join()
            wall = time.perf_counter() - start
    finally:
        nt._C.set_matmul_mode(nt._C.MATMUL_3XTF32)
        nt.cuda.sync()
    assert used[0] > 0.75 * wall


def test_threads_with_graphs_of_their_own(nt):
    """Forward and backward passes of several threads at once, each with its own input and all with one shared leaf: every
    pass is recorded although another thread's sweep is running, and no contribution to the shared gradient is lost."""
    import threading

    threads, passes = 4, 50
    shared = nt.Tensor.from_numpy(np.full(64, 2.0, np.float32), "cuda", requires_grad=True)
    failures = []

    def work(k):
        try:
            for _ in range(passes):
                x = nt.Tensor.from_numpy(np.full((8, 64), float(k), np.float32), "cuda", requires_grad=True)
                (x * shared).sum().backward()
                if not (x.grad.numpy() == 2.0).all():
                    failures.append(k)
        except Exception as e:  # noqa: BLE001
            failures.append(e)

    pool = [threading.Thread(target=work, args=(k,)) for k in range(1, threads + 1)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not failures
    assert (shared.grad.numpy() == 8.0 * passes * sum(range(1, threads + 1))).all()
