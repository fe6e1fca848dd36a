"""`_C`: the native-module surface of nanotorch, bound to libnt_b200.so through its C ABI.

Same names, argument meaning and exception classes as the reference's pybind11 module
(src/cpp/_C.cpp:12-24, typed in src/nanotorch/_C.pyi:1-136): ``Dtype``, ``Device``, ``Storage``,
``TensorView`` and the free functions that take views and return a fresh ``Storage``.  The extra
entry points of include/nt_b200.h (fused backward kernels, SGD update, data-parallel exchange,
matmul mode) are exposed under the same module.  Storages, views and the ops themselves are bound natively
(csrc/engine); what is called once in a while goes through ctypes.

There is no fallback: if the shared library is missing the import fails, and every compute call
on a machine without a GPU raises RuntimeError.
"""

from __future__ import annotations

import ctypes as C
import enum
from pathlib import Path
from typing import Sequence

_LIB_PATH = Path(__file__).resolve().parent / "lib" / "libnt_b200.so"
if not _LIB_PATH.exists():
    raise ImportError(
        f"{_LIB_PATH} is missing: build it with `python nanotorch_b200/build.py` "
        "(there is no CPU or PyTorch fallback for the op kernels)."
    )
_lib = C.CDLL(str(_LIB_PATH))

from . import _engine  # noqa: E402  (links against the library loaded above)

NT_MAX_DIMS = 8


class Dtype(enum.IntEnum):
    """Data storage types; the order is the promotion order (src/cpp/dtype.h:21)."""

    Bool = 0
    Int32 = 1
    Int64 = 2
    Float32 = 3
    Float64 = 4

    def __str__(self) -> str:
        return f"Dtype.{self.name}"

    def __bool__(self) -> bool:
        # a pybind11 enum value is always truthy; the reference's Python layer relies on it
        # (`auto_dtype or Dtype.Float32`, src/nanotorch/core.py:620), and Bool has the value 0
        return True


class Device(enum.Enum):
    """Data storage devices (src/cpp/allocator.h:10)."""

    Cpu = 0
    Cuda = 1


_ITEMSIZE = {Dtype.Bool: 1, Dtype.Int32: 4, Dtype.Int64: 8, Dtype.Float32: 4, Dtype.Float64: 8}
_CTYPE = {
    Dtype.Bool: C.c_bool,
    Dtype.Int32: C.c_int32,
    Dtype.Int64: C.c_int64,
    Dtype.Float32: C.c_float,
    Dtype.Float64: C.c_double,
}


_FORMAT = {Dtype.Bool: "?", Dtype.Int32: "i", Dtype.Int64: "q", Dtype.Float32: "f", Dtype.Float64: "d"}


class _View(C.Structure):
    _fields_ = [
        ("storage", C.c_void_p),
        ("ndim", C.c_int32),
        ("shape", C.c_int64 * NT_MAX_DIMS),
        ("strides", C.c_int64 * NT_MAX_DIMS),
        ("offset", C.c_int64),
    ]


class _Scalar(C.Structure):
    _fields_ = [("kind", C.c_int32), ("i", C.c_int64), ("d", C.c_double)]


_lib.nt_last_error.restype = C.c_char_p
_lib.nt_storage_size.restype = C.c_int64
_lib.nt_storage_itemsize.restype = C.c_int64
_lib.nt_storage_version.restype = C.c_uint64
_lib.nt_storage_data.restype = C.c_void_p
_lib.nt_stream.restype = C.c_void_p
for _name in (
    "nt_storage_size", "nt_storage_itemsize", "nt_storage_dtype", "nt_storage_device",
    "nt_storage_version", "nt_storage_data", "nt_storage_retain", "nt_storage_release",
):
    getattr(_lib, _name).argtypes = [C.c_void_p]

_ERRORS = {1: RuntimeError, 2: ValueError, 3: TypeError, 4: IndexError}


def _check(status: int) -> None:
    if status != 0:
        msg = _lib.nt_last_error()
        raise _ERRORS.get(status, RuntimeError)(msg.decode() if msg else "unknown native error")


def _dtype(d) -> Dtype:
    if not isinstance(d, Dtype):
        raise TypeError(f"expected a Dtype, got {type(d).__name__}")
    return d


def _device(d) -> Device:
    if not isinstance(d, Device):
        raise TypeError(f"expected a Device, got {type(d).__name__}")
    return d


def _scalar(v) -> _Scalar:
    # bool before int: bool is an int subclass (src/cpp/storage.h:72-80)
    if isinstance(v, bool):
        return _Scalar(0, int(v), float(v))
    if isinstance(v, int):
        return _Scalar(1, v, float(v))
    if isinstance(v, float):
        return _Scalar(2, 0, v)
    raise TypeError("Unknown scalar type.")


class Storage(_engine.StorageBase):
    """Pointer to a 1D contiguous, typed memory segment (src/cpp/storage.h:34-66)."""

    __slots__ = ("__weakref__",)

    @staticmethod
    def from_iterable(values: Sequence, dtype: Dtype, device: Device) -> "Storage":
        dtype = _dtype(dtype)
        device = _device(device)
        n = len(values)
        host = Storage.allocate(n, dtype, Device.Cpu)
        if n:
            ctype = _CTYPE[dtype]
            arr = (ctype * n).from_address(host.data_ptr)
            if dtype in (Dtype.Int32, Dtype.Int64):
                for i, v in enumerate(values):
                    if isinstance(v, float):
                        raise TypeError("Unable to cast Python float to an integer storage element")
                    arr[i] = v
            elif dtype == Dtype.Bool:
                for i, v in enumerate(values):
                    arr[i] = bool(v)
            else:
                for i, v in enumerate(values):
                    arr[i] = v
        return host if device == Device.Cpu else host.to(device)

    # Buffer protocol, 1-D, writable (src/cpp/storage.cpp:67-70, 82-95).  As in the reference the
    # exported pointer of a Cuda storage is a device pointer: its length is meaningful, its
    # contents are not readable from the host.
    def __buffer__(self, flags: int) -> memoryview:
        n = self.size
        ctype = _CTYPE[self.dtype]
        fmt = _FORMAT[self.dtype]
        if n == 0:
            return memoryview((ctype * 0)()).cast("B").cast(fmt)
        arr = (ctype * n).from_address(self.data_ptr)
        arr._owner = self  # keep the storage alive while the view is
        return memoryview(arr).cast("B").cast(fmt)


_engine.register_storage(Storage, tuple(Dtype), tuple(Device))
TensorView = _engine.TensorView


def _view_struct(v: TensorView) -> _View:
    if not isinstance(v, TensorView):
        raise TypeError(f"expected a TensorView, got {type(v).__name__}")
    shape, strides = v.shape, v.strides
    nd = len(shape)
    if len(strides) != nd:
        raise RuntimeError("TensorView: shape and strides differ in length.")
    if nd > NT_MAX_DIMS:
        raise RuntimeError("TensorView: more than 8 dimensions are not supported on device.")
    if not isinstance(v.storage, Storage):
        raise TypeError("TensorView: storage must be a Storage.")
    c = _View()
    c.storage = v.storage._h
    c.ndim = nd
    for i in range(nd):
        c.shape[i] = shape[i]
        c.strides[i] = strides[i]
    c.offset = v.offset
    return c


def _vref(v: TensorView):
    return C.byref(_view_struct(v))


def _ret_storage(fn, *args) -> Storage:
    out = C.c_void_p()
    _check(fn(*args, C.byref(out)))
    return Storage._wrap(out.value)


# ---- pointwise (src/cpp/ops/binary_ops.cu:178-196, unary_ops.cu:109-128)
add = _engine.add
subtract = _engine.subtract
multiply = _engine.multiply
divide = _engine.divide
pw_equal = _engine.pw_equal
pw_greater = _engine.pw_greater
pw_greater_eq = _engine.pw_greater_eq
matmul = _engine.matmul
exp = _engine.exp
log = _engine.log
sqrt = _engine.sqrt
tanh = _engine.tanh
sigmoid = _engine.sigmoid
neg = _engine.neg
relu = _engine.relu


def equals(x1: TensorView, x2: TensorView) -> bool:
    out = C.c_int(0)
    _check(_lib.nt_equals(_vref(x1), _vref(x2), C.byref(out)))
    return bool(out.value)


def pow(x: TensorView, power) -> Storage:  # noqa: A001 - the reference's name
    s = _scalar(power)
    return _ret_storage(_lib.nt_pow, _vref(x), C.byref(s))


# ---- reductions (src/cpp/ops/reduction_ops.cu:263-276)
def _axes(axis: Sequence[int]):
    ax = [int(a) for a in axis]
    return (C.c_int64 * len(ax))(*ax), len(ax)


sum = _engine.sum  # noqa: A001  (view, axes, dtype)


def mean_f32(x: TensorView, axis: Sequence[int], count: int) -> "Storage | None":
    """Float32 sum divided by `count` in the launch that finishes the sum (the bits of sum followed by
    divide); None when the view takes none of the single-launch reduction kernels."""
    arr, n = _axes(axis)
    out = C.c_void_p()
    _check(_lib.nt_mean_f32(_vref(x), arr, C.c_int32(n), C.c_float(float(count)), C.byref(out)))
    return Storage._wrap(out.value) if out.value else None


max = _engine.max  # noqa: A001  (view, axes)
min = _engine.min  # noqa: A001
argmax = _engine.argmax
argmin = _engine.argmin
matmul_pair = _engine.matmul_pair
linear = _engine.linear


def set_matmul_pair_overlap(on: bool = True) -> None:
    """Launch the second product of `matmul_pair` as the programmatic dependent of the first (off by default)."""
    _check(_lib.nt_set_matmul_pair_overlap(int(bool(on))))


# ---- in-place (src/cpp/ops/inplace_ops.cu:81-92)
add_inplace = _engine.add_inplace
sub_inplace = _engine.sub_inplace
mul_inplace = _engine.mul_inplace
div_inplace = _engine.div_inplace
copy_inplace = _engine.copy_inplace


# ---- core ops (src/cpp/storage.cpp:96-102, ops/copy_ops.cu:219-233)
def cast(s: Storage, dtype: Dtype) -> Storage:
    return s.cast(dtype)


def to(s: Storage, device: Device) -> Storage:
    return s.to(device)


def copy_view(*, src: TensorView, out: TensorView) -> Storage:
    _check(_lib.nt_copy_view(_vref(src), _vref(out)))
    return out.storage


clone_contiguous_view_from = _engine.clone_contiguous_view_from


# Index-array gather/scatter.  Keyword names are the reference's (src/cpp/ops/copy_ops.cu:219-233);
# the reference runs them on CPU storages only, here they are device kernels.  `checked` / `unique`
# are additions: the caller already validated the indices on the host / vouches that no two source
# positions address one destination (see include/nt_b200.h).
INDEX_CHECKED = 1
INDEX_UNIQUE = 2


def _index_plan(fancy_dims_in_src, fancy_dims_data, out_axis_is_fancy, out_axis_target):
    nf, na = len(fancy_dims_in_src), len(out_axis_is_fancy)
    if len(fancy_dims_data) != nf or len(out_axis_target) != na:
        raise ValueError("index plan: list lengths differ.")
    if nf > NT_MAX_DIMS or na > NT_MAX_DIMS:
        raise RuntimeError("index plan: more than 8 dimensions are not supported on device.")
    dims = (C.c_int64 * (nf or 1))(*fancy_dims_in_src)
    views = (_View * (nf or 1))()
    for i, v in enumerate(fancy_dims_data):
        views[i] = _view_struct(v)
    is_fancy = (C.c_uint8 * (na or 1))(*[1 if f else 0 for f in out_axis_is_fancy])
    target = (C.c_int64 * (na or 1))(*out_axis_target)
    return dims, nf, views, is_fancy, target


def scatter_to_axes(*, src: TensorView, out: TensorView, fancy_dims_in_src, fancy_dims_data, out_axis_is_fancy,
                    out_axis_target, checked: bool = False, unique: bool = False) -> None:
    if len(out_axis_is_fancy) != len(src.shape):
        raise ValueError("scatter_to_axes: one axis entry per dimension of src.")
    dims, nf, views, is_fancy, target = _index_plan(fancy_dims_in_src, fancy_dims_data, out_axis_is_fancy,
                                                    out_axis_target)
    flags = (INDEX_CHECKED if checked else 0) | (INDEX_UNIQUE if unique else 0)
    _check(_lib.nt_scatter_to_axes(_vref(src), _vref(out), dims, C.c_int32(nf), views, is_fancy, target,
                                   C.c_uint32(flags)))


def gather_from_axes(*, x: TensorView, new_shape, fancy_dims_in_src, fancy_dims_data, out_axis_is_fancy,
                     out_axis_target, checked: bool = False) -> Storage:
    if len(out_axis_is_fancy) != len(new_shape):
        raise ValueError("gather_from_axes: one axis entry per dimension of new_shape.")
    dims, nf, views, is_fancy, target = _index_plan(fancy_dims_in_src, fancy_dims_data, out_axis_is_fancy,
                                                    out_axis_target)
    shape = (C.c_int64 * (len(new_shape) or 1))(*new_shape)
    return _ret_storage(_lib.nt_gather_from_axes, _vref(x), shape, C.c_int32(len(new_shape)), dims, C.c_int32(nf),
                        views, is_fancy, target, C.c_uint32(INDEX_CHECKED if checked else 0))


# ---- factories (src/cpp/factory.cu:85-99)
def _factory(fn, *args) -> Storage:
    out = C.c_void_p()
    _check(fn(*args, C.byref(out)))
    return Storage._wrap(out.value)


def zeros(n: int, dtype: Dtype, device: Device) -> Storage:
    return _factory(_lib.nt_zeros, C.c_int64(n), int(_dtype(dtype)), _device(device).value)


def ones(n: int, dtype: Dtype, device: Device) -> Storage:
    return _factory(_lib.nt_ones, C.c_int64(n), int(_dtype(dtype)), _device(device).value)


def full(n: int, value, dtype: Dtype, device: Device) -> Storage:
    s = _scalar(value)
    return _factory(_lib.nt_full, C.c_int64(n), C.byref(s), int(_dtype(dtype)), _device(device).value)


def constant(value, dtype: Dtype) -> Storage:
    """One Cuda element known to hold `value`: no fill launch until something needs its address."""
    s = _scalar(value)
    return _factory(_lib.nt_constant, C.byref(s), int(_dtype(dtype)))


def eye(n: int, dtype: Dtype, device: Device) -> Storage:
    return _factory(_lib.nt_eye, C.c_int64(n), int(_dtype(dtype)), _device(device).value)


def arange(n: int, start: int, step: int, dtype: Dtype, device: Device) -> Storage:
    return _factory(_lib.nt_arange, C.c_int64(n), C.c_int64(start), C.c_int64(step), int(_dtype(dtype)),
                    _device(device).value)


def manual_seed(seed: int) -> None:
    _check(_lib.nt_manual_seed(C.c_uint64(seed)))


def uniform(n: int, dtype: Dtype, device: Device) -> Storage:
    return _factory(_lib.nt_uniform, C.c_int64(n), int(_dtype(dtype)), _device(device).value)


# ---- CUDA (src/cpp/cuda.cpp:3-7)
def is_cuda_available() -> bool:
    return bool(_lib.nt_is_cuda_available())


def cuda_sync() -> None:
    _check(_lib.nt_cuda_sync())


# =============================================================================================
# Extensions beyond the reference's surface (include/nt_b200.h)
def set_device(ordinal: int) -> None:
    _check(_lib.nt_set_device(int(ordinal)))


def device_count() -> int:
    out = C.c_int(0)
    _check(_lib.nt_device_count(C.byref(out)))
    return out.value


def stream_handle() -> int:
    return _lib.nt_stream() or 0


def launch_count() -> int:
    out = C.c_uint64(0)
    _check(_lib.nt_launch_count(C.byref(out)))
    return out.value


def allocator_stats() -> dict:
    a, b, c = C.c_uint64(0), C.c_uint64(0), C.c_uint64(0)
    _check(_lib.nt_allocator_stats(C.byref(a), C.byref(b), C.byref(c)))
    return {"bytes_reserved": a.value, "bytes_in_use": b.value, "n_cuda_malloc": c.value}


def allocator_trim() -> None:
    _check(_lib.nt_allocator_trim())


def allocator_requests() -> int:
    """Requests made to the device arena since load (served from its cache or by cudaMalloc)."""
    n = C.c_uint64(0)
    _check(_lib.nt_allocator_requests(C.byref(n)))
    return n.value


_lib.nt_get_wait_limit_clocks.restype = C.c_int64


def set_wait_limit_clocks(clocks: int) -> None:
    """Limit, in SM clocks, of every bounded spin in device code (default 2**31)."""
    _check(_lib.nt_set_wait_limit_clocks(C.c_int64(int(clocks))))


def get_wait_limit_clocks() -> int:
    return _lib.nt_get_wait_limit_clocks()


def wait_probe() -> None:
    """Launch the one-thread kernel that waits (bounded) on a barrier nothing arrives on."""
    _check(_lib.nt_wait_probe())


TANH_CORRECTLY_ROUNDED = 0
TANH_BIT_EXACT_LIBM = 1


def set_tanh_mode(mode: int) -> None:
    _check(_lib.nt_set_tanh_mode(int(mode)))


def get_tanh_mode() -> int:
    return _lib.nt_get_tanh_mode()


RNG_HOST_MT19937_64 = 0   # the reference's seeded host stream (default)
RNG_DEVICE_PHILOX = 1     # Philox4x32-10 generated on the device


def set_rng_mode(mode: int) -> None:
    _check(_lib.nt_set_rng_mode(int(mode)))


def get_rng_mode() -> int:
    return _lib.nt_get_rng_mode()


MATMUL_EXACT_FP32 = 0
MATMUL_3XTF32 = 1
MATMUL_FP32_UNFUSED = 2
MATMUL_3XTF32_SINGLE_CHAIN = 3


def set_matmul_mode(mode: int) -> None:
    _check(_lib.nt_set_matmul_mode(int(mode)))


_lib.nt_get_matmul_tc_min_macs.restype = C.c_int64


def set_matmul_tc_min_macs(macs: int) -> None:
    """Products of at most this many multiply-adds take the exact FP32 kernel in modes 1 and 3 (default 2**21)."""
    _check(_lib.nt_set_matmul_tc_min_macs(C.c_int64(int(macs))))


def get_matmul_tc_min_macs() -> int:
    return _lib.nt_get_matmul_tc_min_macs()


def set_matmul_operand_planes(natural: bool = True, cached: bool = True) -> None:
    """Mode-1 operand planes: `natural` keeps the source's row-major order (no transposing split, the kernel
    reads either major); `cached` remembers them per storage and view until the storage is written again."""
    _check(_lib.nt_set_matmul_operand_planes(int(bool(natural)), int(bool(cached))))


def set_producer_planes(on: bool = True) -> None:
    """tanh / tanh_backward write the TF32 planes of a large dense 2-D result themselves (see the header)."""
    _check(_lib.nt_set_producer_planes(int(bool(on))))


def set_matmul_schedule(max_splits: int = 8, panel: int = 8) -> None:
    """Split-K limit and tile-panel width of the mode-1 tensor-core kernel (see the header)."""
    _check(_lib.nt_set_matmul_schedule(int(max_splits), int(panel)))


class keep_rounding:
    """While entered, this thread's products keep the rounding of TF32 planes (see nt_matmul_keep_rounding in the header)."""

    def __init__(self, on: bool = True) -> None:
        self._on = on

    def __enter__(self) -> None:
        self._was = _lib.nt_matmul_keep_rounding(int(self._on))

    def __exit__(self, *_exc) -> None:
        _lib.nt_matmul_keep_rounding(self._was)


def matmul_force_fused(tile_n: int = 0, cluster: int = 0) -> None:
    """Which variant of the self-splitting tensor-core kernel this thread's products take; 0, 0 goes by expected time."""
    _check(_lib.nt_matmul_force_fused(int(tile_n), int(cluster)))


def matmul_kernel_counts() -> tuple[int, int, int]:
    """Float32 products launched so far: through operand planes, by the self-splitting kernel, on the CUDA cores."""
    counts = [C.c_uint64() for _ in range(3)]
    _check(_lib.nt_matmul_kernel_counts(*map(C.byref, counts)))
    return tuple(c.value for c in counts)


def set_transposed_tile_pipeline(on: bool = True) -> None:
    """Large fp32 elementwise ops with a transposed operand: TMA-fed persistent kernel (default) or the
    register-staged tile kernel (see the header)."""
    _check(_lib.nt_set_transposed_tile_pipeline(int(bool(on))))


def matmul_split_stats() -> tuple[int, int]:
    """(operand-split launches, operand-plane cache hits) since load."""
    a, b = C.c_uint64(0), C.c_uint64(0)
    _check(_lib.nt_matmul_split_stats(C.byref(a), C.byref(b)))
    return a.value, b.value


def get_matmul_mode() -> int:
    return _lib.nt_get_matmul_mode()


relu_backward = _engine.relu_backward
tanh_backward = _engine.tanh_backward
sigmoid_backward = _engine.sigmoid_backward
exp_backward = _engine.exp_backward
log_backward = _engine.log_backward
sqrt_backward = _engine.sqrt_backward


def pow_backward(g: TensorView, x: TensorView, exponent: float) -> Storage:
    return _ret_storage(_lib.nt_pow_backward, _vref(g), _vref(x), C.c_float(exponent))


div_backward_x2 = _engine.div_backward_x2


def extremum_backward(g_expanded: TensorView, x: TensorView, m_expanded: TensorView, axis: Sequence[int]) -> Storage:
    arr, n = _axes(axis)
    return _ret_storage(_lib.nt_extremum_backward, _vref(g_expanded), _vref(x), _vref(m_expanded), arr, C.c_int32(n))


mul_backward = _engine.mul_backward   # (x2*g, x1*g) in one pass, or None
div_backward = _engine.div_backward   # (g/x2, ((-x1)/x2**2)*g) in one pass, or None


def sgd_update(param: TensorView, grad: TensorView, lr: float, grad_scale: float = 1.0) -> None:
    _check(_lib.nt_sgd_update(_vref(param), _vref(grad), C.c_float(lr), C.c_float(grad_scale)))


def sum_rows_noalloc(src: Storage, n_rows: int, row_len: int, out: Storage) -> None:
    """out[r] = sum of row r of the dense fp32 [n_rows, row_len] matrix at the start of `src`, through
    the entry point that never allocates: both storages are the caller's, the kernel's scratch is a
    fixed array inside the library (see nt_sum_rows_noalloc in include/nt_b200.h for the limits)."""
    for s, need in ((src, n_rows * row_len), (out, n_rows)):
        if s.device != Device.Cuda or s.dtype != Dtype.Float32 or s.size < need:
            raise ValueError("sum_rows_noalloc: Float32 Cuda storages of at least n_rows*row_len and n_rows elements")
    _check(_lib.nt_sum_rows_noalloc(C.c_void_p(src.data_ptr), C.c_int64(n_rows), C.c_int64(row_len),
                                    C.c_void_p(out.data_ptr)))


COMM_ID_BYTES = 128


def comm_unique_id() -> bytes:
    buf = (C.c_uint8 * COMM_ID_BYTES)()
    _check(_lib.nt_comm_unique_id(buf))
    return bytes(buf)


def comm_init(rank: int, world: int, unique_id: bytes) -> None:
    if len(unique_id) != COMM_ID_BYTES:
        raise ValueError("comm_init: unique id must be 128 bytes")
    buf = (C.c_uint8 * COMM_ID_BYTES).from_buffer_copy(unique_id)
    _check(_lib.nt_comm_init(int(rank), int(world), buf))


def comm_init_timeout(rank: int, world: int, unique_id: bytes, timeout_ms: int) -> None:
    """comm_init with an explicit limit on the rendezvous: RuntimeError if a rank has not joined in time."""
    if len(unique_id) != COMM_ID_BYTES:
        raise ValueError("comm_init: unique id must be 128 bytes")
    buf = (C.c_uint8 * COMM_ID_BYTES).from_buffer_copy(unique_id)
    _check(_lib.nt_comm_init_timeout(int(rank), int(world), buf, C.c_int64(int(timeout_ms))))


def comm_group_begin() -> None:
    """Open a bucket: orders the communication stream after the compute stream; the all-reduces issued
    until comm_group_end go out as one NCCL launch."""
    _check(_lib.nt_comm_group_begin())


def comm_group_end() -> None:
    _check(_lib.nt_comm_group_end())


def comm_sgd_update(param: "TensorView", grad: "TensorView", lr: float, grad_scale: float = 1.0) -> None:
    """sgd_update enqueued on the communication stream, behind the collectives issued so far."""
    _check(_lib.nt_comm_sgd_update(_vref(param), _vref(grad), C.c_float(lr), C.c_float(grad_scale)))


def comm_sync(timeout_ms: int) -> None:
    """Host-side wait for the communication stream with a time limit; aborts the communicator past it."""
    _check(_lib.nt_comm_sync(C.c_int64(int(timeout_ms))))


def comm_abort() -> None:
    _check(_lib.nt_comm_abort())


def comm_allreduce_sum(s: Storage) -> None:
    _check(_lib.nt_comm_allreduce_sum(C.c_void_p(s._h)))


def comm_wait() -> None:
    _check(_lib.nt_comm_wait())


def comm_destroy() -> None:
    _check(_lib.nt_comm_destroy())


class Event:
    """CUDA event on the library's compute stream."""

    def __init__(self):
        h = C.c_void_p()
        _check(_lib.nt_event_create(C.byref(h)))
        self._h = h.value

    def record(self) -> "Event":
        _check(_lib.nt_event_record(C.c_void_p(self._h)))
        return self

    def elapsed_ms(self, stop: "Event") -> float:
        ms = C.c_float(0)
        _check(_lib.nt_event_elapsed_ms(C.c_void_p(self._h), C.c_void_p(stop._h), C.byref(ms)))
        return ms.value

    def __del__(self):
        h = getattr(self, "_h", None)
        if h:
            try:
                _lib.nt_event_destroy(C.c_void_p(h))
            except Exception:
                pass
            self._h = None


class Graph:
    """A captured sequence of launches: `with g.capture(): ...` records whatever the block enqueues
    (kernels, NCCL collectives, stream joins), `g.replay()` re-issues it as one CUDA-graph launch.
    Tensors created inside the block keep their device addresses, so results are read from the same
    tensors after every replay."""

    def __init__(self):
        self._id = 0

    def capture(self):
        return _GraphCapture(self)

    def replay(self) -> None:
        _check(_lib.nt_graph_launch(self._id))

    def close(self) -> None:
        if self._id:
            _check(_lib.nt_graph_destroy(self._id))
            self._id = 0

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


class _GraphCapture:
    def __init__(self, graph: Graph):
        self._g = graph

    def __enter__(self):
        gid = C.c_int(0)
        _check(_lib.nt_graph_begin_capture(C.byref(gid)))
        self._g._id = gid.value
        return self._g

    def __exit__(self, exc_type, exc, tb):
        status = _lib.nt_graph_end_capture(self._g._id)
        if exc_type is None:
            _check(status)
        return False


def matmul_profile_enable(on: bool) -> None:
    _check(_lib.nt_matmul_profile_enable(1 if on else 0))


def matmul_profile_read() -> tuple[float, int]:
    total, n = C.c_double(0), C.c_int64(0)
    _check(_lib.nt_matmul_profile_read(C.byref(total), C.byref(n)))
    return total.value, n.value


def upload_async(s: Storage, host_ptr: int, nbytes: int) -> None:
    _check(_lib.nt_storage_upload_async(C.c_void_p(s._h), C.c_void_p(host_ptr), C.c_int64(nbytes)))


def upload_fence() -> None:
    _check(_lib.nt_upload_fence())


def host_register(ptr: int, nbytes: int) -> None:
    _check(_lib.nt_host_register(C.c_void_p(ptr), C.c_int64(nbytes)))


def host_unregister(ptr: int) -> None:
    _check(_lib.nt_host_unregister(C.c_void_p(ptr)))


def exported_symbols() -> list[str]:
    """Every symbol declared in include/nt_b200.h that this library must export."""
    import re

    header = Path(__file__).resolve().parent.parent / "include" / "nt_b200.h"
    text = header.read_text()
    return sorted(set(re.findall(r"\b(nt_[a-z0-9_]+)\s*\(", text)))
