"""The 3xTF32 kernel that splits its operands itself has the bits of the plane-fed one: at the edges of its tiles,
blocks and periods, with one CTA and with a cluster per tile, over several k-parts, in every operand layout."""

import numpy as np
import pytest

from tests.util import bits

pytestmark = pytest.mark.gpu

# (batch, M, K, N): one period and less, ragged periods, k-parts (K >= 1024), more tiles than SMs, batches
SHAPES = [(1, 256, 784, 256), (1, 784, 256, 257), (1, 130, 255, 333), (1, 129, 257, 260), (1, 64, 4096, 64), (1, 300, 2500, 50),
          (1, 512, 1024, 640), (1, 1000, 1100, 1030), (1, 2048, 1024, 1024), (1, 128, 9000, 31), (5, 200, 300, 70), (32, 256, 256, 256)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "strided"])
def test_same_bits_as_the_plane_fed_kernel(nt, shape, layout):
    batch, M, K, N = shape
    lead = (batch,) if batch > 1 else ()
    rng = np.random.default_rng(M + K + N)
    a, b = rng.uniform(-1, 1, (*lead, M, K)).astype(np.float32), rng.uniform(-1, 1, (*lead, K, N)).astype(np.float32)

    def dev(x, turned=False):
        return nt.Tensor.from_numpy(np.ascontiguousarray(np.swapaxes(x, -1, -2)), "cuda").transpose(-2, -1) if turned else nt.Tensor.from_numpy(x, "cuda")

    if layout == "strided":
        ta, tb = dev(np.repeat(a, 2, axis=-1))[..., ::2], dev(np.repeat(b, 2, axis=-1))[..., ::2]
    else:
        ta, tb = dev(a, layout == "tn"), dev(b, layout == "nt")
    ta.enable_grad()  # a recorded product: summed as the tensor cores do, whatever the size
    keep = nt._C.get_matmul_tc_min_macs()
    got = []
    try:
        for min_macs in (0, 1):  # 0: through planes; otherwise by expected time
            nt._C.set_matmul_tc_min_macs(min_macs)
            got.append((ta @ tb).numpy())
            if batch == 1:
                bias = nt.Tensor.from_numpy(np.random.default_rng(5).standard_normal(N).astype(np.float32), "cuda")
                got.append(nt.Tensor._new_contiguous(nt._C.linear(ta._C_view, tb._C_view, bias._C_view), (M, N)).numpy())
    finally:
        nt._C.set_matmul_tc_min_macs(keep)
    half = len(got) // 2
    for x, y in zip(got[:half], got[half:]):
        assert np.array_equal(bits(x), bits(y)), np.abs(x - y).max()
    rows = slice(0, 32)
    scale = np.abs(a[..., rows, :].astype(np.float64)) @ np.abs(b.astype(np.float64))
    assert (np.abs(got[0][..., rows, :] - a[..., rows, :].astype(np.float64) @ b.astype(np.float64)) <= 2e-6 * scale).all()


VARIANTS = [(32, 1), (32, 2), (32, 4), (32, 8), (64, 1), (64, 2), (64, 4), (64, 8), (128, 1)]


@pytest.mark.parametrize("shape", [(1, 512, 2048, 512), (1, 256, 4096, 512), (1, 250, 4100, 500), (1, 130, 255, 333), (1, 300, 2500, 50),
                                   (1, 1024, 1024, 1024), (5, 200, 300, 70), (3, 100, 520, 129)], ids=str)
@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "strided"])
def test_every_variant_has_the_bits_of_the_plane_fed_kernel(nt, shape, layout):
    """Each tile width and cluster size, whichever the expected times would choose, over one and several periods and k-parts;
    the launch counts say which kernel ran."""
    batch, M, K, N = shape
    lead = (batch,) if batch > 1 else ()
    rng = np.random.default_rng(M + K + N)
    a, b = rng.uniform(-1, 1, (*lead, M, K)).astype(np.float32), rng.uniform(-1, 1, (*lead, K, N)).astype(np.float32)

    def dev(x, turned=False):
        return nt.Tensor.from_numpy(np.ascontiguousarray(np.swapaxes(x, -1, -2)), "cuda").transpose(-2, -1) if turned else nt.Tensor.from_numpy(x, "cuda")

    if layout == "strided":
        ta, tb = dev(np.repeat(a, 2, axis=-1))[..., ::2], dev(np.repeat(b, 2, axis=-1))[..., ::2]
    else:
        ta, tb = dev(a, layout == "tn"), dev(b, layout == "nt")
    bias = nt.Tensor.from_numpy(np.random.default_rng(5).standard_normal(N).astype(np.float32), "cuda")

    def products():
        before = nt._C.matmul_kernel_counts()
        out = [nt.Tensor._new_contiguous(nt._C.matmul(ta._C_view, tb._C_view), (*lead, M, N)).numpy()]
        if batch == 1:
            out.append(nt.Tensor._new_contiguous(nt._C.linear(ta._C_view, tb._C_view, bias._C_view), (M, N)).numpy())
        return out, [x - y for x, y in zip(nt._C.matmul_kernel_counts(), before)]

    want, ran = products()
    assert ran == [len(want), 0, 0]
    for tile, cluster in VARIANTS:
        nt._C.matmul_force_fused(tile, cluster)
        try:
            got, ran = products()
        finally:
            nt._C.matmul_force_fused()
        # several k-parts (of 512 and more but for the last, where tiles leave SMs idle) have no room beside 128 columns
        assert ran == [0, len(want), 0] or (tile == 128 and K > 512 and layout != "strided" and ran == [len(want), 0, 0])
        for x, y in zip(got, want):
            assert np.array_equal(bits(x), bits(y)), (tile, cluster, np.abs(x - y).max())


def test_variants_that_do_not_exist_are_refused(nt):
    for tile, cluster in ((128, 2), (16, 1), (32, 3), (0, 1), (64, 0)):
        with pytest.raises(ValueError):
            nt._C.matmul_force_fused(tile, cluster)
