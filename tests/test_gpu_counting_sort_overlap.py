"""The counting sort where an output lies over the keys (an argsort in place,
offsets over the keys they count), at both entry points, with the counts array
on and off a 16-byte boundary: cells of one block's range, cells past the small
ones' rank count, many blocks.  Against numpy's stable argsort."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sort(entry, counts, keys, n, cells, order):
    from lustrine_gb300 import _lib
    lib = _lib.load()
    f = lib.lustrine_counting_sort_noalloc if entry == "noalloc" else lib.lustrine_counting_sort
    return f(C.c_void_p(counts), C.c_void_p(keys), C.c_size_t(n), C.c_size_t(cells), C.c_void_p(order), None)


@pytest.mark.parametrize("entry", ["pool", "noalloc"])
@pytest.mark.parametrize("over", ["order", "order-shifted", "counts", "counts-shifted"])
@pytest.mark.parametrize("n,cells", [(1, 1), (257, 300), (5_000, 40), (40_000, 70_001), (300_001, 400_000)])
def test_outputs_over_keys(n, cells, over, entry):
    import torch
    rng = np.random.default_rng(n + cells)
    keys = rng.integers(0, cells, n).astype(np.int32)
    m = n + cells + 64
    # one array of each: [0, n) keys, then whatever does not lie over them
    buf = torch.full((3 * m,), -7, dtype=torch.int32, device="cuda")
    at = m + 8
    buf[at:at + n] = torch.from_numpy(keys).cuda()
    shift = 5 if over.endswith("shifted") else 0
    order = at - shift if over.startswith("order") else 2 * m + 3
    counts = at - shift if over.startswith("counts") else 2 * m + 3
    torch.cuda.synchronize()
    p = buf.data_ptr()
    assert _sort(entry, p + 4 * counts, p + 4 * at, n, cells, p + 4 * order) == 0
    got = buf.cpu().numpy()
    np.testing.assert_array_equal(got[order:order + n], np.argsort(keys, kind="stable"))
    np.testing.assert_array_equal(got[counts:counts + cells + 1],
                                  np.concatenate([[0], np.cumsum(np.bincount(keys, minlength=cells))]))
    lo, hi = min(order, counts), max(order, counts)
    assert (got[:min(at, lo)] == -7).all() and (got[hi + (n if hi == order else cells + 1):] == -7).all()


@pytest.mark.parametrize("n", [1 << 20, (1 << 20) + 1])
def test_page_locked_keys(n):
    import torch
    keys = np.random.default_rng(n).integers(0, 70_000, n).astype(np.int32)
    k = torch.from_numpy(keys).pin_memory()
    counts = torch.empty(70_001, dtype=torch.int32, device="cuda")
    order = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert _sort("pool", counts.data_ptr(), k.data_ptr(), n, 70_000, order.data_ptr()) == 0
    np.testing.assert_array_equal(order.cpu().numpy(), np.argsort(keys, kind="stable"))


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n,cells", [(0, 5), (33, 4095), (5000, 8193), (1 << 20, 1 << 20)])
def test_noalloc_counts_alignment(n, cells, offset):
    import torch
    keys = np.random.default_rng(n + cells).integers(0, cells, n).astype(np.int32)
    k = torch.from_numpy(keys).cuda()
    counts = torch.full((cells + 5,), -7, dtype=torch.int32, device="cuda")
    order = torch.full((n + 1,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert _sort("noalloc", counts.data_ptr() + 4 * offset, k.data_ptr(), n, cells, order.data_ptr()) == 0
    got = counts.cpu().numpy()
    np.testing.assert_array_equal(got[offset:offset + cells + 1],
                                  np.concatenate([[0], np.cumsum(np.bincount(keys, minlength=cells))]))
    assert (got[:offset] == -7).all() and (got[offset + cells + 1:] == -7).all()
    np.testing.assert_array_equal(order.cpu().numpy()[:n], np.argsort(keys, kind="stable"))
