"""The standalone counting sort where its scan and scratch change path: cell
counts around the scan tile (4,096 cells) and past the 4,096 tiles that are
summed without a scan of their own, a counts array that is not 16-byte
aligned, calls from several threads on their own streams, scratch larger than
the pool keeps, invalid keys after valid ones.  Against numpy's stable argsort."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(keys, cells, offset=0, stream=None):
    import torch
    from lustrine_gb300.sorting import counting_sort
    k = torch.from_numpy(keys).cuda()
    buf = torch.full((cells + 1 + offset,), -7, dtype=torch.int32, device="cuda")
    out = torch.full((len(keys),), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    counting_sort(buf[offset:], k, cells, out, stream)
    hist = np.bincount(keys, minlength=cells)
    want = np.concatenate([[0], np.cumsum(hist)])
    return (np.array_equal(buf[offset:].cpu().numpy(), want)
            and np.array_equal(out.cpu().numpy(), np.argsort(keys, kind="stable"))
            and (buf[:offset].cpu().numpy() == -7).all())


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n,cells", [(0, 4096), (33, 4095), (5000, 4096), (5000, 4097), (70_001, 8195),
                                     (1000, 17_000_001)])
def test_counting_sort_scan_paths(n, cells, offset):
    rng = np.random.default_rng(n + cells)
    assert _check(rng.integers(0, cells, n).astype(np.int32), cells, offset)


def test_counting_sort_threads_and_streams():
    import torch
    ok = [None] * 6

    def work(t):
        rng = np.random.default_rng(t)
        s = torch.cuda.Stream()
        ok[t] = all(_check(rng.integers(0, 1000 * (t + 1), 20_000 * (t + 1)).astype(np.int32), 1000 * (t + 1),
                           t % 2, s) for _ in range(5))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert ok == [True] * 6


def test_counting_sort_large_scratch_invalid_keys_and_release():
    from lustrine_gb300 import LustrineError, _lib
    rng = np.random.default_rng(3)
    big = rng.integers(0, 30_000_000, 4_000_000).astype(np.int32)  # 152 MB of scratch
    assert _check(big, 30_000_000)
    for bad in (-1, 1000, np.iinfo(np.int32).min):
        keys = rng.integers(0, 1000, 5000).astype(np.int32)
        keys[4321] = bad
        with pytest.raises(LustrineError):
            _check(keys, 1000)
        keys[4321] = 999
        assert _check(keys, 1000)
    assert _lib.load().lustrine_release_scratch() == 0
    assert _check(rng.integers(0, 1000, 5000).astype(np.int32), 1000)
