"""The hit merge at the edges of its two forms: where the key table grows with the number of records, ranges
just inside and just beyond it, and calls for which the table form has no room in device memory."""
import numpy as np
import pytest

from oracle import merge as M
from opticks_b200 import scenes
from tests.test_merge import SD, random_records

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(cuda):
    from opticks_b200 import engine as E
    fd, lib, _, _ = scenes.sphere_in_box(1)
    e = E.Engine(fd.arrays(), lib.arrays(), E.default_config(max_photon=64))
    yield e
    e.close()


def _same(a, b):
    assert a.shape == b.shape
    np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))


def _table(n):
    """cells of the table for n records: 32 a record in steps of 2^15, at least 2^24"""
    return max(1 << 24, -(-32 * n // 32768) * 32768)


def _records(n, lite, nbucket, rng):
    """one identity and nbucket 1 ns buckets, the first and the last of them occurring: nbucket cells"""
    rec = random_records(n, lite, rng, num_id=1, tmax=1.0, tq=1.0)
    t = rng.integers(0, nbucket, n).astype(np.float64)
    t[: n // 2] = t[0]                                   # half of the records in one group
    t[0], t[-1] = 0, nbucket - 1
    (rec[:, 1] if lite else rec[:, 0, 3])[...] = t.astype(np.float32)
    u = rec.view(np.uint32)
    if not lite:
        u[:, 3, 1] = 5
    else:
        u[:, 0] = (1 << 16) | 5
    return rec


@pytest.mark.parametrize("lite", [0, 1])
@pytest.mark.parametrize("n", [524_287, 524_288, 524_289, 1_500_001])
def test_table_edge(eng, lite, n):
    # whole nanoseconds below 2^24 are exact in FP32; above, every second or fourth one
    for cells in (_table(n) - 4, _table(n), _table(n) + 4):
        rec = _records(n, lite, cells, np.random.default_rng(n + cells))
        for mask in (0xFFFFFFFF, SD):
            _same(eng.merge_hits(rec, mask, 1.0), M.merge(rec, mask, 1.0))


@pytest.mark.parametrize("lite", [0, 1])
@pytest.mark.parametrize("n", [1, 2048, 2049, 65_537, 300_001])
def test_sorted_ranges(eng, lite, n):
    """32-bit buckets: the sort, with few digits scanned by one block and many by three launches"""
    rec = random_records(n, lite, np.random.default_rng(n), num_id=60_000, tmax=4.0e9, tq=1.0e6)
    for mask in (0xFFFFFFFF, SD, 0):
        _same(eng.merge_hits(rec, mask, 1.0), M.merge(rec, mask, 1.0))


@pytest.mark.parametrize("lite", [0, 1])
def test_no_room_for_the_table(eng, cuda, lite):
    """nearly all device memory taken: the records that few selected ones need still merge"""
    torch = cuda
    n = 3_000_001
    rng = np.random.default_rng(11 + lite)
    rec = random_records(n, lite, rng, num_id=300, tmax=80.0)
    u = rec.view(np.uint32)
    flag = u[:, 3] if lite else u[:, 3, 3]
    flag[...] = np.where(rng.random(n) < 0.01, SD, 0x8)
    ref = M.merge(rec, SD, 1.0)
    d = torch.from_numpy(rec.view(np.int32)).cuda()
    full = torch.zeros_like(d)
    eng.merge_hits_device(d, full, SD, 1.0)                       # both forms' kernels are loaded before memory is short
    eng.merge_hits(random_records(3000, lite, rng, num_id=60_000, tmax=4.0e9, tq=1.0e6), SD, 1.0)
    eng.trim()
    keep = []
    left = 40 << 20                                               # to 72 MB; the table form takes 96 MB here
    for size in (1 << 34, 1 << 30, 1 << 26, 1 << 25):
        while torch.cuda.mem_get_info()[0] > left + size:
            keep.append(torch.empty((size,), dtype=torch.uint8, device="cuda"))
    try:
        nm = eng.merge_hits_device(d, full, SD, 1.0)
        got = full[:nm].cpu().numpy()
    finally:
        del keep
        torch.cuda.empty_cache()
        eng.trim()
    _same(got, ref.view(np.int32))
    nm = eng.merge_hits_device(d, full, SD, 1.0)                  # and through the table again
    _same(full[:nm].cpu().numpy(), ref.view(np.int32))
