"""The trimmed sorting network (NetGeom in network.cuh) on the CPU, against a
plain sort: rows past n are left out of every exchange, and a block of phase
2^K ascends iff bit K of its rows equals bit K of m - 1, where m is n rounded
up to whole tiles; tiles keep the plain directions."""
import numpy as np
import pytest


def trimmed_sort(rows, lt):
    n = len(rows)
    log_n = max(0, (n - 1).bit_length())
    tile = 1 << lt
    m = min(-(-n // tile) * tile, 1 << log_n)
    dirx = (m - 1) & ~(tile - 1) if m < 1 << log_n else 0
    a = np.concatenate([rows, np.full(m - n, np.iinfo(np.uint64).max, np.uint64)])
    i = np.arange(m)
    for k in range(1, log_n + 1):
        for b in range(k - 1, -1, -1):
            lo = i[((i >> b) & 1) == 0]
            lo = lo[lo + (1 << b) < m]  # both rows exist
            hi = lo + (1 << b)
            asc = (((lo ^ dirx) >> k) & 1) == 0
            swap = np.where(asc, a[lo] > a[hi], a[lo] < a[hi])
            a[lo[swap]], a[hi[swap]] = a[hi[swap]], a[lo[swap]]
    return a[:n]


@pytest.mark.parametrize("lt", [0, 2, 3])
def test_trimmed_network_sorts_every_size(lt):
    rng = np.random.default_rng(lt)
    top = np.iinfo(np.uint64).max
    for n in list(range(1, 140)) + [255, 256, 257, 383, 385, 511, 513, 767, 769]:
        for rows in (rng.integers(0, 2**63, n).astype(np.uint64), rng.integers(0, 3, n).astype(np.uint64),
                     np.where(rng.random(n) < 0.5, top, top - 1).astype(np.uint64), np.arange(n, 0, -1).astype(np.uint64)):
            assert np.array_equal(trimmed_sort(rows, lt), np.sort(rows)), (lt, n)
