"""The trimmed sorting network (NetGeom in network.cuh) on the CPU, against a
plain sort: rows past n are left out of every exchange, and a block of phase
2^K ascends iff bit K of its rows equals bit K of m - 1, where m is n rounded
up to whole tiles; tiles keep the plain directions.  Then the padded networks
without their blocks of padding (net_pass_tiles) against the whole networks,
and the merge of descending with ascending rows that the gather takes."""
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


def padded_network(rank, live, skip):
    """Arrangement of the rows of the padded network with strict compares; with
    `skip` phase 2^K stops after the last block of 2^K rows below `live`."""
    np_ = len(rank)
    a, idx = rank.copy(), np.arange(np_)
    for k in range(1, (np_ - 1).bit_length() + 1):
        m = min(np_, -(-live // (1 << k)) << k) if skip else np_
        for b in range(k - 1, -1, -1):
            lo = np.arange(m)
            lo = lo[((lo >> b) & 1) == 0]
            hi = lo + (1 << b)
            swap = np.where(((lo >> k) & 1) == 0, a[lo] > a[hi], a[lo] < a[hi])
            for x in (a, idx):
                x[lo[swap]], x[hi[swap]] = x[hi[swap]], x[lo[swap]]
    return idx


def test_padded_network_without_blocks_of_padding():
    rng = np.random.default_rng(1)
    for n in list(range(1, 70)) + [129, 160, 191, 255, 257, 300, 385, 513]:
        np_ = 1 << max(0, (n - 1).bit_length())
        for pad in (2, 1, 0):  # above, among and below the rows' own values
            rank = np.full(np_, pad)
            rank[:n] = rng.integers(0, 3, n)
            assert np.array_equal(padded_network(rank, n, True), padded_network(rank, n, False)), (n, pad)


def compact_network(rows, marks, n, skip, fused):
    """ORCompact bottom-up; with `skip` a fused pass of `fused` levels stops
    after the last block of its highest level that holds a row below n."""
    np_ = len(rows)
    row, mark = rows.copy(), marks.copy()
    pre = np.concatenate([[0], np.cumsum(marks)])
    log_n = (np_ - 1).bit_length()
    for b in range(log_n):
        top = min(log_n, (b // fused + 1) * fused)
        m = min(np_, -(-n // (1 << top)) << top) if skip else np_
        half = 1 << b
        lo = np.arange(m)
        lo = lo[((lo >> b) & 1) == 0]
        hi, start = lo + half, lo & ~(2 * half - 1)
        off, left = pre[start] & (2 * half - 1), pre[start + half] - pre[start]
        if b == 0:
            swap = ((mark[lo] == 0) & (mark[hi] != 0)) != (off == 1)
        else:
            swap = ((((off & (half - 1)) + left) >= half) != (off >= half)) != \
                ((lo & (half - 1)) >= ((off + left) & (half - 1)))
        for x in (row, mark):
            x[lo[swap]], x[hi[swap]] = x[hi[swap]], x[lo[swap]]
    return row, mark


@pytest.mark.parametrize("fused", [1, 2, 3])
def test_compaction_without_blocks_of_padding(fused):
    rng = np.random.default_rng(fused)
    for n in list(range(2, 70)) + [129, 160, 255, 257, 300, 513]:
        np_ = 1 << (n - 1).bit_length()
        for density in (0.0, 0.3, 1.0):
            marks, rows = np.zeros(np_, int), np.full(np_, -1)
            marks[:n], rows[:n] = rng.random(n) < density, np.arange(n)
            want = compact_network(rows, marks, n, False, fused)
            got = compact_network(rows, marks, n, True, fused)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), n
            assert np.array_equal(want[0][: marks.sum()], np.flatnonzero(marks))


@pytest.mark.parametrize("lt", [0, 2])
def test_descending_then_ascending_rows_merge(lt):
    rng = np.random.default_rng(lt)
    for n in list(range(1, 100)) + [129, 255, 257, 400]:
        m = min(-(-n // (1 << lt)) << lt, 1 << max(0, (n - 1).bit_length()))
        for down in {0, 1, n // 3, n - 1, n}:
            rows = rng.integers(0, 40, n)
            a = np.concatenate([-np.sort(-rows[:down]), np.sort(rows[down:]), np.full(m - n, 99)])
            for b in range((m - 1).bit_length() - 1, -1, -1):
                lo = np.arange(m)
                lo = lo[((lo >> b) & 1) == 0]
                lo = lo[lo + (1 << b) < m]
                a[lo], a[lo + (1 << b)] = np.minimum(a[lo], a[lo + (1 << b)]), np.maximum(a[lo], a[lo + (1 << b)])
            assert np.array_equal(a[:n], np.sort(rows)), (n, down)
