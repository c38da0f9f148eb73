"""A/B timing of one load tune of the network passes against the plain
kernels, on the seeded workloads, with CUDA events on the launching stream.

    python -m velodb_b200.tune_ab tensor_tile_loads
    python -m velodb_b200.tune_ab merge_pipeline

For each workload (the 1.5 M x 6 M join + group-by + top-10, GROUP BY a BIGINT
key with a sum over 2 M rows, ORDER BY (DOUBLE, DATE) of 1.5 M rows, key-payload
sorts of 2^20, 3 M, 2^23 and 2^24 rows; the filter + group-by's key sort has no
tuned form) and each setting (off, on): 3 warm-up calls, the mean of 10 timed calls, then one call
with the library's pass timer for the per-pass-kind means, and whether the
outputs of the two settings are identical.  Prints one JSON object.
"""
from __future__ import annotations

import argparse
import json

import numpy as np
import torch

from . import capi
from . import workloads as W


def _timed(fn, reps=10):
    for _ in range(3):
        fn()
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(reps):
        fn()
    e.record()
    torch.cuda.synchronize()
    return s.elapsed_time(e) / reps


def _pass_means(fn):
    capi.set_pass_timing(True)
    capi.clear_pass_times()
    fn()
    torch.cuda.synchronize()
    pt = capi.last_pass_times()
    capi.set_pass_timing(False)
    out = {}
    for kind in ("tile_sort", "merge", "global", "compact_tile", "compact_global"):
        ms = [p[3] for p in pt if p[0] == kind]
        if ms:
            out[kind] = {"passes": len(ms), "mean_us": float(np.mean(ms)) * 1e3}
    return out


def _workloads():
    """(name, call, reset): reset restores the input of an in-place sort."""
    dim, fact = W.join_tables()
    dt = capi.join_to_device(dim, fact)
    jsc = torch.empty(capi.join_groupby_topk_scratch_bytes(len(dim["key"]), len(fact["fk"])), dtype=torch.uint8,
                      device="cuda")
    yield "join_groupby_top10", lambda: capi.join_groupby_topk(dt, W.JOIN_PRED, W.JOIN_TOPK, scratch=jsc), None
    n = 2_000_003
    gk = torch.from_numpy((W.splitmix64(3, n, 0) % np.uint64(100_000)).astype(np.int64)).cuda()
    gv = torch.from_numpy((W.splitmix64(3, n, 1) % np.uint64(10**7)).astype(np.int64)).cuda()

    def group_by():
        keys, sums, counts, groups = capi.ogroupby(gk, 5, n, sums=[gv])
        return keys, sums[0], counts, groups

    yield "groupby_bigint_2m", group_by, None
    n_ord = 1_500_000
    price = torch.zeros(1 << 21, dtype=torch.float64, device="cuda")
    date = torch.zeros(1 << 21, dtype=torch.int32, device="cuda")
    price0 = torch.from_numpy((W.splitmix64(4, n_ord, 0) % np.uint64(10**7)).astype(np.float64)).cuda()
    date0 = torch.from_numpy((W.splitmix64(4, n_ord, 1) % np.uint64(2557)).astype(np.int32)).cuda()

    def order_by():
        return price, date, capi.sort_columns([price, date], [7, 10], [False, True], n_ord)

    def order_by_reset():
        price[:n_ord].copy_(price0)
        date[:n_ord].copy_(date0)

    yield "orderby_double_date_1.5m", order_by, order_by_reset
    for rows in (1 << 20, 3_000_000, 1 << 23, 1 << 24):
        keys, pay = W.sort_kp(rows, seed=rows.bit_length())
        cap = capi.next_pow2(rows)
        k0, p0 = capi.to_dev_u64(keys, cap), capi.to_dev_u32(pay, cap)
        k, p = k0.clone(), p0.clone()

        def sort(k=k, p=p, rows=rows):
            capi.osort_kp(k, p, rows)
            return k, p

        def reset(k=k, p=p, k0=k0, p0=p0):
            k.copy_(k0)
            p.copy_(p0)

        yield f"sort_kp_{rows}", sort, reset


def main(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("tune", choices=sorted(capi.TUNES))
    a = ap.parse_args(argv)
    switch = capi.TUNES[a.tune]
    res = {"tune": a.tune, "workloads": {}}
    try:
        for name, fn, reset in _workloads():
            row, outs = {}, {}
            for on in (False, True):
                switch(on)
                if reset is not None:
                    reset()
                out = fn()
                torch.cuda.synchronize()
                outs[on] = [t.clone() for t in out]
                row["on" if on else "off"] = {"ms": _timed(fn), "passes": _pass_means(fn)}
            # the sorts run in place: the checked call of each setting sorts
            # the same input, the timed calls re-sort sorted rows (the same
            # passes: the network does not depend on the data)
            row["identical"] = all(torch.equal(x, y) for x, y in zip(outs[False], outs[True]))
            res["workloads"][name] = row
            torch.cuda.empty_cache()
    finally:
        switch(False)
    print(json.dumps(res))


if __name__ == "__main__":
    main()
