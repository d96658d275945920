"""GPU parity of the one-CTA sort of 8-byte keys around the runs of equal upper
halves that it puts in order in place: one long run or several among distinct
upper halves, a little shorter and longer than the rule allows."""
from __future__ import annotations

import numpy as np
import pytest

import bulk_b200
from tests.gpu_util import NP, dev, host

pytestmark = pytest.mark.gpu


def _keys(tag, n, runs, order, rng):
    upper = rng.permutation(n).astype(np.uint64) + np.uint64(0x3FF00000)  # as f64: finite, positive
    low = rng.integers(0, 1 << 32, n, dtype=np.uint64)
    places = rng.permutation(n)
    at = 0
    for i, length in enumerate(runs):
        p = np.sort(places[at:at + length])
        at += length
        upper[p] = np.uint64(0x3FF80000 + i)
        if order == "descending":
            low[p] = np.arange(p.size, 0, -1, dtype=np.uint64) // np.uint64(2)  # pairs tie
        elif order == "equal":
            low[p] = np.uint64(7)
    k = (upper << np.uint64(32)) | low
    if tag == "f64":
        k[::37] = np.uint64(1) << np.uint64(63)
        k[1::37] = np.uint64(0)  # the two zeros tie
    elif tag == "i64":
        k[::2] |= np.uint64(1) << np.uint64(63)
    return k.view(NP[tag])


@pytest.mark.parametrize("order", ["random", "descending", "equal"])
@pytest.mark.parametrize("key,value", [("u64", "u32"), ("i64", "u64"), ("f64", None)])
def test_runs_in_one_cta(cuda, key, value, order):
    rng = np.random.default_rng(21)
    for n in (70, 1000, 1024, 1025, 2048, 2049, 3001, 4096):
        for runs in ([2], [33], [63], [64], [65], [66], [200], [64] * 3, [60, 70], [n // 2], [32] * (n // 64), [5] * (n // 6),
                     [7] * (n // 8)):
            runs = [r for r in runs if r <= n // 2] or [n // 2]
            keys = _keys(key, n, runs, order, rng)
            want = np.argsort(keys, kind="stable")
            if value is None:
                got = host(bulk_b200.stable_sort_by_key(dev(keys)))
            else:
                vals = np.arange(n, dtype=NP[value])
                got, gv = (host(t) for t in bulk_b200.stable_sort_by_key(dev(keys), dev(vals)))
                assert np.array_equal(gv, vals[want]), (n, runs)
            assert got.tobytes() == keys[want].tobytes(), (n, runs)
