"""GPU parity of the merge where its splits are found in different ways: by
the loader warp (few tiles a CTA) and by the partition kernel (many), with
inputs whose splits run along either array's edge."""
from __future__ import annotations

import numpy as np
import pytest

import bulk_b200
from tests.gpu_util import NP, dev, host

pytestmark = pytest.mark.gpu

GRID = 3 * 148  # CTAs of a B200's full grid


def _arrays(tag, na, nb, kind, rng):
    if kind == "a first":
        a, b = np.arange(na), np.arange(na, na + nb)
    elif kind == "b first":
        a, b = np.arange(nb, nb + na), np.arange(nb)
    elif kind == "ties":
        a, b = np.zeros(na), np.zeros(nb)
    elif kind == "blocks":  # long stretches of one array, then of the other
        a = np.sort(rng.integers(0, 64, na)) * 2.0
        b = np.sort(rng.integers(0, 64, nb)) * 2.0 + 1
    else:
        a, b = np.sort(rng.integers(0, 1 << 24, na)), np.sort(rng.integers(0, 1 << 24, nb))
    return a.astype(NP[tag]), b.astype(NP[tag])


@pytest.mark.parametrize("kind", ["random", "a first", "b first", "ties", "blocks"])
@pytest.mark.parametrize("key,value,tile,many", [("f32", None, 4096, 17), ("i32", "u32", 4096, 17), ("u64", None, 2048, 17),
                                                 ("f64", "u32", 2048, 9), ("u32", "u64", 4096, 17)])
def test_splits(cuda, key, value, tile, many, kind):
    rng = np.random.default_rng(3)
    totals = [tile * GRID - 1, tile * GRID + 1, tile * GRID * 2 + 7, tile * GRID * 5 // 2]
    if kind in ("random", "blocks"):
        totals.append(tile * GRID * many + 5)
    for total in totals:
        for na in (total // 2, 3, total - 1):
            nb = total - na
            a, b = _arrays(key, na, nb, kind, rng)
            both = np.concatenate([a, b])
            order = np.argsort(both, kind="stable")
            if value is None:
                got = host(bulk_b200.merge(dev(a), dev(b)))
                assert np.array_equal(got, both[order]), (total, na)
            else:
                vals = np.arange(total, dtype=NP[value])
                gk, gv = bulk_b200.merge(dev(a), dev(b), dev(vals[:na]), dev(vals[na:]))
                assert np.array_equal(host(gk), both[order]) and np.array_equal(host(gv), vals[order]), (total, na)
            assert bulk_b200.workspace_status() == 0
