"""GPU parity of scan and reduce_by_key around the sizes up to which they run
as one cluster that clears its own status words: every tile count from one to
nine, full and ragged last tiles, on a workspace that other calls have used."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import bulk_b200
import oracle
from tests.gpu_util import assert_within_bound, dev, gen, host

pytestmark = pytest.mark.gpu


def _dirty(cuda):
    """Leave other algorithms' scratch where the status words will lie."""
    k = torch.randint(-(1 << 31), 1 << 31, (200_003,), device=cuda, dtype=torch.int64).to(torch.int32)
    bulk_b200.stable_sort_by_key(k, k.clone())


@pytest.mark.parametrize("tag,tile", [("i32", 8192), ("f32", 8192), ("i64", 4096), ("f64", 4096)])
def test_scan(cuda, tag, tile):
    for tiles in range(1, 10):
        for n in (tile * tiles - 1, tile * tiles):
            x = gen(tag, n, tiles)
            _dirty(cuda)
            got = host(bulk_b200.inclusive_scan(dev(x)))
            if tag[0] == "f":
                assert_within_bound(got, np.cumsum(x.astype(np.longdouble)), np.cumsum(np.abs(x.astype(np.float64))), n,
                                    x.dtype, f"n={n}")
            else:
                assert np.array_equal(got, np.cumsum(x, dtype=x.dtype)), n
            assert bulk_b200.workspace_status() == 0


@pytest.mark.parametrize("key,value,tile", [("i32", "i32", 4096), ("i64", "i64", 2048)])
def test_reduce_by_key(cuda, key, value, tile):
    for tiles in range(1, 10):
        for n in (tile * tiles - 1, tile * tiles):
            keys = oracle.gen_runs_geometric(n, tiles, 16.0).astype(np.int32 if key == "i32" else np.int64)
            vals = gen(value, n, 50 + tiles)
            _dirty(cuda)
            gk, gv, count = bulk_b200.reduce_by_key(dev(keys), dev(vals))
            starts = np.flatnonzero(np.r_[True, keys[1:] != keys[:-1]])
            assert count == starts.size
            assert np.array_equal(host(gk), keys[starts])
            assert np.array_equal(host(gv), np.add.reduceat(vals, starts))
            assert bulk_b200.workspace_status() == 0
