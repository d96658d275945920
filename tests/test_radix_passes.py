"""GPU parity of the sort's global-memory radix passes at the sizes where their
tiling turns: tile and group edges, more groups than one look-back round
reads, partly filled groups, and digit distributions from one value to all."""
from __future__ import annotations

import numpy as np
import pytest

import bulk_b200
from tests.gpu_util import NP, dev, host

pytestmark = pytest.mark.gpu

# keys a tile, as csrc/radix_sort.cu chooses them by bytes a pair; four tiles a group (two in ragged batches)
TILE = {8: 416 * 16, 12: 288 * 16, 16: 288 * 12}


def _keys(tag, n, kind, rng):
    if kind == "one":
        return np.full(n, 3, dtype=NP[tag])
    if kind == "few":
        return rng.integers(0, 5, n).astype(NP[tag])
    if kind == "sorted":
        return np.arange(n).astype(NP[tag])
    if tag in ("f32", "f64"):
        return rng.standard_normal(n).astype(NP[tag])
    info = np.iinfo(NP[tag])
    return rng.integers(info.min, info.max, n, dtype=NP[tag], endpoint=True)


def _check(keys, vals, gk, gv):
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(host(gk), keys[order]), keys.size
    if vals is not None:
        assert np.array_equal(host(gv), vals[order]), keys.size


@pytest.mark.parametrize("kind", ["full", "few", "one", "sorted"])
@pytest.mark.parametrize("key,value", [("u32", "u32"), ("i32", None), ("f32", "u64"), ("u64", "u32"), ("f64", "u64")])
def test_tile_and_group_edges(cuda, key, value, kind):
    size = np.dtype(NP[key]).itemsize + (np.dtype(NP[value]).itemsize if value else 0)
    t = TILE[max(size, 8)]
    first = 131073 // t + 1  # below, one cluster launch sorts the array
    sizes = [first * t - 1, first * t, first * t + 1, 4 * first * t + 1, 4 * 33 * t - 1, 4 * 33 * t + t, 4 * 80 * t + 5]
    rng = np.random.default_rng(5)
    for n in sizes:
        keys = _keys(key, n, kind, rng)
        vals = np.arange(n, dtype=NP[value]) if value else None
        if value is None:
            _check(keys, None, bulk_b200.stable_sort_by_key(dev(keys)), None)
        else:
            _check(keys, vals, *bulk_b200.stable_sort_by_key(dev(keys), dev(vals)))
        assert bulk_b200.workspace_status() == 0


@pytest.mark.parametrize("key,value", [("u32", "u32"), ("i64", "u64")])
@pytest.mark.parametrize("many", [False, True])
def test_batches_with_full_and_ragged_groups(cuda, key, value, many):
    t = TILE[8 if key == "u32" else 16]
    sizes = [40 * t, 400 * t + 1, 3 * t] if not many else [2, t - 1, t, t + 1, 2 * t, 2 * t + 1, 9 * t, 1, 0, 100 * t] * 3
    rng = np.random.default_rng(6)
    keys = [_keys(key, n, "few" if i % 3 == 2 else "full", rng) for i, n in enumerate(sizes)]
    vals = [np.arange(n, dtype=NP[value]) for n in sizes]
    src_k, src_v = [dev(k) for k in keys], [dev(v) for v in vals]
    out_k, out_v = bulk_b200.stable_sort_by_key_copy_batch(src_k, src_v)
    for k, v, gk, gv, sk in zip(keys, vals, out_k, out_v, src_k):
        _check(k, v, gk, gv)
        assert np.array_equal(host(sk), k)
    assert bulk_b200.workspace_status() == 0
