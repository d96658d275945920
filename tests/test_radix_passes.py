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


# ---- 8-byte keys from 2^22 on: upper digits first, then the short runs that agree there
PLAN_MIN = 1 << 22


def _wide(tag, kind, n, rng):
    full = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    if kind == "runs of a few":      # about eight keys an upper half
        k = (rng.integers(0, n // 8, n, dtype=np.uint64) << np.uint64(32)) | (full & np.uint64(0xFF))
    elif kind == "few upper halves":  # the sample sends it to all eight passes
        k = (rng.integers(0, 1000, n, dtype=np.uint64) << np.uint64(40)) | (full & np.uint64(0xFFFFFF))
    elif kind in ("long run", "longest run"):  # too long to sort in place, too rare for the sample
        k = full.copy()
        at = n // 3 + (np.arange(400) if kind == "long run" else np.arange(256))
        k[at] = (np.uint64(77) << np.uint64(32)) | (full[at] & np.uint64(0xF))
    else:
        k = full
    if tag == "f64":
        k = k.copy()
        k[(k >> np.uint64(52) & np.uint64(0x7FF)) == 0x7FF] = 0x3FF0000000000000  # no NaN
        k[::1000] = 0x8000000000000000
        k[1::1000] = 0  # the two zeros tie
    return k.view(NP[tag])


@pytest.mark.parametrize("kind", ["full", "runs of a few", "few upper halves", "long run", "longest run"])
@pytest.mark.parametrize("key,value", [("u64", "u32"), ("i64", None), ("f64", "u64")])
def test_wide_keys_by_upper_digits(cuda, key, value, kind):
    rng = np.random.default_rng(7)
    for n in (PLAN_MIN, PLAN_MIN + 4097):
        keys = _wide(key, kind, n, rng)
        if value is None:
            _check(keys, None, bulk_b200.stable_sort_by_key(dev(keys)), None)
        else:
            vals = np.arange(n, dtype=NP[value])
            gk, gv = bulk_b200.stable_sort_by_key(dev(keys), dev(vals))
            _check(keys, vals, gk, gv)
            assert np.array_equal(host(gk).view(np.uint64), keys[np.argsort(keys, kind="stable")].view(np.uint64))
        assert bulk_b200.workspace_status() == 0
