"""GPU parity of the small sorts: one CTA (up to 4096 keys) and one cluster
(tiles of 1024, 2048, 4096 and 8192 keys), at the sizes where they change, with
keys that share digits, halves or everything."""
from __future__ import annotations

import numpy as np
import pytest

import bulk_b200
from tests.gpu_util import NP, dev, host

pytestmark = pytest.mark.gpu

SIZES = [2, 31, 33, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097, 16384, 16385, 32767, 32769, 65536, 65537]


def _keys(tag, n, kind, rng):
    dt = NP[tag]
    if tag in ("f32", "f64"):
        k = rng.standard_normal(n).astype(dt)
        if kind == "few":
            k = np.round(k).astype(dt)
        elif kind == "one":
            k[:] = -2.5
        elif kind != "full":
            k[::3] = -0.0
            k[1::3] = 0.0  # the two zeros tie
        return k
    bits = 8 * np.dtype(dt).itemsize
    full = rng.integers(0, 1 << bits, n, dtype=np.uint64, endpoint=False) if bits == 32 else \
        rng.integers(0, (1 << 64) - 1, n, dtype=np.uint64, endpoint=True)
    if kind == "few":
        full = full % np.uint64(5)
    elif kind == "one":
        full[:] = np.uint64(77)
    elif kind == "same upper":  # differ in the lower half alone
        full = full & np.uint64(0xFFFF if bits == 32 else 0xFFFFFFFF)
    elif kind == "upper ties":  # few upper halves, lower halves out of order
        half = np.uint64(bits // 2)
        full = ((full % np.uint64(7)) << half) | (full >> half)
    return full.astype(dt)


@pytest.mark.parametrize("kind", ["full", "few", "one", "same upper", "upper ties"])
@pytest.mark.parametrize("key,value", [("u32", "u32"), ("i32", None), ("f32", "u64"), ("u64", "u32"), ("i64", "u64"),
                                       ("f64", None)])
def test_one_cta_and_one_cluster(cuda, key, value, kind):
    rng = np.random.default_rng(12)
    for n in SIZES:
        keys = _keys(key, n, kind, rng)
        order = np.argsort(keys, kind="stable")
        if value is None:
            gk = host(bulk_b200.stable_sort_by_key(dev(keys)))
        else:
            vals = np.arange(n, dtype=NP[value])
            gk, gv = (host(t) for t in bulk_b200.stable_sort_by_key(dev(keys), dev(vals)))
            assert np.array_equal(gv, vals[order]), n
        assert gk.tobytes() == keys[order].tobytes(), n


@pytest.mark.parametrize("key,value", [("u32", "u32"), ("i64", "u32")])
def test_batches_of_one_cta_each(cuda, key, value):
    rng = np.random.default_rng(13)
    for sizes in ([0, 1, 2, 900, 1024, 5], [2048, 3, 1500], [4096, 0, 1, 1, 2049, 31] * 20):
        keys = [_keys(key, n, ("full", "few", "upper ties")[i % 3], rng) for i, n in enumerate(sizes)]
        vals = [np.arange(n, dtype=NP[value]) for n in sizes]
        src = [dev(k) for k in keys]
        ok, ov = bulk_b200.stable_sort_by_key_copy_batch(src, [dev(v) for v in vals])
        for k, v, gk, gv, sk in zip(keys, vals, ok, ov, src):
            order = np.argsort(k, kind="stable")
            assert np.array_equal(host(gk), k[order]) and np.array_equal(host(gv), v[order]), k.size
            assert np.array_equal(host(sk), k)
