"""The items of a batched call are packed in one go: the bytes must be what
the C structs (their ctypes mirrors) hold, init values converted as C does."""
from __future__ import annotations

import struct

import pytest

from bulk_b200 import batch


@pytest.mark.parametrize("tag", ["i32", "u32", "i64", "u64", "f32", "f64"])
@pytest.mark.parametrize("init", [0, 7, -1, -(1 << 31), (1 << 32) - 1, (1 << 63), 1e40, float("inf"), 0.1])
def test_scan_items(tag, init):
    item = batch.scan_item_type(tag)()
    try:
        item.d_in, item.d_out, item.n, item.init = 0x1111, 0x2222, 33, init
    except TypeError:
        with pytest.raises(TypeError):
            batch._init_value(tag, init)
        return
    assert struct.pack("=3Q" + batch._INIT_CODE[tag], 0x1111, 0x2222, 33, batch._init_value(tag, init)) == bytes(item)


def test_pair_items():
    rbk = batch.rbk_item_type("i32", "f32")(1, 2, 3, 4, 5, 6)
    assert struct.pack("=6Q", 1, 2, 3, 4, 5, 6) == bytes(rbk)
    sort = batch.sort_item_type("u32", "u32")(1, 2, 3)
    assert struct.pack("=3Q", 1, 2, 3) == bytes(sort)
    copy = batch.sort_copy_item_type("u32", "u32")(1, 2, 3, 4, 5)
    assert struct.pack("=5Q", 1, 2, 3, 4, 5) == bytes(copy)
