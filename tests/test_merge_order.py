"""GPU parity of the merge where the source of its splits and the order of its
tiles change: few tiles a CTA (the loader finds the splits) and many (a partition
kernel does), interleaved tiles and runs of them."""
from __future__ import annotations

import pytest
import torch

import bulk_b200

pytestmark = pytest.mark.gpu

SMS = 148
SIGNED = {"i32": torch.int32, "u32": torch.int32, "f32": torch.float32, "i64": torch.int64, "u64": torch.int64,
          "f64": torch.float64}
CASES = [("i32", None), ("f32", "u32"), ("u32", "u64"), ("u64", None), ("f64", "u32"), ("i64", "u64")]


def _view(t, tag):
    return t.view({"u32": torch.uint32, "u64": torch.uint64}[tag]) if tag in ("u32", "u64") else t


def _keys(tag, n, top, g, cuda):
    """Sorted and non-negative, so that their signed and unsigned orders agree."""
    return torch.randint(0, top, (n,), device=cuda, generator=g, dtype=torch.int32).sort().values.to(SIGNED[tag])


def _shifted(t, off):
    y = torch.empty(t.numel() + off, dtype=t.dtype, device=t.device)[off:]
    return y.copy_(t)


def check_merge(tag, value, na, nb, top, cuda, offsets=(0, 0, 0, 0, 0)):
    g = torch.Generator(device=cuda).manual_seed(na + nb)
    a, b = _keys(tag, na, top, g, cuda), _keys(tag, nb, top, g, cuda)
    want, order = torch.sort(torch.cat([a, b]), stable=True)
    out = _view(_shifted(torch.zeros_like(want), offsets[4]), tag)
    a, b = _view(_shifted(a, offsets[0]), tag), _view(_shifted(b, offsets[1]), tag)
    if value is None:
        bulk_b200.merge(a, b, out=out)
    else:
        dt = torch.int32 if value == "u32" else torch.int64
        vals = torch.arange(na + nb, device=cuda, dtype=dt)
        out_vals = torch.empty_like(vals)
        bulk_b200.merge(a, b, _shifted(vals[:na], offsets[2]), _shifted(vals[na:], offsets[3]), out=out,
                        out_vals=out_vals)
        assert torch.equal(out_vals, order.to(dt)), (na, nb)
    assert torch.equal(out.view(SIGNED[tag]), want), (na, nb)
    assert bulk_b200.workspace_status() == 0


@pytest.mark.parametrize("per_cta", [8, 16, 32])
@pytest.mark.parametrize("key,value", CASES)
def test_tiles_a_cta(cuda, key, value, per_cta):
    tile = 4096 if key[1:] == "32" else 2048
    grid = SMS * (2 if key == "u32" and value == "u64" else 3)
    for total in (tile * grid * per_cta - 1, tile * (grid * per_cta - 1), tile * (grid * per_cta + 1) + 3):
        check_merge(key, value, total // 3, total - total // 3, 1 << 30, cuda)
        check_merge(key, value, total - 1000, 1000, 1 << 30, cuda)
