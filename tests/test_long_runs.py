"""GPU parity of the planned sort of 8-byte keys where one run of keys with
equal upper halves is too long to be sorted in place and is out of order at one
place alone: two sorted tables put one after the other.  The place is swept over
a warp's chunk of 256 keys and over the run, wherever in a chunk the run begins."""
from __future__ import annotations

import pytest
import torch

import bulk_b200

pytestmark = pytest.mark.gpu

N = 1 << 22  # the smallest planned array
CHUNK = 256


class _OneRun:
    """N shuffled keys, distinct in their upper halves but for the run at sorted positions [at, at + length)."""

    def __init__(self, tag, value, at, length, cuda):
        g = torch.Generator(device=cuda).manual_seed(at)
        upper = torch.arange(N, dtype=torch.int64, device=cuda)
        upper[at:at + length] = at
        if tag == "i64":
            upper -= N // 2  # both signs
        elif tag == "f64":
            upper += 0x3FF00000  # finite, positive
        self.sorted = (upper << 32) | 5
        at_input = torch.randperm(N, generator=g, device=cuda)  # sorted position i is input element at_input[i]
        at_input[at:at + length] = at_input[at:at + length].sort().values  # the run's keys in input order
        self.keys = torch.empty_like(self.sorted)
        self.keys[at_input] = self.sorted
        self.at_input = at_input
        self.vals = None if value is None else torch.arange(N, device=cuda).to(value)
        self.dtype = {"u64": torch.uint64, "i64": torch.int64, "f64": torch.float64}[tag]
        self.run = slice(at, at + length)
        self.high = int(upper[at]) << 32

    def check(self, low):
        """Sorts with the run's lower halves, in input order, being `low`."""
        keys, want = self.keys.clone(), self.sorted.clone()
        keys[self.at_input[self.run]] = self.high + low
        order = torch.sort(low, stable=True).indices
        want[self.run] = self.high + low[order]
        if self.vals is None:
            got = bulk_b200.stable_sort_by_key(keys.view(self.dtype))
        else:
            got, vals = bulk_b200.stable_sort_by_key(keys.view(self.dtype), self.vals.clone())
            want_at = self.at_input.clone()
            want_at[self.run] = want_at[self.run][order]
            assert torch.equal(vals, want_at.to(vals.dtype))
        assert torch.equal(got.view(torch.int64), want)


def _one_break(length, at, cuda):
    """Ascending, but for one descent before element `at`."""
    low = torch.arange(length, device=cuda)
    low[:at] += 1000
    low[at:] -= at
    return low


@pytest.mark.parametrize("start", [0, 1, 63, 64, 65, 100, 255])
@pytest.mark.parametrize("tag,value", [("u64", torch.int32), ("u64", None), ("i64", torch.int64), ("f64", torch.int32)])
def test_one_descent_in_a_long_run(cuda, tag, value, start):
    length = 400
    case = _OneRun(tag, value, 1000 * CHUNK + start, length, cuda)
    edges = (0, 1, 63, 64, 65, 255)
    for at in range(1, length):
        if (tag == "u64" and value is not None) or (start + at) % CHUNK in edges:
            try:
                case.check(_one_break(length, at, cuda))
            except AssertionError:
                raise AssertionError(f"{tag} {value}: run from {start}, descent at {at}") from None
    assert bulk_b200.workspace_status() == 0


@pytest.mark.parametrize("length", [63, 64, 65, 66])
def test_runs_about_as_long_as_the_longest_sorted_in_place(cuda, length):
    for start in (100, 190, 200, 255):  # inside a chunk, up to its end, over it
        case = _OneRun("u64", torch.int32, 1000 * CHUNK + start, length, cuda)
        for at in range(1, length):
            case.check(_one_break(length, at, cuda))
    assert bulk_b200.workspace_status() == 0


def _outside_the_sample(n, cuda):
    """The positions that the sample (rs_sample_kernel: 32 windows of 65,536 keys) does not read."""
    outside = torch.ones(n, dtype=torch.bool, device=cuda)
    for cta in range(32):
        h = (cta + 1) * 0x9E3779B1 % (1 << 32)
        h = (h ^ h >> 15) * 0x85EBCA6B % (1 << 32)
        h = (h ^ h >> 13) * 0xC2B2AE35 % (1 << 32)
        h ^= h >> 16
        window = h * (n - 65536) >> 32
        outside[window:window + 65536] = False
    return outside.nonzero()[:, 0]


def _check_runs(tag, value, runs, cuda, low_bits=32, n=N, unseen=False):
    """Runs of the given lengths at random places (unseen: that the sample does not read) among keys of distinct
    upper halves, lower halves random."""
    g = torch.Generator(device=cuda).manual_seed(len(runs) + runs[0])
    upper = torch.randperm(n, device=cuda, generator=g)
    low = torch.randint(0, 1 << low_bits, (n,), device=cuda, generator=g)
    places = _outside_the_sample(n, cuda) if unseen else torch.arange(n, device=cuda)
    places = places[torch.randperm(places.numel(), device=cuda, generator=g)]
    lengths = torch.tensor(runs, device=cuda)
    members = places[:int(lengths.sum())]
    assert members.numel() == int(lengths.sum())
    upper[members] = torch.repeat_interleave(n + torch.arange(len(runs), device=cuda) * 3, lengths)
    if tag == "i64":
        upper -= n
    elif tag == "f64":
        upper += 0x3FF00000
    keys = (upper << 32) | low
    if tag == "f64":  # a run at zero: the two zeros tie, the least numbers share their upper half
        zero = places[-300:]
        keys[zero[:100]] = -(1 << 63)
        keys[zero[100:200]] = 0
        keys[zero[200:]] = low[zero[200:]]
    dtype = {"u64": torch.uint64, "i64": torch.int64, "f64": torch.float64}[tag]
    want, order = torch.sort(keys.view(torch.float64) if tag == "f64" else keys, stable=True)
    want = keys[order]
    if value is None:
        got = bulk_b200.stable_sort_by_key(keys.clone().view(dtype))
    else:
        got, vals = bulk_b200.stable_sort_by_key(keys.clone().view(dtype), torch.arange(n, device=cuda).to(value))
        assert torch.equal(vals, order.to(value)), (runs[:3], len(runs))
    assert torch.equal(got.view(torch.int64), want), (runs[:3], len(runs))
    assert bulk_b200.workspace_status() == 0


@pytest.mark.parametrize("tag,value", [("u64", torch.int32), ("i64", None), ("f64", torch.int64)])
def test_runs_sorted_by_a_warp_or_a_cta(cuda, tag, value):
    # a warp's, around its last key and its rounds of 128; a CTA's, around a warp's share, a tile and several
    for length in (65, 66, 67, 68, 127, 128, 129, 255, 256, 257, 511, 513, 8191, 8192, 8193, 16385, 50_000):
        _check_runs(tag, value, [length], cuda)
        _check_runs(tag, value, [length], cuda, low_bits=1)
    _check_runs(tag, value, [65, 9000, 70, 8192, 300, 20_000, 66, 256, 257], cuda)
    _check_runs(tag, value, [131_071, 66], cuda, unseen=True)
    _check_runs(tag, value, [131_072, 5000, 5000], cuda, unseen=True)


@pytest.mark.parametrize("tag,value", [("u64", torch.int32), ("i64", None), ("f64", torch.int64)])
def test_longer_and_more_runs_than_those(cuda, tag, value):
    _check_runs(tag, value, [131_073], cuda, unseen=True)
    _check_runs(tag, value, [300_000, 100], cuda, unseen=True)
    n = 1 << 24
    _check_runs(tag, value, [258] * 30_000, cuda, n=n, unseen=True)
    tile = 3456 if value == torch.int64 else 4608  # the list: a word a digit and group of four tiles, less one in 256 keys
    room = (n + 4 * tile - 1) // (4 * tile) * 256 - n // 256
    for count in (10_000, room - 1, room, room + 1):
        if count * 65 < 14_000_000:
            _check_runs(tag, value, [65] * count, cuda, n=n, unseen=True)
