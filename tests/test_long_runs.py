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
