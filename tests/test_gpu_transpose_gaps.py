"""Transposes of operands with long stretches of empty rows: the rows of a sort
tile (4,096 entries) are walked while they are few and searched for above that;
both sides of the line, and the time of a stretch inside a tile against the same
stretch between two tiles."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff
from test_gpu_transpose import stable_transpose

pytestmark = pytest.mark.gpu


def with_gaps(lens, gaps, cols, seed):
    """Rows of lens[i] entries, each followed by gaps[i] empty rows."""
    rng = np.random.default_rng(seed)
    counts = np.zeros(len(lens) + int(np.sum(gaps)), np.int64)
    counts[np.arange(len(lens)) + np.concatenate([[0], np.cumsum(gaps)[:-1]])] = lens
    rp = np.concatenate([[0], np.cumsum(counts)])
    return sg.Csr.from_arrays(len(counts), cols, rp, rng.integers(0, cols, rp[-1]), rng.uniform(-1, 1, rp[-1]))


@pytest.mark.parametrize("gap", [16_384, 32_766, 32_767, 32_768, 32_769, 100_000, 3_000_000])
@pytest.mark.parametrize("lens", [[1, 1], [4095, 1], [4096, 1], [1, 4096], [3000, 3000, 3000], [1] * 40])
def test_rows_across_gaps(engine, gap, lens):
    gaps = [0] * len(lens)
    gaps[len(lens) // 2 - 1] = gap
    gaps[-1] = 5
    a = with_gaps(lens, gaps, 70_000, gap + len(lens))
    got, want = engine.transpose(a), stable_transpose(a)
    assert csr_bits_equal(got, want), explain_diff(got, want)


@pytest.mark.parametrize("per_entry", [4, 25])
def test_many_rows_of_few_entries(engine, per_entry):
    # every tile's rows are 4 or 25 times its entries
    a = with_gaps(np.ones(20_000, np.int64), np.full(20_000, per_entry - 1), 300, 3)
    got, want = engine.transpose(a), stable_transpose(a)
    assert csr_bits_equal(got, want), explain_diff(got, want)


def test_gap_inside_a_tile_costs_no_more(engine):
    import torch

    def best(a):
        d = a.to_device()
        times = []
        for _ in range(7):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            stream = torch.cuda.ExternalStream(engine.stream)
            start.record(stream)
            r = engine.transpose(d, out="device")
            end.record(stream)
            end.synchronize()
            r.free()
            times.append(start.elapsed_time(end))
        return min(times)

    # 20 M empty rows after 4,096 entries (a tile's end) and after 2,000 of them
    between = best(with_gaps([4096, 904], [20_000_000, 0], 1000, 1))
    inside = best(with_gaps([2000, 3000], [20_000_000, 0], 1000, 1))
    assert inside < 3 * between, (inside, between)
