"""Rows of at most 64 products whose entries mostly meet empty rows of B: the sizes
on both sides of the rule that gives a warp several of them."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [9727, 9728, 20_000])
@pytest.mark.parametrize("entries,width,share", [(16, 1, 0.8), (40, 1, 0.3), (64, 4, 0.15), (65, 4, 0.15), (300, 1, 0.05),
                                                 (1500, 1, 0.01)])
def test_mostly_empty_segments(engine, port, rows, entries, width, share):
    rng = np.random.default_rng(entries + rows)
    inner = 4000
    lens = (rng.random(inner) < share) * width
    brp = np.concatenate([[0], np.cumsum(lens)])
    b = sg.Csr.from_arrays(inner, 9000, brp, rng.integers(0, 9000, brp[-1]), rng.uniform(-1, 1, brp[-1]))
    a = sg.Csr.from_arrays(rows, inner, np.arange(rows + 1) * entries, rng.integers(0, inner, rows * entries),
                           rng.uniform(-1, 1, rows * entries))
    want = port.serial_spgemm(a, b)
    for mode in ("upper_bound", "exact"):
        with sg.Engine(0, mode=mode) as eng:
            got = eng.multiply(a, b)
        assert csr_bits_equal(got, want), explain_diff(got, want)
