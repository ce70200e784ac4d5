"""Rows whose columns repeat often (summed four products at a time): every run length
around a multiple of four, rows of every kernel, both layouts, sums that depend on
their order."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["upper_bound", "exact"])
@pytest.mark.parametrize("per_row,width", [(20, 20), (30, 30), (40, 30), (50, 50), (60, 60), (75, 70), (90, 80), (120, 100), (160, 110)])
@pytest.mark.parametrize("cols", [1, 3, 40])
def test_long_runs(port, mode, per_row, width, cols):
    rng = np.random.default_rng(per_row + cols)
    inner, rows = 300, 37
    far = rng.choice(2**31 - 1, cols, replace=False)  # columns too far apart for packed words
    for table, ncols in ((np.arange(cols), cols), (far, 2**31 - 1)):
        bcol = table[rng.integers(0, cols, inner * width)]
        b = sg.Csr.from_arrays(inner, ncols, np.arange(inner + 1) * width, bcol, rng.uniform(-1, 1, inner * width) * 10.0 ** rng.integers(-9, 9, inner * width))
        lens = per_row - rng.integers(0, 6, rows)
        arp = np.concatenate([[0], np.cumsum(lens)])
        a = sg.Csr.from_arrays(rows, inner, arp, rng.integers(0, inner, arp[-1]), rng.uniform(-1, 1, arp[-1]))
        want = port.serial_spgemm(a, b)
        with sg.Engine(0, mode=mode) as eng:
            got = eng.multiply(a, b)
        assert csr_bits_equal(got, want), explain_diff(got, want)


@pytest.mark.parametrize("mode", ["upper_bound", "exact"])
def test_every_run_length(port, mode):
    # rows of 800 products: runs of 33 and more beside runs of 1 to 13
    rng = np.random.default_rng(1)
    runs = np.concatenate([np.arange(1, 14), [33, 34, 35, 36, 37, 64, 65]])
    col = np.repeat(np.arange(len(runs)) * 7, runs)
    col = np.concatenate([col, 1000 + np.arange(800 - len(col))])
    rows = 40
    val = rng.uniform(-1, 1, (rows, 800)) * 10.0 ** rng.integers(-9, 9, (rows, 800))
    b = sg.Csr.from_arrays(rows, 3000, np.arange(rows + 1) * 800, np.concatenate([rng.permutation(col) for _ in range(rows)]),
                           val.ravel())
    a = sg.Csr.from_arrays(rows, rows, np.arange(rows + 1), np.arange(rows), np.ones(rows))
    want = port.serial_spgemm(a, b)
    with sg.Engine(0, mode=mode) as eng:
        got = eng.multiply(a, b)
    assert csr_bits_equal(got, want), explain_diff(got, want)
