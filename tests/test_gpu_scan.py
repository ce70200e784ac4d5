"""The prefix of the per-row products (K3) at the edges of its tiles and of its
one-, two- and three-launch forms, through spg_partition_rows, and the bin lists
(K1b) of a product with that many rows."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 2047, 2048, 2049, 4096, 4100, 300_001, 2048 * 2048, 2048 * 2048 + 1, 4_500_001])
def test_partition_follows_the_prefix(engine, rows):
    rng = np.random.default_rng(rows)
    lens = rng.integers(0, 3, size=rows)
    rp = np.concatenate([[0], np.cumsum(lens)])
    col = rng.integers(0, 3, size=int(rp[-1])).astype(np.int32)
    a = sg.Csr(rows, 3, rp.astype(np.int64), col, np.ones(len(col)))
    b = sg.Csr.from_arrays(3, 4, [0, 1, 3, 6], [0, 1, 2, 1, 2, 3], np.ones(6))
    prefix = np.concatenate([[0], np.cumsum(np.array([1, 2, 3])[col])])[rp]  # products before every row
    total, parts = int(prefix[-1]), 97
    got = engine.partition_rows(a, b, parts)
    if total == 0:
        want = [rows * k // parts for k in range(parts + 1)]
    else:
        want = [0] + [int(np.searchsorted(prefix, total * k // parts, side="left")) for k in range(1, parts)] + [rows]
    assert got.tolist() == want


@pytest.mark.parametrize("rows", [1023, 1024, 1025, 300_001])
def test_rows_of_every_bin_are_found(engine, port, rows):
    # row lengths mixed over the bins: every row must appear in its bin's list once
    rng = np.random.default_rng(rows)
    b = sg.Csr.from_arrays(6, 700, [0, 0, 1, 40, 140, 440, 1140],
                           np.concatenate([[5], *(rng.permutation(700)[:n] for n in (39, 100, 300, 700))]),
                           rng.uniform(-1, 1, 1140))
    col = rng.choice(6, size=rows, p=[0.3, 0.6, 0.09, 0.006, 0.003, 0.001])
    a = sg.Csr.from_arrays(rows, 6, np.arange(rows + 1), col, rng.uniform(-1, 1, rows))
    got, want = engine.multiply(a, b), port.serial_spgemm(a, b)
    assert csr_bits_equal(got, want), explain_diff(got, want)
