"""Compaction of rows written with holes where rows of more slots than a warp
takes stand among short and empty ones, singly and in a batch."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu

# scalar products of the long rows: about the line (4096), a CTA's step (2048 slots) and its multiples
LONG = [4095, 4096, 4097, 6143, 6144, 6145, 8192, 8193, 20480, 100001]


def operands(shorts, seed, cols):
    """Rows of exactly LONG products, each after `shorts` short rows: B's rows
    0-3999 hold one entry each, row 4000 + k holds 64."""
    rng = np.random.default_rng(seed)
    rows = []
    for n in LONG:
        rows += [rng.integers(0, 4000, rng.integers(0, 4)) for _ in range(shorts)]
        rows.append(np.concatenate([4000 + rng.integers(0, 500, n // 64), rng.integers(0, 4000, n % 64)]))
    rows += [rows[-1], rows[0]]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    a = sg.Csr.from_arrays(len(rows), 4500, rp, np.concatenate(rows), rng.uniform(-1, 1, rp[-1]))
    brp = np.concatenate([np.arange(4000), 4000 + 64 * np.arange(501)])
    b = sg.Csr.from_arrays(4500, cols, brp, rng.integers(0, cols, brp[-1]), rng.uniform(-1, 1, brp[-1]))
    return a, b


@pytest.mark.parametrize("shorts", [0, 1, 40, 600])
@pytest.mark.parametrize("cols", [3000, 2_000_000])
def test_long_rows_among_short(engine, port, shorts, cols):
    a, b = operands(shorts, shorts + cols, cols)
    got, want = engine.multiply(a, b), port.serial_spgemm(a, b)
    assert csr_bits_equal(got, want), explain_diff(got, want)


def test_long_rows_in_batch(engine, port):
    pairs = [operands(s, s, 5000) for s in (70, 0, 3)]
    for got, (a, b) in zip(engine.multiply_batch(pairs), pairs):
        want = port.serial_spgemm(a, b)
        assert csr_bits_equal(got, want), explain_diff(got, want)
