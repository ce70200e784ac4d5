"""Short rows whose segments of B hold one entry or none, alone, beside longer
segments and after an addend, with enough rows for several per warp."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu

ROWS = 24_000  # above 64 rows per SM in either bin


def operands(lo, hi, b_lens, cols, seed):
    rng = np.random.default_rng(seed)
    lens = rng.integers(lo, hi + 1, ROWS)
    rp = np.concatenate([[0], np.cumsum(lens)])
    a = sg.Csr.from_arrays(ROWS, 4000, rp, rng.integers(0, 4000, rp[-1]), rng.uniform(-1, 1, rp[-1]))
    blen = rng.choice(b_lens, 4000)
    brp = np.concatenate([[0], np.cumsum(blen)])
    b = sg.Csr.from_arrays(4000, cols, brp, rng.integers(0, cols, brp[-1]), rng.uniform(-1, 1, brp[-1]))
    return a, b


@pytest.mark.parametrize("lo,hi", [(1, 32), (31, 33), (33, 64), (64, 64)])
@pytest.mark.parametrize("b_lens", [[1], [0, 1], [1] * 60 + [2], [0, 0, 0, 1]])
@pytest.mark.parametrize("cols", [50, 1 << 30])
def test_single_entries(engine, port, lo, hi, b_lens, cols):
    a, b = operands(lo, hi, b_lens, cols, lo + len(b_lens))
    got, want = engine.multiply(a, b), port.serial_spgemm(a, b)
    assert csr_bits_equal(got, want), explain_diff(got, want)


def test_single_entries_after_addend(engine, port):
    stages = [operands(4, 8, [0, 1], 60, s) for s in range(3)]
    got = engine.accumulate(ROWS, 60, stages)
    want = port.accumulate(ROWS, 60, stages)
    assert csr_bits_equal(got, want), explain_diff(got, want)


def test_bad_column_in_single_entry(engine):
    a, b = operands(32, 32, [1], 50, 3)
    col = b.col.copy()
    col[17] = 50
    with pytest.raises(sg.SpgError) as e:
        engine.multiply(a, sg.Csr(b.rows, b.cols, b.row_ptr, col, b.val))
    assert e.value.name == "SPG_INVALID_ARGUMENT"
