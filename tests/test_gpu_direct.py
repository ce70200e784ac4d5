"""Calls whose compaction follows the numeric phase without a wait: products on
both sides of the size where that ends, with no entry to drop, some, all, and
with errors found by the numeric phase."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu


def blocks(products, cols, value=None, seed=0):
    """A: one column per entry, 4 to a row; B: 16 entries per row over `cols` columns."""
    rng = np.random.default_rng(seed)
    rows = products // 64
    a = sg.Csr.from_arrays(rows, 256, np.arange(rows + 1) * 4, rng.integers(0, 256, rows * 4), rng.uniform(-1, 1, rows * 4))
    if cols == 16 * 256:  # rows without a common column
        bcol = np.arange(16 * 256)
        a = sg.Csr.from_arrays(rows, 256, np.arange(rows + 1) * 4,
                               np.stack([rng.permutation(256)[:4] for _ in range(512)])[rng.integers(0, 512, rows)].ravel(), a.val)
    else:
        bcol = rng.integers(0, cols, 16 * 256)
    val = rng.uniform(-1, 1, 16 * 256) if value is None else np.full(16 * 256, value)
    b = sg.Csr.from_arrays(256, cols, np.arange(257) * 16, bcol, val)
    return a, b


@pytest.mark.parametrize("products", [64, 6400, (1 << 22) - 64, 1 << 22, (1 << 22) + 64])
@pytest.mark.parametrize("cols,value", [(16 * 256, None), (40, None), (40, 0.0)])
def test_direct(port, products, cols, value):
    a, b = blocks(products, cols, value)
    want = port.serial_spgemm(a, b)
    with sg.Engine(0) as eng:
        assert eng.scalar_multiplication_count(a, b) == products
        for _ in range(2):
            got = eng.multiply(a, b)
            assert csr_bits_equal(got, want), explain_diff(got, want)
            dev = eng.multiply(a, b, out="device")
            got = dev.download()
            dev.free()
            assert csr_bits_equal(got, want), explain_diff(got, want)


def test_error_in_numeric_phase(port):
    a, b = blocks(64000, 40)
    col = b.col.copy()
    col[777] = 40
    with sg.Engine(0) as eng:
        for out in ("host", "device"):
            with pytest.raises(sg.SpgError) as e:
                eng.multiply(a, sg.Csr(b.rows, b.cols, b.row_ptr, col, b.val), out=out)
            assert e.value.name == "SPG_INVALID_ARGUMENT"
            got, want = eng.multiply(a, b), port.serial_spgemm(a, b)
            assert csr_bits_equal(got, want), explain_diff(got, want)


def test_accumulate_stages(port):
    stages = [blocks(1 << 18, 16 * 256, seed=s) for s in range(3)]
    with sg.Engine(0) as eng:
        got = eng.accumulate(stages[0][0].rows, 16 * 256, stages)
    want = port.accumulate(stages[0][0].rows, 16 * 256, stages)
    assert csr_bits_equal(got, want), explain_diff(got, want)
