"""Row work (products per row, input checks) for rows of A from empty to much
longer than the average, against the reference's scalarMultiplicationCount
(spgemm_common.cpp:474-487) and serial product, and its errors
(spgemm_common.cpp:141-143)."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu

# lengths at the edges of 4 and 8 lanes with four entries each, and of the warp's steps
EDGES = [0, 1, 3, 4, 5, 15, 16, 17, 31, 32, 33, 143, 144, 145, 159, 160, 161, 5000]


def operands(mean, seed):
    rng = np.random.default_rng(seed)
    lens = np.concatenate([EDGES, rng.integers(0, 2 * mean + 1, size=700), EDGES[::-1]])
    rp = np.concatenate([[0], np.cumsum(lens)])
    a = sg.Csr.from_arrays(len(lens), 900, rp, rng.integers(0, 900, rp[-1]), rng.uniform(-1, 1, rp[-1]))
    blen = rng.integers(0, 4, 900)
    brp = np.concatenate([[0], np.cumsum(blen)])
    b = sg.Csr.from_arrays(900, 700, brp, rng.integers(0, 700, brp[-1]), rng.uniform(-1, 1, brp[-1]))
    return a, b


@pytest.mark.parametrize("mean", [2, 60])
def test_counts_and_product(engine, port, mean):
    a, b = operands(mean, mean)
    assert engine.scalar_multiplication_count(a, b) == sg.scalar_products_host(a, b)
    got, want = engine.multiply(a, b), port.serial_spgemm(a, b)
    assert csr_bits_equal(got, want), explain_diff(got, want)


@pytest.mark.parametrize("mean", [2, 60])
@pytest.mark.parametrize("bad", [-1, 900])
def test_bad_column_anywhere(engine, mean, bad):
    a, b = operands(mean, mean)
    first = int(a.row_ptr[len(EDGES) - 1])  # the row of 5,000 entries
    for at in (first, first + 16, first + 47, first + 4999, a.nnz - 1):
        col = a.col.copy()
        col[at] = bad
        with pytest.raises(sg.SpgError) as e:
            engine.multiply(sg.Csr(a.rows, a.cols, a.row_ptr, col, a.val), b)
        assert e.value.name == "SPG_OUT_OF_RANGE_COLUMN"


def test_bad_offsets(engine):
    a, b = operands(2, 5)
    rp = b.row_ptr.copy()
    rp[450] = rp[-1] + 5
    with pytest.raises(sg.SpgError) as e:
        engine.multiply(a, sg.Csr(b.rows, b.cols, rp, b.col, b.val))
    assert e.value.name == "SPG_INVALID_ARGUMENT"
