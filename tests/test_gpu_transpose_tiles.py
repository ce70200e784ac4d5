"""Transposes at the edges of the sort's tiles (4,096 entries) and of its passes
(one per 8 column bits), against a stable host sort by column; malformed
operands are refused."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff
from test_gpu_transpose import stable_transpose

pytestmark = pytest.mark.gpu


def matrix(rows, cols, nnz, seed, empty=0.5):
    """Rows of very different lengths, a share of them empty (first and last too)."""
    rng = np.random.default_rng(seed)
    cuts = rng.integers(0, nnz + 1, size=max(int(rows * (1 - empty)) - 1, 0))
    starts = np.sort(rng.choice(np.concatenate([cuts, np.zeros(1, int), np.full(1, nnz)]), size=rows - 1)) if rows > 1 else []
    rp = np.concatenate([[0], starts, [nnz]]).astype(np.int64)
    col = rng.integers(0, cols, size=nnz)
    if nnz:
        col[0], col[-1] = cols - 1, 0
    return sg.Csr.from_arrays(rows, cols, rp, col, rng.uniform(-1, 1, nnz))


@pytest.mark.parametrize("cols", [1, 2, 256, 257, 65536, 65537, (1 << 24) + 3])
@pytest.mark.parametrize("nnz", [1, 4095, 4096, 4097, 30000])
def test_tiles_and_passes(engine, cols, nnz):
    for rows in (1, 3, 20000):
        a = matrix(rows, cols, nnz, rows + nnz + cols)
        got, want = engine.transpose(a), stable_transpose(a)
        assert csr_bits_equal(got, want), explain_diff(got, want)


def test_long_stretch_of_empty_rows(engine):
    # one tile whose rows lie 400,000 empty rows apart
    rp = np.zeros(400_003, np.int64)
    rp[2:], rp[400_002:] = 1000, 5000
    a = sg.Csr.from_arrays(400_002, 90_000, rp, np.random.default_rng(1).integers(0, 90_000, 5000), np.arange(5000.0))
    got, want = engine.transpose(a), stable_transpose(a)
    assert csr_bits_equal(got, want), explain_diff(got, want)


def test_malformed_operands_are_refused(engine):
    a = matrix(500, 70_000, 9000, 4)
    for at, bad in ((0, -1), (8999, 70_000), (4096, 1 << 30)):
        col = a.col.copy()
        col[at] = bad
        with pytest.raises(sg.SpgError) as e:
            engine.transpose(sg.Csr(a.rows, a.cols, a.row_ptr, col, a.val))
        assert e.value.name == "SPG_INVALID_ARGUMENT"
    rp = a.row_ptr.copy()
    rp[250] = rp[251] + 1
    with pytest.raises(sg.SpgError) as e:
        engine.transpose(sg.Csr(a.rows, a.cols, rp, a.col, a.val))
    assert e.value.name == "SPG_INVALID_ARGUMENT"
