"""Device memory of a transpose: besides its operand and its result, 20 bytes per
entry at most, whatever the number of its passes (12 column bits: two, 17: three,
25: four)."""
from __future__ import annotations

import numpy as np
import pytest

import alloc_shim
import spgemm_gb300 as sg

pytestmark = pytest.mark.gpu


def peak_of(shim, rows, cols, nnz):
    rng = np.random.default_rng(1)
    rp = np.linspace(0, nnz, rows + 1).astype(np.int64)
    a = sg.Csr.from_arrays(rows, cols, rp, rng.integers(0, cols, nnz), rng.uniform(-1, 1, nnz))
    with sg.Engine(0) as eng:
        shim.start()
        t = eng.transpose(a)
        peak = shim.stats()["peak"]
    order = np.argsort(a.col, kind="stable")
    row_of = np.repeat(np.arange(rows), np.diff(rp))
    same = np.array_equal(t.col, row_of[order]) and np.array_equal(t.val, a.val[order])
    return [peak, bool(same)]


@pytest.mark.parametrize("cols", [200, 4000, 70_000, 20_000_000])
def test_scratch_per_entry(tmp_path, cols):
    rows, nnz = 5000, 1 << 23
    peak, same = alloc_shim.run(tmp_path, "test_gpu_transpose_memory", "peak_of", rows, cols, nnz)
    assert same
    operand, result = 12 * nnz + 8 * (rows + 1), 12 * nnz + 8 * (cols + 1)
    tables = 8 * 256 * (nnz // 4096 + 1) + cols // 256 * 8 + (1 << 20)  # digit counts of every tile, sums of the scans
    blocks = 2 << 20  # a block's rounding
    assert peak <= operand + result + 20 * nnz + tables + 8 * blocks, (peak - operand - result) / nnz
