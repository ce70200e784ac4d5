"""Device memory of a product copied to the host in row blocks: the blocks' results,
all held until the last copy ends, take their entries and little more, however many
products share an entry."""
from __future__ import annotations

import pytest

import alloc_shim
import spgemm_gb300 as sg

pytestmark = pytest.mark.gpu


def peak_of(shim):
    import numpy as np
    rows, per_row, inner, width, cols = 1 << 19, 8, 64, 48, 40
    rng = np.random.default_rng(1)
    a = sg.Csr.from_arrays(rows, inner, np.arange(rows + 1) * per_row, rng.integers(0, inner, rows * per_row),
                           rng.uniform(-1, 1, rows * per_row))
    b = sg.Csr.from_arrays(inner, cols, np.arange(inner + 1) * width, rng.integers(0, cols, inner * width),
                           rng.uniform(-1, 1, inner * width))
    rp, ci, va = np.empty(rows + 1, np.int64), np.empty(rows * cols, np.int32), np.empty(rows * cols)
    with sg.Engine(0) as eng:
        want = eng.multiply(a, b)
        shim.start()
        before = shim.stats()["held"]
        nnz = eng.multiply_to_host(a, b, rp, ci, va)
        peak = shim.stats()["peak"]
    same = np.array_equal(rp, want.row_ptr) and np.array_equal(ci[:nnz], want.col) and np.array_equal(va[:nnz], want.val)
    operands = sum(8 * (m.rows + 1) + 12 * m.nnz for m in (a, b))
    return [peak - before - operands, nnz, rows * per_row * width, rows, bool(same)]


def test_peak(tmp_path):
    extra, nnz, products, rows, same = alloc_shim.run(tmp_path, "test_gpu_to_host_memory", "peak_of")
    assert same
    block = products // 8 + (1 << 16)
    # held results, those written without knowing their size (2^25 products in all), a
    # block's own arrays before and after its compaction, per-row arrays
    assert extra <= 12 * nnz + 12 * (1 << 25) + 24 * block + 64 * rows + (64 << 20), extra
