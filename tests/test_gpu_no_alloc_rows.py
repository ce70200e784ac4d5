"""The allocation-free multiply takes as many rows as its scratch holds at 32 bytes a
row and a word per 4,096 rows, and refuses more than that by far."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from test_zz_no_alloc import noalloc, same

pytestmark = pytest.mark.gpu


def scratch(rows):
    """Bytes of control block, per-row arrays and one word per 4,096 rows."""
    used = 0
    for n in (192, 704, 16, 8 * rows, 8 * (rows + 1), 8 * (rows + 1), 8 * rows, 8 * ((rows + 4096) // 4096 + 1)):
        used = (used + 255) // 256 * 256 + n
    return used


def last_rows():
    lo, hi = 1, 1 << 21
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if scratch(mid) <= 32 << 20 else (lo, mid)
    return lo


def operand(rows, lens):
    rp = np.zeros(rows + 1, np.int64)
    rp[1:len(lens) + 1] = np.cumsum(lens)
    rp[len(lens) + 1:] = rp[len(lens)]
    rng = np.random.default_rng(rows)
    n = int(rp[-1])
    return sg.Csr.from_arrays(rows, 50, rp, rng.integers(0, 50, n), rng.uniform(-1, 1, n))


def test_most_rows():
    lib = sg.library()
    rows = last_rows()
    assert rows > 1_040_000
    a, b = operand(rows, [2]), sg.synth_uniform(50, 50, 1, 1, seed=2)
    st, nnz, err, out = noalloc(lib, a.to_device(), b.to_device(), 100)
    assert st == 0, err
    with sg.Engine(0) as eng:
        assert same(out, eng.multiply(a, b))
    more = operand(rows + 4096, [2])
    assert noalloc(lib, more.to_device(), b.to_device(), 100)[0] == 5  # SPG_BUDGET_EXCEEDED


@pytest.mark.parametrize("rows", [1, 2047, 2048, 2049, 4096, 4097, 100_000])
def test_offsets_across_scan_tiles(port, rows):
    lib = sg.library()
    rng = np.random.default_rng(rows)
    a = operand(rows, rng.integers(0, 4, rows))  # many rows empty, the sums of the scans' tiles in nz between
    b = sg.synth_uniform(50, 60, 1, 5, seed=2)
    want = port.serial_spgemm(a, b)
    for _ in range(2):
        st, nnz, err, out = noalloc(lib, a.to_device(), b.to_device(), want.nnz)
        assert st == 0, err
        assert same(out, want)
