"""Rows of at most 512 products (one per warp, sorted in registers) at the edges
of every bin and of the packed 32-bit (column, sequence) word, bit for bit
against the serial reference product (spgemm_common.cpp:131-178)."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu

CAPS = [32, 64, 96, 128, 192, 256, 384, 512]


def rows_of(sizes, ncols, lo, seed):
    """One output row per entry of `sizes`: A row i holds 1-7 entries whose B rows
    hold sizes[i] products in all, columns in [lo, ncols) with repeats, both
    ends of the range in every row of at least two products."""
    rng = np.random.default_rng(seed)
    alen, blen, bcol = [], [], []
    for p in sizes:
        k = int(min(p, rng.integers(1, 8)))
        cut = np.sort(rng.choice(np.arange(1, p), size=k - 1, replace=False)) if k > 1 else np.zeros(0, int)
        alen.append(k)
        blen += np.diff(np.concatenate([[0], cut, [p]])).tolist()
        c = rng.integers(lo, ncols, size=p)
        c[rng.integers(0, p, size=p // 4)] = c[0]  # repeated columns, out of order
        if p >= 2:
            c[0], c[-1] = lo, ncols - 1
        bcol.append(c)
    a = sg.Csr.from_arrays(len(sizes), len(blen), np.concatenate([[0], np.cumsum(alen)]), np.arange(len(blen)),
                           rng.uniform(-1, 1, len(blen)))
    b = sg.Csr.from_arrays(len(blen), ncols, np.concatenate([[0], np.cumsum(blen)]), np.concatenate(bcol),
                           rng.uniform(-1, 1, int(np.sum(blen))))
    return a, b


@pytest.mark.parametrize("bits", [4, 20, 22, 23, 24, 25, 26, 27, 28, 30])
def test_warp_rows_at_bin_edges(engine, port, bits):
    # sequence numbers take 5-9 bits: ranges of 23-27 bits fill the packed word at some capacity
    sizes = sorted({1, 2, 3, *(c + d for c in CAPS for d in (-1, 0, 1) if c + d <= 512)}) * 3
    for lo in (0, 5):
        a, b = rows_of(sizes, (1 << bits) + lo, lo, seed=bits + lo)
        got, want = engine.multiply(a, b), port.serial_spgemm(a, b)
        assert csr_bits_equal(got, want), explain_diff(got, want)
