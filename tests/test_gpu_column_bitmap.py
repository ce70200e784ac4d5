"""Exact layout: distinct columns counted in a bitmap or in a hash table, by the
columns of B and the products of a row: both sides of every line, columns that
follow one another and columns spread out."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu

# products of a row: every kernel, at the sizes where its table doubles
PRODUCTS = [1, 32, 33, 64, 65, 512, 513, 1024, 1025, 2048, 2049, 4097, 8192, 8193, 16384, 16385, 70000]


def operands(cols, spread, seed):
    rng = np.random.default_rng(seed)
    brows, width = 3000, min(64, cols)
    rows = []
    for p in PRODUCTS * 2:
        full = p // width
        rows.append(np.concatenate([rng.integers(0, brows - 1, full), np.full(p - full * width, brows - 1)]))
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    a = sg.Csr.from_arrays(len(rows), brows, rp, np.concatenate(rows), rng.uniform(-1, 1, rp[-1]))
    lens = np.full(brows, width)
    lens[-1] = 1
    brp = np.concatenate([[0], np.cumsum(lens)])
    if spread:
        col = rng.integers(0, cols, brp[-1])
    else:
        col = np.concatenate([s + np.arange(n) for s, n in zip(rng.integers(0, cols - width + 1, brows), lens)])
    b = sg.Csr.from_arrays(brows, cols, brp, col, rng.uniform(-1, 1, brp[-1]))
    return a, b


@pytest.mark.parametrize("cols", [1, 31, 33, 2048, 2049, 32 * 1024, 32 * 1024 + 1, 131071, 131073, 1 << 20, (1 << 20) + 1,
                                  1 << 30])
@pytest.mark.parametrize("spread", [True, False])
def test_exact_counts(port, cols, spread):
    a, b = operands(cols, spread, cols % 1000 + spread)
    want = port.serial_spgemm(a, b)
    with sg.Engine(0, mode="exact") as eng:
        got = eng.multiply(a, b)
        assert csr_bits_equal(got, want), explain_diff(got, want)


def test_batch_of_widths(port):
    pairs = [operands(c, True, c % 7) for c in (40, 1 << 21, 5000)]
    with sg.Engine(0, mode="exact") as eng:
        for got, (a, b) in zip(eng.multiply_batch(pairs), pairs):
            want = port.serial_spgemm(a, b)
            assert csr_bits_equal(got, want), explain_diff(got, want)
