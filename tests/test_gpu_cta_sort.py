"""Rows of 513-8,192 products (one per CTA: buckets, then each warp's share
settled in registers) at the edges of the bins, of the packed words and of the
bucket size that the register step takes, bit for bit against the serial
reference product (spgemm_common.cpp:131-178)."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu

CAPS = [512, 768, 1024, 1536, 2048, 3072, 4096, 6144, 8192]


def product_of(columns):
    """A and B whose output row i has the products' columns columns[i], in order:
    B rows of 1-64 entries, unsorted."""
    rng = np.random.default_rng(len(columns))
    alen, blen = [], []
    for c in columns:
        lens = []
        while sum(lens) < len(c):
            lens.append(int(min(rng.integers(1, 65), len(c) - sum(lens))))
        alen.append(len(lens))
        blen += lens
    a = sg.Csr.from_arrays(len(columns), len(blen), np.concatenate([[0], np.cumsum(alen)]), np.arange(len(blen)),
                           rng.uniform(-1, 1, len(blen)))
    ncols = int(max(c.max() for c in columns)) + 1
    b = sg.Csr.from_arrays(len(blen), ncols, np.concatenate([[0], np.cumsum(blen)]), np.concatenate(columns),
                           rng.uniform(-1, 1, int(np.sum(blen))))
    return a, b


def check(engine, port, columns):
    a, b = product_of(columns)
    got, want = engine.multiply(a, b), port.serial_spgemm(a, b)
    assert csr_bits_equal(got, want), explain_diff(got, want)


@pytest.fixture(scope="module", params=["upper_bound", "exact"])
def eng(request):
    with sg.Engine(0, mode=request.param) as e:
        yield e


@pytest.mark.parametrize("bits", [3, 12, 18, 19, 20, 22, 24, 30])
def test_bin_edges(eng, port, bits):
    # sequence numbers take 10-13 bits: rows of 18-24 bits fit packed words as a
    # whole, share by share, or not at all
    rng = np.random.default_rng(bits)
    columns = []
    for p in sorted({513, *(c + d for c in CAPS for d in (-1, 0, 1) if 512 < c + d <= 8192)}):
        c = rng.integers(0, 1 << bits, size=p)
        c[:2] = 0, (1 << bits) - 1
        columns.append(c)
    check(eng, port, columns)


@pytest.mark.parametrize("bits", [20, 28])
def test_dense_and_sparse_parts(eng, port, bits):
    # most products in a narrow band, the rest anywhere; and all but one in a band
    rng = np.random.default_rng(bits + 100)
    columns = []
    for p in (700, 1000, 1500, 2000, 3000, 4000, 6000, 8000):
        for sparse in (p // 3, 1):
            c = (1 << bits) // 3 + rng.integers(0, max(p // 2, 64), size=p)
            c[rng.choice(p, sparse, replace=False)] = rng.integers(0, 1 << bits, size=sparse)
            columns.append(c)
    check(eng, port, columns)


@pytest.mark.parametrize("repeat", [2, 31, 32, 33, 64, 600])
def test_repeated_columns(eng, port, repeat):
    # some columns repeated `repeat` times, among them the first and the last; 33
    # is one above what the register step takes
    rng = np.random.default_rng(repeat)
    columns = []
    for p in (640, 1024, 1300, 2048, 2500, 4096, 5000, 8192):
        c = rng.permutation(1 << 20)[:p]
        at = rng.permutation(p)
        for i, col in enumerate((0, (1 << 20) - 1, 12345)):
            c[at[i * repeat:(i + 1) * repeat][:p]] = col
        columns.append(c)
    columns.append(np.full(900, 7))
    check(eng, port, columns)
