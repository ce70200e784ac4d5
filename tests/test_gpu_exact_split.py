"""Rows above 8,192 products in the exact layout: where memory allows they are
split by column range, written to slots and moved to their counted places, else
run whole.  Bit for bit against the serial reference product
(spgemm_common.cpp:131-178), alone, in a batch, with zero sums and with rows that
cannot be split."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu


def heavy_product(seed, ncols=30000, rows=24):
    """Output rows of 8,193-40,000 products between short ones; every fifth repeats
    one column more often than a piece holds; some sums cancel."""
    rng = np.random.default_rng(seed)
    nb = 3000
    blen = rng.integers(1, 40, size=nb)
    brp = np.concatenate([[0], np.cumsum(blen)])
    bcol = rng.integers(0, ncols, size=int(brp[-1]))
    bcol[brp[:-1]] = np.where(rng.random(nb) < 0.5, 11, bcol[brp[:-1]])
    bval = rng.integers(-3, 4, size=len(bcol)).astype(float)  # whole numbers: sums that are exactly zero
    b = sg.Csr.from_arrays(nb, ncols, brp, bcol, bval)
    cols, arp = [], [0]
    for r in range(2 * rows):
        if r % 2:
            k = rng.integers(0, nb, size=int(rng.integers(0, 30)))
        elif r % 10 == 0:
            k = rng.choice(np.nonzero(bcol[brp[:-1]] == 11)[0], size=4500)  # over 4,096 products in column 11
        else:
            k = rng.integers(0, nb, size=int(rng.integers(450, 1900)))
        cols.append(k)
        arp.append(arp[-1] + len(k))
    a = sg.Csr.from_arrays(2 * rows, nb, arp, np.concatenate(cols), rng.integers(-2, 3, size=arp[-1]).astype(float))
    return a, b


@pytest.mark.parametrize("rows", [1, 3, 24, 200])
def test_heavy_rows(port, rows):
    a, b = heavy_product(rows, rows=rows)
    want = port.serial_spgemm(a, b)
    with sg.Engine(0, mode="exact") as eng:
        for _ in range(2):
            got = eng.multiply(a, b)
            assert csr_bits_equal(got, want), explain_diff(got, want)


def test_heavy_rows_in_a_batch(port):
    pairs = [heavy_product(s, ncols=n, rows=12) for s, n in ((5, 9000), (6, 1 << 21), (7, 20000))]
    with sg.Engine(0, mode="exact") as eng:
        for (a, b), got in zip(pairs, eng.multiply_batch(pairs)):
            want = port.serial_spgemm(a, b)
            assert csr_bits_equal(got, want), explain_diff(got, want)


def test_budget_that_fits_whole_rows_only(port):
    # the whole rows' slabs take 40 x 24 bytes x the largest row's products (about 70
    # MB); a budget between the two ways' footprints is served as before
    a, b = heavy_product(9, rows=40)
    want = port.serial_spgemm(a, b)
    served = 0
    for mib in (1, 16, 64, 72, 80, 96, 112, 128, 160, 256):
        with sg.Engine(0, mode="exact", hbm_budget_bytes=mib << 20) as eng:
            try:
                got = eng.multiply(a, b)
            except sg.SpgError as e:
                assert e.name == "SPG_BUDGET_EXCEEDED" and served == 0
                continue
            served += 1
            assert csr_bits_equal(got, want), explain_diff(got, want)
    assert served >= 2
