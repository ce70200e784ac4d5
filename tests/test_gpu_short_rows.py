"""Products of many rows of at most 64 products, which run several to a warp, bit
for bit against the serial reference product (spgemm_common.cpp:131-178), with an
addend (matrix_blocks.cpp:152-200) and with a bad column among them."""
from __future__ import annotations

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu


def short_rows(rows, most, ncols, seg, seed):
    """Output rows of 1 to `most` products; B rows of 0 to `seg` entries, unsorted,
    columns repeated."""
    rng = np.random.default_rng(seed)
    nb = 4000
    blen = rng.integers(0, seg + 1, size=nb)
    blen[0] = 1
    blen[1] = 0
    brp = np.concatenate([[0], np.cumsum(blen)])
    bcol = np.where(rng.random(int(brp[-1])) < 0.3, rng.integers(0, 5, int(brp[-1])), rng.integers(0, ncols, int(brp[-1])))
    bcol[:2] = 0, ncols - 1
    b = sg.Csr.from_arrays(nb, ncols, brp, bcol, rng.uniform(-1, 1, len(bcol)))
    entries, arp = [], [0]
    for r in range(rows):
        want = int(rng.integers(1, most + 1)) if r % 7 else most
        cols, got = [], 0
        while got < want:
            k = int(rng.integers(0, nb))
            if got + blen[k] > want:
                k = int(rng.integers(0, 2))  # one product, or none
            cols.append(k)
            got += blen[k]
        entries += cols
        arp.append(len(entries))
    a = sg.Csr.from_arrays(rows, nb, arp, entries, rng.uniform(-1, 1, len(entries)))
    return a, b


@pytest.mark.parametrize("mode", ["upper_bound", "exact"])
@pytest.mark.parametrize("most,seg,bits", [(32, 1, 20), (32, 9, 27), (32, 32, 30), (64, 7, 21), (64, 64, 26), (64, 3, 30)])
def test_short_rows(port, mode, most, seg, bits):
    # 32-product rows leave the packed words 27 bits, 64-product rows 26
    a, b = short_rows(25013, most, 1 << bits, seg, seed=most + seg + bits)
    with sg.Engine(0, mode=mode) as eng:
        got = eng.multiply(a, b)
    want = port.serial_spgemm(a, b)
    assert csr_bits_equal(got, want), explain_diff(got, want)


def test_short_rows_with_addend_and_batch(engine, port):
    pairs = [short_rows(21003, m, 1 << 18, s, seed=m + s) for m, s in ((20, 4), (30, 6), (24, 2))]
    rows, cols = pairs[0][0].rows, pairs[0][1].cols
    got = engine.accumulate(rows, cols, pairs)
    want = port.accumulate(rows, cols, pairs)
    assert csr_bits_equal(got, want), explain_diff(got, want)
    for (a, b), c in zip(pairs, engine.multiply_batch(pairs)):
        want = port.serial_spgemm(a, b)
        assert csr_bits_equal(c, want), explain_diff(c, want)


def test_bad_column_is_refused(engine):
    a, b = short_rows(25000, 32, 1000, 5, seed=3)
    for bad in (-1, b.cols):
        col = b.col.copy()
        col[int(b.row_ptr[2])] = bad
        with pytest.raises(sg.SpgError) as e:
            engine.multiply(a, sg.Csr(b.rows, b.cols, b.row_ptr, col, b.val))
        assert e.value.name == "SPG_INVALID_ARGUMENT"
