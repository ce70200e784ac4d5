"""Device memory that a kept result takes: no more than twice its entries, or 1 MiB
more than them, however many scalar products share an entry."""
from __future__ import annotations

import numpy as np
import pytest

import alloc_shim
import spgemm_gb300 as sg
from helpers import csr_bits_equal

pytestmark = pytest.mark.gpu


def compressed(rows, per_row, width, cols, seed):
    """rows x rows products of per_row * width products a row into `cols` columns."""
    rng = np.random.default_rng(seed)
    a = sg.Csr.from_arrays(rows, 64, np.arange(rows + 1) * per_row, rng.integers(0, 64, rows * per_row),
                           rng.uniform(-1, 1, rows * per_row))
    b = sg.Csr.from_arrays(64, cols, np.arange(65) * width, rng.integers(0, cols, 64 * width), rng.uniform(-1, 1, 64 * width))
    return a, b


# rows, entries a row of A, of B, columns: 4 M products into 64 K, 1 M, 2.1 M entries; few
# products; no entry at all
SHAPES = [(2000, 64, 32, 32), (2000, 64, 32, 512), (2000, 64, 32, 2048), (130, 16, 8, 4), (2000, 64, 32, 40)]


def sizes_of(shim):
    from oracle import build as obuild
    from oracle.oracle import Port
    obuild.build_oracle()
    port, out = Port(), []
    with sg.Engine(0) as eng:
        for i, s in enumerate(SHAPES):
            a, b = compressed(*s, seed=i)
            if i == 4:
                b.val[:] = 0.0
            want = port.serial_spgemm(a, b)
            for _ in range(2):
                r = eng.multiply(a, b, out="device")
                same = csr_bits_equal(r.download(), want)
                out.append([sum(shim.size(p) for p in r.pointers[1:]), r.nnz, r.products, bool(same)])
                r.free()
    return out


def test_kept_results(tmp_path):
    for held, nnz, products, same in alloc_shim.run(tmp_path, "test_gpu_result_sizes", "sizes_of"):
        assert same
        assert products <= 1 << 22
        assert held <= 12 * nnz + max(12 * nnz, 1 << 20) + 1024, (held, nnz, products)
