"""What a handle holds of the device between calls: little whatever it multiplied,
never more than its budget, no array of a result larger than asked for; and a slow
allocation of one handle keeps no other waiting."""
from __future__ import annotations

import threading
import time

import pytest

import alloc_shim
import spgemm_gb300 as sg

pytestmark = pytest.mark.gpu
ME = "test_gpu_handle_memory"


def idle_after(shim, mode):
    """Bytes held by an idle handle after products of several sizes."""
    held = []
    with sg.Engine(0, mode=mode) as eng:
        shim.start()
        for n in (200_000, 1000, 50_000, 120_000):
            a = sg.synth_uniform(n, n, 16, 24, seed=n)
            eng.multiply(a, a, out="device").free()
            eng.multiply(a, a)
            eng.transpose(a, out="device").free()
            held.append(shim.stats()["held"])
        eng.accumulate(1000, 1000, [(sg.synth_uniform(1000, 1000, 5, 9, seed=i),) * 2 for i in range(3)])
        held.append(shim.stats()["held"])
    return held + [shim.stats()["held"]]


@pytest.mark.parametrize("mode", ["auto", "exact"])
def test_idle_handle_keeps_little(tmp_path, mode):
    *idle, closed = alloc_shim.run(tmp_path, ME, "idle_after", mode)
    assert max(idle) <= 128 << 20, idle
    assert closed == 0


def budgeted(shim, budget):
    out = []
    with sg.Engine(0, hbm_budget_bytes=budget) as eng:
        shim.start()
        for n in (9000, 3000, 700, 8000, 40, 5000, 9500):
            a = sg.synth_uniform(n, n, 4, 12, seed=n)
            r = eng.multiply(a, a, out="device")
            sizes = [shim.size(p) for p in r.pointers]
            want = [8 * (n + 1), 4 * r.nnz, 8 * r.nnz]
            full = r.nnz == r.products
            r.free()
            out.append([sizes, want, full, shim.stats()["held"]])
    return out


def test_budget_bounds_what_is_kept(tmp_path):
    budget = 24 << 20
    for sizes, want, full, held in alloc_shim.run(tmp_path, ME, "budgeted", budget):
        assert held <= budget
        assert not full
        assert sizes == want


def handed_over(shim):
    """Sizes of the arrays of results that need no compaction."""
    import numpy as np
    out = []
    with sg.Engine(0) as eng:
        for n in (5000, 4900, 100_000, 70_000):
            d = sg.Csr.from_arrays(n, n, np.arange(n + 1), np.arange(n), np.ones(n))
            b = sg.synth_uniform(n, n, 3, 9, seed=n)
            for _ in range(2):
                r = eng.multiply(d, b, out="device")
                out.append([[shim.size(p) for p in r.pointers], [8 * (n + 1), 4 * r.nnz, 8 * r.nnz], r.nnz == r.products])
                r.free()
    return out


def test_arrays_handed_over_have_their_size(tmp_path):
    for sizes, want, full in alloc_shim.run(tmp_path, ME, "handed_over"):
        assert full
        assert all(w <= s <= w + max(w // 8, 512) for s, w in zip(sizes, want)), (sizes, want)


def beside_a_slow_one(shim):
    """Longest call of a handle with small products while another handle's large
    allocations take 400 ms each."""
    big, small = sg.synth_uniform(100_000, 100_000, 16, 16, seed=1), sg.synth_uniform(200, 200, 4, 8, seed=2)
    with sg.Engine(0) as e1, sg.Engine(0) as e2:
        e1.multiply(small, small)
        e2.multiply(small, small)
        shim.slow(50 << 20, 400)
        other = threading.Thread(target=lambda: e1.multiply(big, big, out="device").free())
        t0 = time.perf_counter()
        other.start()
        longest = 0.0
        while other.is_alive():
            t = time.perf_counter()
            e2.multiply(small, small)
            longest = max(longest, time.perf_counter() - t)
        return [longest, time.perf_counter() - t0]


def test_no_waiting_for_another_handles_allocation(tmp_path):
    longest, slow = alloc_shim.run(tmp_path, ME, "beside_a_slow_one")
    assert slow > 0.8
    assert longest < 0.2
