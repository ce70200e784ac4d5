"""Device memory that a handle keeps between calls: results stay intact while
later calls of other sizes run and blocks are handed back and reused, across
handles, threads and host or device results; and the memory goes back."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import spgemm_gb300 as sg
from helpers import csr_bits_equal, explain_diff

pytestmark = pytest.mark.gpu


def operand(n, seed):
    return sg.synth_uniform(n, n, 2, 30, seed=seed)


def test_results_outlive_later_calls(port):
    sizes = [3000, 200, 5000, 3000, 1, 800, 5000, 3001, 64]
    mats = [operand(n, n) if n > 30 else sg.Csr.from_arrays(1, 1, [0, 1], [0], [2.0]) for n in sizes]
    want = [port.serial_spgemm(a, a) for a in mats]
    with sg.Engine(0) as e1, sg.Engine(0, mode="exact") as e2:
        dev = [m.to_device() for m in mats]
        held = []
        for rnd in range(3):
            for i, a in enumerate(dev):
                held.append((i, (e1 if (i + rnd) % 2 else e2).multiply(a, a, out="device")))
                if len(held) > 5:  # the oldest are checked and freed while the others live
                    j, r = held.pop(0)
                    got = r.download()
                    r.free()
                    assert csr_bits_equal(got, want[j]), explain_diff(got, want[j])
        for j, r in held:
            got = r.download()
            assert csr_bits_equal(got, want[j]), explain_diff(got, want[j])


def test_result_freed_by_another_handle(port):
    a = operand(2000, 5)
    want = port.serial_spgemm(a, a)
    with sg.Engine(0) as e1, sg.Engine(0) as e2:
        for _ in range(6):
            r = e1.multiply(a, a, out="device")
            assert sg.library().spg_result_free(e2.h, sg.C.byref(r._res)) == 0
            r._res = None
            keep = [e.multiply(a, a, out="device") for e in (e2, e1, e2)]
            for k in keep:
                got = k.download()
                assert csr_bits_equal(got, want), explain_diff(got, want)
        r = e1.multiply(a, a, out="device")
        sg.library().spg_csr_release(sg.C.byref(r._res))  # without a handle
        r._res = None
        got = e1.multiply(a, a)
        assert csr_bits_equal(got, want), explain_diff(got, want)


def test_handles_on_threads(port):
    mats = [operand(n, n + 1) for n in (500, 1500, 2500, 4000)]
    want = [port.serial_spgemm(a, a) for a in mats]
    bad = []

    def work(k):
        with sg.Engine(0) as eng:
            for r in range(12):
                i = (k + r) % len(mats)
                got = eng.multiply(mats[i], mats[i])
                if not csr_bits_equal(got, want[i]):
                    bad.append((k, r))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_memory_goes_back_with_the_handle():
    import torch
    a = sg.synth_uniform(200_000, 200_000, 20, 20, seed=3).to_device()
    with sg.Engine(0) as eng:
        eng.multiply(a, a, out="device").free()
    first = None
    for _ in range(4):  # handle after handle: what one kept serves the next through the pool
        with sg.Engine(0) as eng:
            eng.multiply(a, a, out="device").free()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        first = free if first is None else first
        assert free > first - (512 << 20)
