"""Calls on a device whose memory runs out: with every allocation failing in turn,
once or from there on, a call gives its result bit for bit or SPG_OUT_OF_MEMORY, the
handle's next call is right, and nothing stays allocated behind the handle; and what
fits without arrays of the upper bound's size for C does not fail for want of them."""
from __future__ import annotations

import numpy as np
import pytest

import alloc_shim
import spgemm_gb300 as sg
from helpers import csr_bits_equal, random_csr, row_sizes_for_bins
from test_gpu_result_sizes import compressed

pytestmark = pytest.mark.gpu
ME = "test_gpu_out_of_memory"


def operands():
    a, b = row_sizes_for_bins(5)  # every bin, heavy rows too
    c, d = random_csr(400, 300, 9, 1), random_csr(300, 350, 7, 2)
    return (a, b), (c, d), compressed(500, 16, 16, 40, 3)


def call_of(kind, eng):
    """A call's results as host matrices."""
    (a, b), (c, d), (e, f) = operands()

    def device(r):
        m = r.download()
        r.free()
        return m

    def to_host(x, y):
        p = sg.scalar_products_host(x, y)
        rp, ci, va = np.empty(x.rows + 1, np.int64), np.empty(max(p, 1), np.int32), np.empty(max(p, 1))
        n = eng.multiply_to_host(x, y, rp, ci, va)
        return [sg.Csr(x.rows, y.cols, rp, ci[:n], va[:n])]

    return {
        "bins": lambda: [device(eng.multiply(a, b, out="device"))],
        "small": lambda: [device(eng.multiply(e, f, out="device")), eng.multiply(c, d)],
        "batch": lambda: [device(r) for r in eng.multiply_batch([(a, b), (c, d), (e, f)], out="device")],
        "batch_host": lambda: eng.multiply_batch([(c, d), (e, f)]),
        "accumulate": lambda: [eng.accumulate(500, 40, [(e, f), (e, f.scaled(0.5)), (e, f)])],
        "to_host": lambda: to_host(a, b),
        "transpose": lambda: [eng.transpose(b), device(eng.transpose(d, out="device"))],
    }[kind]


def sweep(shim, kind, mode):
    outcomes = {"ok": 0, "oom": 0}
    with sg.Engine(0, mode=mode) as eng:
        want = call_of(kind, eng)()
    for lasting in (1, 1 << 40):
        for warm in (False, True):  # the handle keeps blocks from a call before
            n = 0
            while True:
                shim.start()
                base = shim.stats()["held"]
                with sg.Engine(0, mode=mode) as eng:
                    call = call_of(kind, eng)
                    if warm:
                        call()
                    shim.start(n, lasting)
                    try:
                        got = call()
                    except sg.SpgError as e:
                        got = None
                        assert e.name == "SPG_OUT_OF_MEMORY", (kind, mode, n, e)
                    failed = shim.stats()["failed"]
                    shim.start()
                    assert got is None or all(csr_bits_equal(x, y) for x, y in zip(got, want)), (kind, mode, n)
                    assert all(csr_bits_equal(x, y) for x, y in zip(call(), want)), (kind, mode, n, "next call")
                assert shim.stats()["held"] == base, (kind, mode, n, "left behind")
                if not failed:
                    break
                outcomes["ok" if got is not None else "oom"] += 1
                n += 1
    return outcomes


@pytest.mark.parametrize("mode", ["auto", "exact", "upper_bound"])
@pytest.mark.parametrize("kind", ["bins", "small", "batch", "batch_host", "accumulate", "to_host", "transpose"])
def test_every_allocation_failing(tmp_path, kind, mode):
    outcomes = alloc_shim.run(tmp_path, ME, "sweep", kind, mode)
    assert outcomes["oom"] > 0
    if mode == "auto" and kind in ("bins", "small", "accumulate", "to_host"):
        assert outcomes["ok"] > 0  # the exact layout, or the kept blocks given back


def plans(shim):
    """Plan creation with every allocation failing; the handle after it."""
    import torch
    torch.zeros(1, device="cuda")
    (a, b), (c, d), _ = operands()
    seen = 0
    with sg.Engine(0) as eng:
        want = [eng.multiply(a, b), eng.multiply(c, d)]
        pairs = [(a.to_device(), b.to_device()), (c.to_device(), d.to_device())]
        n = 0
        while True:
            shim.start(n, 1 << 40)
            try:
                plan = eng.plan(pairs)
            except sg.SpgError as e:
                assert e.name == "SPG_OUT_OF_MEMORY", e
                plan = None
                seen += 1
            shim.start()
            assert csr_bits_equal(eng.multiply(c, d), want[1])
            if plan is not None:
                plan.execute()
                assert all(csr_bits_equal(plan.result(i), w) for i, w in enumerate(want))
                plan.close()
                return seen
            n += 1


def test_plans(tmp_path):
    assert alloc_shim.run(tmp_path, ME, "plans") > 5


def tight(shim, out):
    """A product of 4.1 M products into 64,000 entries where C_tmp fits, a second set of
    that size does not."""
    a, b = compressed(2000, 64, 32, 32, 1)
    products, res = 2000 * 64 * 32, []
    with sg.Engine(0) as eng:
        want = eng.multiply(a, b)
    for mode in ("upper_bound", "auto"):
        with sg.Engine(0, mode=mode) as eng:
            shim.limit(12 * products + (12 << 20))
            r = eng.multiply(a, b, out=out)
            got = r.download() if out == "device" else r
            shim.limit()
            res.append(bool(csr_bits_equal(got, want)))
    return res


@pytest.mark.parametrize("out", ["device", "host"])
def test_direct_results_are_not_needed(tmp_path, out):
    assert all(alloc_shim.run(tmp_path, ME, "tight", out))
