"""The serving loop charges an uncollected device result by its entries: its arrays
have that size, also when a bad request in the batch made its neighbours run alone."""
from __future__ import annotations

import pytest

import alloc_shim
import spgemm_gb300 as sg

pytestmark = pytest.mark.gpu


def sizes_beside_a_bad_request(shim):
    good = [sg.synth_uniform(n, n, 20, 30, seed=n) for n in (1000, 1500)]
    bad = (sg.Csr.from_arrays(2, 3, [0, 1, 2], [0, 1], [1.0, 1.0]),
           sg.Csr.from_arrays(3, 2, [0, 1, 2, 3], [0, 5, 0], [1.0, 1.0, 1.0]))  # column 5 of 2
    big = sg.synth_uniform(60_000, 60_000, 16, 16, seed=1)
    out = []
    with sg.Server(0, lanes=1, max_batch=16) as srv:
        first = srv.submit(big, big)  # the others queue up behind it
        tickets = [srv.submit(good[0], good[0]), srv.submit(*bad), srv.submit(good[1], good[1])]
        for t in [first] + tickets:
            st, res, info = srv.poll(t)
            if res is not None:
                r = res._res
                out.append([st, sum(shim.size(p) for p in (r.col, r.val)), 12 * r.nnz, r.products, info["batch_requests"]])
                res.free()
            else:
                out.append([st, 0, 0, 0, info["batch_requests"]])
    return out


def test_rerun_requests(tmp_path):
    big, one, bad, two = alloc_shim.run(tmp_path, "test_gpu_server_memory", "sizes_beside_a_bad_request")
    assert bad[0] == "SPG_INVALID_ARGUMENT"
    assert one[4] == bad[4] == two[4] == 3  # one batch
    for st, held, entries, products, _ in (one, two):
        assert st == "SPG_OK"
        assert entries < 12 * products
        assert held <= entries + 1024, (held, entries, products)
