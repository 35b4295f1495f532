"""A device allocation that fails half-way through a call leaves the graph as it was: the call
returns JGPM_ENOMEM, and the same call afterwards gives the exact result.  The failure is made on
the host (jgpm_fail_alloc_ refuses the k-th allocation), for every k that the call reaches."""
import ctypes

import numpy as np
import pytest

import oracle_api as O

pytestmark = pytest.mark.gpu

ENOMEM = -2
N, EF, SEED = 4096, 12, 9


def refuse(gpu, k):
    gpu.lib().jgpm_fail_alloc_(ctypes.c_int64(k))


@pytest.fixture(scope="module")
def sym():
    return O.rmat_graph(N, EF, 0.5, 0.2, 0.2, SEED)


CALLS = {
    "csr": lambda gpu, g: [x.tolist() for x in g.csr(dag=True)],
    "4-clique": lambda gpu, g: g.count("4-clique"),
    "diamond": lambda gpu, g: g.count("diamond"),
    "tailed triangle": lambda gpu, g: g.count("tailed-triangle", induced=True),
    "4-cycle": lambda gpu, g: g.count("4-cycle"),
    "P5": lambda gpu, g: g.count("P5"),
    "P9": lambda gpu, g: g.count("P9"),
    "census": lambda gpu, g: g.census4(),
    "batch": lambda gpu, g: gpu.batch_count([(g, p) for p in ("triangle", "diamond", "4-cycle")])[0],
}


@pytest.mark.parametrize("call", list(CALLS))
def test_call_after_a_failed_allocation(gpu, sym, call):
    run = CALLS[call]
    with gpu.Graph.from_csr(sym.rowptr, sym.col, use_dag=False) as g:
        want = run(gpu, g)
    failed = 0
    for k in range(64):
        with gpu.Graph.from_csr(sym.rowptr, sym.col, use_dag=False) as g:
            refuse(gpu, k)
            try:
                assert run(gpu, g) == want
                done = True
            except gpu.JgpmError as e:
                assert e.code == ENOMEM
                done = False
            finally:
                refuse(gpu, -1)
            failed += not done
            assert run(gpu, g) == want, k
        if done:
            break
    assert done and failed > 0


def test_served_graph_after_a_failed_restore(gpu, sym):
    """Two graphs in turn under a budget that holds one: every query restores the evicted one."""
    want = O.count("P13", O.orient(sym))[0]
    with gpu.Graph.from_csr(sym.rowptr, sym.col) as g:
        g.count("4-clique")
        size = g.info()["device_bytes"]
    s = gpu.Server(memory_budget_bytes=int(1.7 * size), max_inflight=1, max_batch=4)
    with s:
        ids = [s.add_graph(gpu.Graph.from_csr(sym.rowptr, sym.col)) for _ in range(2)]
        for k in range(24):
            refuse(gpu, k)
            try:
                assert s.wait(s.submit(ids[k & 1], "4-clique"), 20000)[0] == want, k
            except gpu.JgpmError as e:  # refused after the restore, in the launch itself
                assert e.code == ENOMEM
            finally:
                refuse(gpu, -1)
            assert s.wait(s.submit(ids[k & 1], "4-clique"), 20000)[0] == want, k
        assert s.stats()["restores"] >= 24
