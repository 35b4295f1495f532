"""Root arcs of two long rows (192 neighbours and more) that the nested-loop plans split over warps:
three hubs, adjacent to one another, share 220 neighbours, and a sparse random graph lies around
them.  Every split plan against the oracle, with a queue that holds the six hub arcs, with one that
holds two of them (the others run unsplit) and with none."""
import ctypes

import numpy as np
import pytest

import oracle_api as O

pytestmark = pytest.mark.gpu

PLANS = ["P3", "P4", "P5", "P6", "P7", "P8", "P9", "P10", "P11", "P12", "vsgm_last_pattern"]


@pytest.fixture(scope="module")
def hubs():
    rng = np.random.default_rng(3)
    n, shared = 600, 220
    hub = np.repeat([0, 1, 2], shared)
    leaf = np.tile(3 + np.arange(shared), 3)
    src = np.concatenate([[0, 0, 1], hub, rng.integers(3, n, 900)]).astype(np.int32)
    dst = np.concatenate([[1, 2, 2], leaf, rng.integers(3, n, 900)]).astype(np.int32)
    keep = src != dst
    p = rng.permutation(n).astype(np.int32)
    return O.build_csr(n, p[src[keep]], p[dst[keep]])


@pytest.mark.parametrize("plan", PLANS)
def test_split_plan(gpu, hubs, plan):
    want = O.count(plan, hubs)[0]
    queue = gpu.lib().jgpm_heavy_queue_
    with gpu.Graph.from_csr(hubs.rowptr, hubs.col, use_dag=False) as g:
        try:
            for cap in (1 << 20, 2, 0):
                queue(ctypes.c_int64(cap))
                assert g.count(plan, flags=gpu.COUNT_FORCE_PLAN) == want, cap
        finally:
            queue(ctypes.c_int64(1 << 20))


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("n,ef", [(400, 1), (3000, 2), (3000, 6)])
def test_sparse_graphs(gpu, plan, n, ef):
    """Most arcs have no or one common neighbour."""
    sym = O.rmat_graph(n, ef, 0.45, 0.1375, 0.1375, n + ef)
    with gpu.Graph.from_csr(sym.rowptr, sym.col, use_dag=False) as g:
        want, elems = O.count(plan, sym)[:2]
        assert g.count(plan, flags=gpu.COUNT_FORCE_PLAN) == want
        count, st = g.count(plan, stats=True, flags=gpu.COUNT_FORCE_PLAN)
        assert (count, st["setop_elements"]) == (want, elems)
