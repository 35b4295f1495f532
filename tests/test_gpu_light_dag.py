"""Graphs that are counted on the id DAG, by scans (out-degrees up to 32; on graphs of 4 M arcs and
more up to 64, with few vertices above 32), and the borders of that rule: planted complete graphs
bring roots of out-degree 32, 33, 63, 64 and 65 into sparse graphs; weakly skewed R-MAT graphs have
short rows outside the bitmap.  Counts are integers: equality with the oracle, single calls,
batches and shards."""
import numpy as np
import pytest

import oracle_api as O

pytestmark = pytest.mark.gpu

PLAIN = {"triangle": "P0", "4-clique": "P13", "5-clique": "P14", "6-clique": "P15"}


def sparse_with_cliques(n, sizes, seed):
    """A random graph of n vertices and 6 n edges with a complete graph planted for each size."""
    rng = np.random.default_rng(seed)
    src, dst = [rng.integers(0, n, 6 * n)], [rng.integers(0, n, 6 * n)]
    free = rng.permutation(n)
    for s in sizes:
        at, free = free[:s], free[s:]
        i, j = np.triu_indices(s, 1)
        src.append(at[i])
        dst.append(at[j])
    src, dst = np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)
    keep = src != dst
    return O.build_csr(n, src[keep], dst[keep])


def wanted(sym):
    dag = O.orient(sym)
    want = {k: O.count(p, dag)[0] for k, p in PLAIN.items()}
    want["diamond"] = O.count("P2", sym)[0]
    return want, O.count("induced-tailed-triangle", sym)[0], dag


def check(gpu, sym, p5=True):
    want, tt, dag = wanted(sym)
    with gpu.Graph.from_csr(sym.rowptr, sym.col, use_dag=False) as g:
        for k, w in want.items():
            assert g.count(k) == w, k
        for k, p in PLAIN.items():  # the accounting pass recounts as well
            count, st = g.count(k, stats=True)
            assert (count, st["setop_elements"]) == O.count(p, dag)[:2], k
            assert sum(g.count_shard(k, s, 3) for s in range(3)) == count, k
        assert g.count("tailed-triangle", induced=True) == tt
        assert g.census4()[2] == tt
        jobs = [(g, k) for k in want] + [(g, "induced:tailed-triangle"), (g, "k-clique:7")]
        got = gpu.batch_count(jobs)[0]
        assert got[:-1] == list(want.values()) + [tt]
        assert got[-1] == g.count("k-clique:7")
        if p5:  # may move the graph to the rank DAG; the counts stay
            p5 = O.count("P5", sym)[0]
            assert [g.count("P5") for _ in range(3)] == [p5] * 3
        assert g.count("triangle") == want["triangle"]


@pytest.mark.parametrize("sizes", [(), (33,), (34,), (33, 34, 40), (64,), (65,), (66,), (20,) * 40])
def test_planted_cliques(gpu, sizes):
    check(gpu, sparse_with_cliques(30000, sizes, len(sizes)))


# 5 M arcs: roots above 32 are scanned by a CTA each up to out-degree 64, and the graph with one of
# 65 has a rank DAG
@pytest.mark.parametrize("sizes", [(34, 50, 65), (66,)])
def test_planted_cliques_in_a_large_graph(gpu, sizes):
    check(gpu, sparse_with_cliques(850000, sizes, 7), p5=False)


@pytest.mark.parametrize("n,ef,a,b", [(300, 3, .45, .1375), (2500, 16, .45, .1375),
                                      (2500, 32, .45, .1375), (50000, 4, .45, .1375),
                                      (20000, 10, .45, .2391), (9000, 16, .5, .125)])
def test_weakly_skewed(gpu, n, ef, a, b):
    check(gpu, O.rmat_graph(n, ef, a, b, b, n))


def test_p5_after_many_calls(gpu):
    """The nested loops of the first calls and the per-arc counters of the later ones agree."""
    sym = O.rmat_graph(2000, 4, .5, .2, .2, 5)
    want = O.count("P5", sym)[0]
    with gpu.Graph.from_csr(sym.rowptr, sym.col, use_dag=False) as g:
        methods = set()
        for _ in range(400):
            count, st = g.count("P5", details=True)
            assert count == want
            methods.add(st["method"])
        assert len(methods) == 2
