"""Tiles of short rows counted by single bits of the hub rows or by flattened
searches (wedge_kernel), on a graph whose rows mix hub and other targets on
both sides of the 65536-hub boundary, against the CPU oracle and PULL."""
import numpy as np
import pytest

import hetegeneous_parallel_programming_gb300 as tc
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    with tc.Engine(0) as eng:
        yield eng


def graph(n, fans, core, links, noise, seed):
    """`fans` vertices linked to `links` of a dense `core`; random edges among the others."""
    rng = np.random.default_rng(seed)
    ids = rng.permutation(n)
    i, j = np.triu_indices(core, 1)
    keep = rng.random(len(i)) < 0.3
    s = [ids[i[keep]], ids[core + np.repeat(np.arange(fans), links)], ids[core + rng.integers(0, n - core, noise)]]
    d = [ids[j[keep]], ids[rng.integers(0, core, fans * links)], ids[core + rng.integers(0, n - core, noise)]]
    return oracle.csr_from_edges(n, np.concatenate(s).astype(np.int32), np.concatenate(d).astype(np.int32))


@pytest.mark.parametrize("n,fans,core,links,noise", [
    (40000, 30000, 400, 6, 50000),       # every vertex is a hub; short suffixes
    (40000, 30000, 400, 24, 50000),      # suffixes that PULL would take
    (66000, 30000, 400, 24, 200000),     # 464 vertices below the hubs
    (300000, 60000, 700, 20, 1500000),   # most targets of the noise are no hubs
    (65536, 4097, 300, 33, 1),
])
def test_wedge_tests(engine, n, fans, core, links, noise):
    rowptr, colidx = graph(n, fans, core, links, noise, 7)
    total, per_edge, orow, ocol = oracle.triangles(rowptr, colidx, per_edge=True)
    # unvalidated calls take the general path whatever the size
    got, pe, st = engine.count(rowptr, colidx, edge_counts=True, validate=False)
    assert got == total and np.array_equal(pe, per_edge)
    assert st["tiles_per_arm"]["bsearch4"] > 0
    assert engine.count(rowptr, colidx, validate=False)[0] == total
    assert engine.count(rowptr, colidx, validate=False, force_arm="pull")[0] == total
    got, pv, _ = engine.count_vertices(rowptr, colidx, validate=False)
    want = engine.count_vertices(rowptr, colidx)[1]  # direct counting, where the graph is small enough
    assert got == total and int(pv.sum()) == 3 * total and np.array_equal(pv, want)
    labels = (np.arange(n) * 5 % 4).astype(np.uint8)
    sums = []
    for lab in range(4):
        a, ape, _ = engine.count_labelled(rowptr, colidx, labels, lab, edge_counts=True, validate=False)
        sums.append(ape.astype(np.int64))
        assert a == int(ape.sum())
    assert np.array_equal(sum(sums), per_edge)
    assert engine.load_shipped_selector()
    assert engine.count(rowptr, colidx, validate=False, selector="learned")[0] == total


@pytest.mark.parametrize("n,k,cliques,pull", [
    (100000, 100, 1000, "most"),   # even lists, m / n = 49: PULL shares its tables over most tiles
    (30000, 100, 300, "most"),     # the same, too few tiles for hub bit rows
    (156000, 60, 2600, "none"),    # m / n = 29
    (1000000, 100, 100, "none"),   # a few tiles of them among many vertices
    (300000, 400, 60, "some"),     # m / n = 16, rows of up to 399 entries
])
def test_long_even_lists_of_attributed_counts(engine, n, k, cliques, pull):
    """Disjoint cliques of k vertices on interleaved ids; per-vertex and labelled counts choose between wedge tests
    and PULL for the tiles that the fixed rule leaves to other arms."""
    i, j = np.triu_indices(k, 1)
    first = np.arange(cliques)[:, None]
    s, d = (first + cliques * i).ravel(), (first + cliques * j).ravel()
    rowptr, colidx = engine.csr_from_edges(n, s.astype(np.int32), d.astype(np.int32))
    total, per_vertex, st = engine.count_vertices(rowptr, colidx, validate=False)
    assert total == cliques * k * (k - 1) * (k - 2) // 6
    used = np.arange(n) < cliques * k
    assert np.array_equal(per_vertex, np.where(used, (k - 1) * (k - 2) // 2, 0).astype(np.uint64))
    labels = (np.arange(n) % 2).astype(np.uint8)
    parts = [engine.count_labelled(rowptr, colidx, labels, lab, validate=False) for lab in (0, 1)]
    assert parts[0][0] + parts[1][0] == total
    for tiles, arms in [(x["tiles"], x["tiles_per_arm"]) for x in (st, parts[0][2])]:
        share = arms["pull"] / tiles
        assert {"most": share > 0.5, "none": share == 0, "some": 0 < share < 1}[pull], (share, arms)
