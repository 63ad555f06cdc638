"""Kept entries compacted per chunk, then placed (csrc/orient.cu,
kept_count_kernel and place_kernel): chunks that keep all, none or a few of
their entries, and sizes around a tile of 2048.  Whole numbers, so equality."""
import numpy as np
import pytest

import hetegeneous_parallel_programming_gb300 as tc
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    with tc.Engine(0) as eng:
        yield eng


def graph(n, s, d):
    return oracle.csr_from_edges(n, np.asarray(s, np.int32), np.asarray(d, np.int32))


def hubs(first, leaves):
    """3 mutually joined hubs from id `first` on, joined to every leaf: the leaves keep all, the hubs next to none."""
    n = leaves + 3
    hub = np.arange(first, first + 3)
    leaf = np.setdiff1d(np.arange(n), hub)
    s = np.concatenate([np.repeat(hub, leaves), hub])
    return graph(n, s, np.concatenate([np.tile(leaf, 3), np.roll(hub, 1)]))


GRAPHS = {
    "one_edge": lambda: graph(5, [1], [3]),
    "nnz_2046": lambda: graph(1200, np.arange(1023), np.arange(1, 1024)),
    "nnz_2048": lambda: graph(1200, np.arange(1024), np.arange(1, 1025)),
    "nnz_2050": lambda: graph(1200, np.arange(1025), np.arange(1, 1026)),
    "hubs_first": lambda: hubs(0, 30011),
    "hubs_last": lambda: hubs(30011, 30011),
    "rmat_17": lambda: graph(*tc.gen_edges_host(tc.GenSpec("rmat", scale=17, seed=3))),
}


@pytest.mark.parametrize("name", GRAPHS)
def test_placement(engine, name):
    rowptr, colidx = GRAPHS[name]()
    total, per_edge, orow, ocol = oracle.triangles(rowptr, colidx, per_edge=True)
    got, counts, _ = engine.count(rowptr, colidx, force_arm="bsearch4", edge_counts=True)
    assert got == total and np.array_equal(counts, per_edge)
    got, _, _ = engine.count(rowptr, colidx, force_arm="merge32", validate=False)
    assert got == total
    drow, dcol = engine.orient(rowptr, colidx)[:2]
    assert np.array_equal(drow, orow) and np.array_equal(dcol, ocol)


def test_batch_after_a_change_of_chunks(engine):
    """The batch's captured second half holds the chunk geometry: a new one is captured when it changes."""
    batch = tc.gen_batch_host(num_graphs=160, n_min=64, n_max=16384, seed=4)
    want, _ = engine.batch_count(*batch)
    was = engine.get_tuning()["orient_blocks_per_sm"]
    for blocks in (was, 1, 9, was):
        engine.set_tuning(orient_blocks_per_sm=blocks)
        got, _ = engine.batch_count(*batch, validate=False)
        assert np.array_equal(got, want)
