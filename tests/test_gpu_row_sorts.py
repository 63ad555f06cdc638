"""Per-edge counts come back in the input's order through the relabelled
rows' payload: rows of every sort class and at the edges of the classes, in
graphs on both sides of the id widths that the packed keys hold (2^22 and
2^24 vertices), against the CPU oracle."""
import numpy as np
import pytest

import hetegeneous_parallel_programming_gb300 as tc
from oracle import oracle

pytestmark = pytest.mark.gpu
LENGTHS = (list(range(1, 36)) + [63, 64, 65, 127, 128, 129, 191, 255, 256, 257, 300, 511, 512]) * 3


@pytest.fixture(scope="module")
def engine():
    with tc.Engine(0) as eng:
        yield eng


@pytest.mark.parametrize("n", [1 << 22, (1 << 22) + 1, 1 << 24, (1 << 24) + 1])
def test_payload_follows_the_rows(engine, n):
    rng = np.random.default_rng(n)
    pool, leaves = 600, 900  # targets of more neighbours than the longest row
    s, d = [], []
    for i, length in enumerate(LENGTHS):
        s.append(np.full(length, pool + i))
        d.append(rng.choice(pool, length, replace=False))
    first_leaf = pool + len(LENGTHS)
    s.append(first_leaf + np.arange(pool * leaves))
    d.append(np.repeat(np.arange(pool), leaves))
    i, j = np.triu_indices(pool, 1)
    keep = rng.random(len(i)) < 0.2
    s.append(i[keep])
    d.append(j[keep])
    ids = rng.choice(n, first_leaf + pool * leaves, replace=False)
    rowptr, colidx = oracle.csr_from_edges(n, ids[np.concatenate(s)].astype(np.int32),
                                           ids[np.concatenate(d)].astype(np.int32))
    total, per_edge, orow, _ = oracle.triangles(rowptr, colidx, per_edge=True)
    assert set(LENGTHS) <= set(np.diff(orow).tolist())
    got, pe, _ = engine.count(rowptr, colidx, edge_counts=True, validate=False)  # the general path
    assert got == total and np.array_equal(pe, per_edge)
    assert engine.count(rowptr, colidx, validate=False, force_arm="merge8")[0] == total


@pytest.mark.parametrize("n", [1 << 27, (1 << 27) + 1])
def test_short_rows_on_both_sides_of_the_packed_ids(engine, n):
    """Rows of at most 32 entries sort packed up to 2^27 vertices and one by one beyond: rows of 1 to 33 entries
    over a small dense part, on ids up to the last."""
    rng = np.random.default_rng(n)
    pool, leaves = 60, 200
    s, d = [], []
    lengths = list(range(1, 34)) * 40
    for i, length in enumerate(lengths):
        s.append(np.full(length, pool + i))
        d.append(rng.choice(pool, length, replace=False))
    first_leaf = pool + len(lengths)
    s.append(first_leaf + np.arange(pool * leaves))
    d.append(np.repeat(np.arange(pool), leaves))
    i, j = np.triu_indices(pool, 1)
    s.append(i)
    d.append(j)
    used = first_leaf + pool * leaves
    ids = np.unique(rng.integers(0, n - 1, 2 * used))[:used - 1]
    ids = rng.permutation(np.append(ids, n - 1))
    rowptr, colidx = engine.csr_from_edges(n, ids[np.concatenate(s)].astype(np.int32),
                                           ids[np.concatenate(d)].astype(np.int32))
    total, per_edge, orow, _ = oracle.triangles(rowptr, colidx, per_edge=True)
    assert set(range(1, 34)) <= set(np.diff(orow).tolist())
    got, pe, _ = engine.count(rowptr, colidx, edge_counts=True, force_arm="bsearch4")
    assert got == total and np.array_equal(pe, per_edge)
    assert engine.count(rowptr, colidx, force_arm="merge8")[0] == total
