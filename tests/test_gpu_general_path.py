"""The general path where small graphs would be counted directly: its own
checks of the input (kept_count_kernel, validate_rowptr_kernel) and the
captured pipeline of unvalidated batches."""
import numpy as np
import pytest

import hetegeneous_parallel_programming_gb300 as tc
from oracle import oracle

pytestmark = pytest.mark.gpu
MANY = (1 << 22) + 5  # vertices: more than the direct path takes


@pytest.fixture(scope="module")
def engine():
    with tc.Engine(0) as eng:
        yield eng


@pytest.mark.parametrize("rowptr,colidx", [
    ([0, 2, 1, 3], [1, 2, 0]),          # rowptr not monotone
    ([0, 1, 2, 2], [1, 3]),             # id out of range
    ([0, 1, 2, 2], [1, -1]),
    ([0, 2, 3, 3], [2, 1, 0]),          # row not ascending
    ([0, 1, 2, 2], [0, 0]),             # self loop
    ([0, 2, 2, 2], [1, 1]),             # duplicate neighbour
    ([0, 1, 2, 5], [1, 0]),             # rowptr[n] != nnz
    ([1, 1, 2, 2], [1, 0]),             # rowptr[0] != 0
])
def test_small_faults(engine, rowptr, colidx):
    n = len(rowptr) - 1
    wide = np.concatenate([rowptr, np.full(MANY - n, rowptr[-1])])
    cols = np.where(np.array(colidx) == n, MANY, colidx)
    calls = [lambda: engine.count(np.array(rowptr), np.array(colidx), force_arm="merge32"),
             lambda: engine.count(wide, cols), lambda: engine.count_vertices(wide, cols),
             lambda: engine.count_labelled(wide, cols, np.zeros(MANY, np.uint8), 0), lambda: engine.orient(wide, cols)]
    for call in calls:
        with pytest.raises(tc.TCError) as ei:
            call()
        assert ei.value.status == 2
    tri = (np.array([0, 2, 4, 6]), np.array([1, 2, 0, 2, 0, 1]))  # the ctx stays usable
    assert engine.count(*tri, force_arm="merge32")[0] == 1


@pytest.mark.parametrize("fault", ["range", "negative", "loop", "duplicate", "unsorted"])
@pytest.mark.parametrize("at", [1, 255, 2047, 2048, 2049, 4096, -1])
def test_faults_at_tile_ends(engine, at, fault):
    """One fault in a complete graph of 80 vertices, on both sides of the 2048-entry tiles."""
    k = 80
    s, d = np.triu_indices(k, 1)
    rowptr, colidx = oracle.csr_from_edges(k, s.astype(np.int32), d.astype(np.int32))
    row = np.repeat(np.arange(k), k - 1)
    at %= len(colidx)
    if fault in ("duplicate", "unsorted"):
        while row[at] != row[at - 1]:
            at += 1
    bad = colidx.copy()
    bad[at] = {"range": k, "negative": -1, "loop": row[at], "duplicate": colidx[at - 1], "unsorted": colidx[at - 1] - 1}[fault]
    for arm in ("merge32", "pull"):
        with pytest.raises(tc.TCError) as ei:
            engine.count(rowptr, bad, force_arm=arm)
        assert ei.value.status == 2
    assert engine.count(rowptr, colidx, force_arm="merge32")[0] == k * (k - 1) * (k - 2) // 6


def test_unvalidated_batches_follow_the_tuning(engine):
    """The captured graphs of the batched pipeline are keyed by every setting they bake in."""
    n, s, d = tc.gen_edges_host(tc.GenSpec("rmat", scale=16, edge_factor=16, seed=6))
    rowptr, colidx = oracle.csr_from_edges(n, s, d)
    ref = oracle.triangles(rowptr, colidx)
    batch = (np.array([0, n, 2 * n]), np.concatenate([rowptr, rowptr[1:] + rowptr[-1]]), np.tile(colidx, 2))
    old = engine.get_tuning()
    try:
        for change in ({"pull_item": 32, "pull_item_min": 32}, {"pull_item": 4096, "pull_item_min": 64}, {},
                       {"pull_block_tiles": 64}, {"pull_dense_num": 4}, {"pull_dense_den": 4},
                       {"orient_blocks_per_sm": 1}, {"orient_blocks_per_sm": 12}):
            engine.set_tuning(**{**old, **change})
            for _ in range(2):  # captured, then replayed
                totals, st = engine.batch_count(*batch, validate=False)
                assert totals.tolist() == [ref, ref], change
                assert st["tiles_per_arm"]["flat"] == 0
        engine.autotune_pull(rowptr, colidx, candidates=(128, 2048), reps=1)
        assert engine.batch_count(*batch, validate=False)[0].tolist() == [ref, ref]
    finally:
        engine.set_tuning(**old)
