"""One pass over a caller-oriented DAG's entries: checks, sources, in-degrees
(csrc/orient.cu, dag_entries_kernel).  The general path is reached by a forced
arm or without validation; results are whole numbers."""
import numpy as np
import pytest

import hetegeneous_parallel_programming_gb300 as tc
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    with tc.Engine(0) as eng:
        yield eng


def layers(fan_in):
    """fan_in sources -> 64 targets in 8 slots of the in-degree table -> 40 sinks."""
    ids = np.arange(1000, 200000, dtype=np.uint32)
    mid = ids[((ids * np.uint32(2654435761)) >> np.uint32(16) & np.uint32(2047)) < 8][:64].astype(np.int32)
    assert len(mid) == 64
    n = 200100
    sinks = np.arange(n - 40, n, dtype=np.int32)
    deg = np.zeros(n, np.int64)
    deg[:fan_in] = 64
    deg[mid] = 40
    return np.concatenate([[0], np.cumsum(deg)]), np.concatenate([np.tile(mid, fan_in), np.tile(sinks, 64)])


@pytest.mark.parametrize("fan_in,pull", [(255, 0), (256, 4)])
def test_in_degrees_decide_the_arm(engine, fan_in, pull):
    rowptr, colidx = layers(fan_in)  # PULL from a mean in-degree of 256 on
    total, _, stats = engine.count_dag(rowptr, colidx, validate=False)
    assert total == 0 and stats["tiles_per_arm"]["pull"] == pull


@pytest.mark.parametrize("m", [1, 2047, 2048, 2049, 4097])
def test_sources_at_tile_ends(engine, m):
    s, d = np.triu_indices(100, 1)
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(s[:m], minlength=100))])
    colidx = d[:m].astype(np.int32)
    rows = [set(colidx[rowptr[u]:rowptr[u + 1]].tolist()) for u in range(100)]
    want = np.array([len(rows[u] & rows[v]) for u, v in zip(s[:m], d[:m])], np.uint32)
    for validate in (True, False):
        total, per_edge, _ = engine.count_dag(rowptr, colidx, force_arm="merge32", edge_counts=True,
                                              validate=validate)
        assert total == want.sum() and np.array_equal(per_edge, want)


@pytest.mark.parametrize("at", [1, 2047, 2048, 4949])
@pytest.mark.parametrize("fault", ["range", "negative", "loop", "order"])
def test_faults_are_refused(engine, at, fault):
    s, d = np.triu_indices(100, 1)
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(s, minlength=100))])
    colidx = d.astype(np.int32)
    if fault == "order":
        while s[at] != s[at - 1]:
            at -= 1
        colidx[at] = colidx[at - 1]
    else:
        colidx[at] = {"range": 100, "negative": -1, "loop": s[at]}[fault]
    with pytest.raises(tc.TCError):
        engine.count_dag(rowptr, colidx, force_arm="merge32")


def oriented(engine, spec):
    """Device CSR of the generator's graph, oriented by degree: rowptr, colidx on the host."""
    torch = pytest.importorskip("torch")
    k, n = spec.num_samples, spec.num_vertices
    s, d = (torch.empty(k, dtype=torch.int32, device="cuda") for _ in range(2))
    rowptr = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    colidx = torch.empty(2 * k, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    engine.gen_edges_device(spec, s.data_ptr(), d.data_ptr(), k)
    nnz = engine.csr_from_edges_device(n, k, s.data_ptr(), d.data_ptr(), rowptr.data_ptr(), colidx.data_ptr(), 2 * k)
    return engine.orient(rowptr.cpu().numpy(), colidx[:nnz].cpu().numpy())


def test_rows_between_the_entries_are_shared_out(engine):
    """The pass over the entries of a skewed sparse graph, whose empty rows lie together, against an even one of as
    many vertices and edges (it was 4 x as slow)."""
    ms = {}
    for kind, kw in (("rmat", dict(scale=25, edge_factor=1.0)), ("er", dict(n=1 << 25, avg_degree=2.0))):
        rowptr, colidx = oriented(engine, tc.GenSpec(kind, seed=5, **kw))
        ms[kind] = min(engine.count_dag(rowptr, colidx, validate=False)[-1]["ms_validate"] for _ in range(5))
    assert ms["rmat"] < 3 * ms["er"], ms
