"""Direct counting of small graphs (csrc/direct.cu): validated calls with the
fixed selector below its size limits.  Counts are whole numbers, so every
comparison is for equality."""
import time

import numpy as np
import pytest

import hetegeneous_parallel_programming_gb300 as tc
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    with tc.Engine(0) as eng:
        yield eng


def csr_of(n, s, d):
    return oracle.csr_from_edges(n, np.asarray(s, np.int32), np.asarray(d, np.int32))


def rmat(scale, degree, seed=1):
    return csr_of(*tc.gen_edges_host(tc.GenSpec("rmat", scale=scale, edge_factor=degree / 2, seed=seed)))


def path_with_rows(entries, n):
    """`entries` (even) adjacency entries: a path, so the last 32-entry group and 1024-entry block are ragged."""
    k = entries // 2
    return csr_of(n, np.arange(k), np.arange(1, k + 1))


def clique(k, n, first):
    i, j = np.triu_indices(k, 1)
    return csr_of(n, i + first, j + first)


CASES = {
    "no_edges": lambda: csr_of(40, [], []),
    "one_edge_last_ids": lambda: csr_of(70000, [69998], [69999]),
    "path_1022": lambda: path_with_rows(1022, 600),
    "path_1024": lambda: path_with_rows(1024, 600),
    "path_1026_many_empty_rows": lambda: path_with_rows(1026, 200000),
    "star_and_rim": lambda: csr_of(5000, [0] * 4999 + list(range(1, 4999)), list(range(1, 5000)) + list(range(2, 5000))),
    "clique_ends_16384": lambda: clique(130, 16384, 16384 - 130),
    "clique_ends_16385": lambda: clique(130, 16385, 16385 - 130),
    "clique_ends_65536": lambda: clique(70, 65536, 65536 - 70),
    "clique_across_65536": lambda: clique(300, 65700, 65700 - 300),
    "rmat_13_degree_60": lambda: rmat(13, 60),
    "rmat_17_degree_6": lambda: rmat(17, 6),
    "chung_lu_130k": lambda: csr_of(*tc.gen_edges_host(tc.GenSpec("chung_lu", n=130001, avg_degree=9, seed=2))),
    "declined_clique_1300": lambda: clique(1300, 1300, 0),  # lists longer than the limit: the general path counts
}


@pytest.mark.parametrize("name", CASES)
def test_direct_counts(engine, name):
    rowptr, colidx = CASES[name]()
    n = len(rowptr) - 1
    total, per_edge, orow, ocol = oracle.triangles(rowptr, colidx, per_edge=True)
    got, pe, st = engine.count(rowptr, colidx, edge_counts=True)
    assert got == total and np.array_equal(pe, per_edge) and st["m"] == len(ocol)
    assert engine.count(rowptr, colidx)[0] == total
    gen, gpe, _ = engine.count(rowptr, colidx, edge_counts=True, validate=False)  # the general path
    assert gen == total and np.array_equal(gpe, pe)
    src = np.repeat(np.arange(n), np.diff(orow))
    got, pv, _ = engine.count_vertices(rowptr, colidx)
    gen, gpv, _ = engine.count_vertices(rowptr, colidx, validate=False)
    assert got == gen == total and np.array_equal(pv, gpv) and int(pv.sum()) == 3 * total
    labels = (np.arange(n) * 7 % 3).astype(np.uint8)
    for lab in (0, 2):
        a, ape, _ = engine.count_labelled(rowptr, colidx, labels, lab, edge_counts=True)
        b, bpe, _ = engine.count_labelled(rowptr, colidx, labels, lab, edge_counts=True, validate=False)
        assert a == b and np.array_equal(ape, bpe)
    got, pe, _ = engine.count_dag(orow, ocol, edge_counts=True)
    assert got == total and np.array_equal(pe, per_edge)
    for lo, hi in ((0, n), (n // 3, n - n // 4), (n // 2, n // 2)):
        got, pe, st = engine.count_dag_range(orow, ocol, lo, hi, edge_counts=True)
        assert st["m"] == orow[hi] - orow[lo]
        assert np.array_equal(pe, per_edge[orow[lo]:orow[hi]]) and got == int(per_edge[orow[lo]:orow[hi]].sum())
    assert len(src) == len(ocol)


def test_direct_refuses_what_the_general_path_refuses(engine):
    rowptr, colidx = rmat(9, 12)
    row = int(np.argmax(np.diff(rowptr)))
    a = int(rowptr[row])
    bad_id, loop, unsorted, dup = (colidx.copy() for _ in range(4))
    bad_id[-1] = len(rowptr) - 1
    loop[a] = row
    unsorted[a], unsorted[a + 1] = colidx[a + 1], colidx[a]
    dup[a + 1] = dup[a]
    bad_row = rowptr.copy()
    bad_row[5] = bad_row[6] + 3
    for r, c in ((rowptr, bad_id), (rowptr, loop), (rowptr, unsorted), (rowptr, dup), (bad_row, colidx)):
        for call in (engine.count, engine.count_vertices, engine.count_dag):
            with pytest.raises(tc.TCError) as e:
                call(r, c)
            assert e.value.status == 2
    assert engine.count(rowptr, colidx)[0] == oracle.triangles(rowptr, colidx)


@pytest.mark.parametrize("sizes", [
    [1], [3, 1, 2], [40] * 70, [16384, 5, 16384], [16385, 900], [32769, 64, 2], [65536, 65537, 300], [70000, 1, 1, 9]])
def test_direct_batches(engine, sizes):
    """Batches of graphs around the bitmap widths (16384, 32768, 65536 ids), with empty and one-vertex
    graphs, edges of several graphs in one group of 32, and cliques on the last ids of each graph."""
    rowptr, colidx, off, want = [np.zeros(1, np.int64)], [], [0], []
    for i, n in enumerate(sizes):
        k = min(n, 11 + 17 * (i % 3))
        s, d = np.triu_indices(k, 1)
        s, d = list(s + n - k), list(d + n - k)
        s += list(range(0, n - 1, 1 + i % 4))
        d += [x + 1 for x in range(0, n - 1, 1 + i % 4)]
        r, c = csr_of(n, s, d)
        want.append(oracle.triangles(r, c))
        rowptr.append(r[1:] + rowptr[-1][-1])
        colidx.append(c)
        off.append(off[-1] + n)
    rowptr, colidx = np.concatenate(rowptr), np.concatenate(colidx)
    got, st = engine.batch_count(np.array(off), rowptr, colidx)
    assert got.tolist() == want and st["m"] == len(colidx) // 2
    assert engine.batch_count(np.array(off), rowptr, colidx, validate=False)[0].tolist() == want
    if len(colidx) > 2:
        bad = colidx.copy()
        bad[-1] = sizes[-1]  # outside its graph
        with pytest.raises(tc.TCError) as e:
            engine.batch_count(np.array(off), rowptr, bad)
        assert e.value.status == 2


def test_direct_batch_declines_long_lists(engine):
    """Complete graphs have lists longer than the limit per entry: the general path counts them."""
    k, graphs = 700, 3
    r, c = clique(k, k, 0)
    rowptr = np.concatenate([[0]] + [r[1:] + g * r[-1] for g in range(graphs)])
    got, _ = engine.batch_count(np.arange(graphs + 1) * k, rowptr, np.tile(c, graphs))
    assert got.tolist() == [k * (k - 1) * (k - 2) // 6] * graphs


@pytest.mark.parametrize("graphs,n_min,n_max,deg", [(1, 65537, 65537, 30.5), (1, 65537, 65537, 32.1),
                                                    (9, 9000, 16384, 29.0), (400, 700, 900, 7.0),
                                                    (3000, 64, 400, 3.0), (3000, 64, 400, 5.0)])
def test_direct_batches_around_two_million_entries(engine, graphs, n_min, n_max, deg):
    """The rows pass of a batch takes 8 groups a warp from 2^21 entries on, 4 below."""
    vtx, rowptr, colidx = tc.gen_batch_host(num_graphs=graphs, n_min=n_min, n_max=n_max, deg_min=deg, deg_max=deg + 1,
                                            seed=11)
    totals, stats = engine.batch_count(vtx, rowptr, colidx)
    for g in range(0, graphs, max(1, graphs // 40)):
        a, b = int(vtx[g]), int(vtx[g + 1])
        lo, hi = int(rowptr[a]), int(rowptr[b])
        assert totals[g] == oracle.triangles(rowptr[a:b + 1] - lo, colidx[lo:hi])
    assert np.array_equal(totals, engine.batch_count(vtx, rowptr, colidx, validate=False)[0])
    assert stats["m"] * 2 == len(colidx)


@pytest.mark.parametrize("n,degree,count,direct", [(65536, 24.0, 4, True), (65537, 6.0, 2, True), (65537, 6.0, 60, True),
                                                   (100000, 24.0, 3, True), (100000, 24.0, 4, False),
                                                   (100000, 24.0, 16, False), (70000, 60.0, 6, False)])
def test_batches_of_large_graphs_take_the_quicker_path(engine, n, degree, count, direct):
    """Beyond 65536 vertices hits are confirmed by searches: a list entry costs several times as much there, so
    such batches go direct only with short lists (8 per entry), or few (3 * 2^25)."""
    r, c = csr_of(*tc.gen_edges_host(tc.GenSpec("er", n=n, avg_degree=degree, seed=8)))
    rowptr = np.concatenate([[0]] + [r[1:] + g * r[-1] for g in range(count)])
    totals, stats = engine.batch_count(np.arange(count + 1) * n, rowptr, np.tile(c, count))
    assert (stats["tiles_per_arm"]["flat"] == stats["tiles"]) == direct
    assert totals.tolist() == [engine.count(r, c, validate=False)[0]] * count


def in_many(k, n, edges=0):
    """A clique among n vertices, and a path over the first `edges` of them."""
    i, j = np.triu_indices(k, 1)
    a = np.arange(edges)
    return csr_of(n, np.concatenate([i * (n // k), a]), np.concatenate([j * (n // k), a + 1]))


def test_limits_of_the_direct_path(engine):
    """A call goes direct while its lists sum to no more than the limit of its kind, above and below 65536 vertices
    (exact and hashed bitmaps): a clique of k vertices sums to k (k - 1)^2 / 2."""
    n = {"exact": 65536, "hashed": 65537}
    limits = {("count", "exact"): 1 << 30, ("count", "hashed"): 7 << 24, ("dag", "hashed"): 5 << 25,
              ("labelled", "exact"): 21 << 24, ("labelled", "hashed"): 3 << 25,
              ("vertices", "exact"): 15 << 23, ("vertices", "hashed"): 5 << 24}
    for (kind, size), limit in limits.items():
        k = 1
        while (k + 1) * k * k // 2 <= limit:
            k += 1
        for clique_size, direct in ((k, True), (k + 1, False)):
            r, c = in_many(clique_size, n[size])
            want = clique_size * (clique_size - 1) * (clique_size - 2) // 6
            if kind == "count":
                total, _, st = engine.count(r, c)
            elif kind == "dag":
                total, _, st = engine.count_dag(*oracle.orient(r, c))
            elif kind == "labelled":
                total, _, st = engine.count_labelled(r, c, np.zeros(n[size], np.uint8), 0)
            else:
                total, _, st = engine.count_vertices(r, c)
            assert total == want
            if direct is False or clique_size * (clique_size - 1) < 1 << 20:  # from 2^20 entries a sample decides first
                assert (st["tiles_per_arm"]["flat"] == st["tiles"]) == direct, (kind, size, clique_size)


@pytest.mark.parametrize("k,direct", [(1020, True), (1030, False)])
def test_oriented_graphs_of_long_lists_take_the_general_path(engine, k, direct):
    """Below 65536 vertices an oriented graph also goes direct only with lists of 1024 on average at most."""
    total, _, st = engine.count_dag(*oracle.orient(*in_many(k, 65536)))
    assert total == k * (k - 1) * (k - 2) // 6
    assert (st["tiles_per_arm"]["flat"] == st["tiles"]) == direct


@pytest.mark.parametrize("small", [False, True])  # 2^20 entries and more are sampled first
def test_a_row_range_is_judged_by_its_own_lists(engine, small):
    """A range goes direct by the lists of its own rows, however long those of the rest of the graph are."""
    k, n = 1030 if small else 1500, 65536  # a clique that a whole count leaves to the general path
    rowptr, colidx = oracle.orient(*in_many(k, n))
    total = k * (k - 1) * (k - 2) // 6
    got, _, st = engine.count_dag(rowptr, colidx)
    assert got == total and st["tiles_per_arm"]["flat"] == 0
    at = (n // k) * (k // 2)  # one row of the clique: k - 1 - k // 2 targets, their lists meet in every pair
    d = k - 1 - k // 2
    for lo, hi, want in ((at, at + 1, d * (d - 1) // 2), (at + 1, at + 2, 0)):
        got, pe, st = engine.count_dag_range(rowptr, colidx, lo, hi, edge_counts=True)
        assert got == int(pe.sum()) == want and st["m"] == (d if want else 0)
        assert st["tiles_per_arm"]["flat"] == st["tiles"], (lo, hi)
    assert sum(engine.count_dag_range(rowptr, colidx, a, a + n // 8)[0] for a in range(0, n, n // 8)) == total


def test_times_of_a_direct_call_cover_its_copies(engine):
    """The parts of a call with host input and output: none overlaps another, the whole holds them all."""
    rowptr, colidx = rmat(16, 16)
    labels = np.zeros(len(rowptr) - 1, np.uint8)
    for call in (lambda: engine.count_vertices(rowptr, colidx), lambda: engine.count(rowptr, colidx, edge_counts=True),
                 lambda: engine.count_labelled(rowptr, colidx, labels, 0, edge_counts=True)):
        call()
        st = call()[-1]
        assert st["tiles_per_arm"]["flat"] == st["tiles"]
        assert st["ms_h2d"] > 0 and st["ms_orient"] > 0 and st["ms_count"] > 0 and st["ms_d2h"] > 0
        parts = st["ms_h2d"] + st["ms_orient"] + st["ms_count"] + st["ms_d2h"]
        assert parts <= 1.001 * st["ms_total"] + 0.002  # events and the device's clock resolve about a microsecond
    assert engine.count(rowptr, colidx)[-1]["ms_d2h"] == 0


def quickest(call, reps=5):
    call()
    times = []
    for _ in range(reps):
        t = time.perf_counter()
        st = call()[-1]
        times.append((time.perf_counter() - t) * 1e3)
    return min(times), st


def test_declined_host_calls_upload_once(engine):
    """What a declined call has uploaded stays for the general path: unvalidated calls take that path at once and
    upload once too, so the difference of the times is less than half an upload (tens of MB)."""
    n, s, d = tc.gen_edges_host(tc.GenSpec("rmat", scale=22, edge_factor=0.95, seed=3))
    rowptr, colidx = engine.csr_from_edges(n, s, d)
    assert (1 << 22) < len(colidx) <= (1 << 23)
    labels = (np.arange(n) % 3).astype(np.uint8)
    drow, dcol = engine.orient(rowptr, colidx)
    k, graphs = 700, 30
    r, c = clique(k, k, 0)
    batch = (np.arange(graphs + 1) * k, np.concatenate([[0]] + [r[1:] + g * r[-1] for g in range(graphs)]), np.tile(c, graphs))
    for call in (lambda v: engine.count(rowptr, colidx, validate=v), lambda v: engine.count_vertices(rowptr, colidx, validate=v),
                 lambda v: engine.count_labelled(rowptr, colidx, labels, 1, validate=v),
                 lambda v: engine.batch_count(*batch, validate=v)):
        declined, st = quickest(lambda: call(True))
        general, gen = quickest(lambda: call(False))
        assert st["tiles_per_arm"]["flat"] == 0 and st["h2d_bytes"] == gen["h2d_bytes"] > 1 << 25
        assert np.array_equal(call(True)[0], call(False)[0])
        assert st["ms_h2d"] > 0 and declined < general + 0.5 * st["ms_h2d"], (declined, general, st["ms_h2d"])
        assert st["ms_total"] >= st["ms_h2d"] + st["ms_orient"] + st["ms_count"]
    with tc.Engine(0) as fresh:  # the arena grows between the two paths
        assert fresh.count_labelled(rowptr, colidx, labels, 1)[0] == engine.count_labelled(rowptr, colidx, labels, 1)[0]
    with tc.Engine(0) as fresh:
        assert fresh.batch_count(*batch)[0].tolist() == [k * (k - 1) * (k - 2) // 6] * graphs
    with tc.Engine(0) as fresh:
        assert fresh.count_dag(drow, dcol)[0] == engine.count(rowptr, colidx)[0]


def test_autotuners_time_the_path_they_tune(engine):
    """The settings belong to the general path, so that is what a trial runs, also on a graph that counts directly."""
    rowptr, colidx = rmat(16, 16)
    old = engine.get_tuning()

    def device_ms(validate):
        return min(engine.count(rowptr, colidx, validate=validate)[-1]["ms_total"] for _ in range(6))
    direct, general = device_ms(True), device_ms(False)
    assert direct < general
    try:
        _, ms = engine.autotune_pull(rowptr, colidx, candidates=(256, 512), reps=3)
        assert min(ms.values()) > (direct + general) / 2, (ms, direct, general)
        _, best, trials = engine.autotune(rowptr, colidx, reps=3)
        assert trials > 4 and best > (direct + general) / 2, (best, direct, general)
    finally:
        engine.set_tuning(**old)


@pytest.mark.parametrize("n", [1 << 21, (1 << 21) + 1])  # from one copy of the counts per 2^22 / n warps to a single one
def test_refused_calls_leave_the_outputs_alone(engine, n):
    torch = pytest.importorskip("torch")
    rowptr = np.full(n + 1, 6, np.int64)
    rowptr[:4] = [0, 2, 4, 6]
    good, bad = np.array([1, 2, 0, 2, 0, 1]), np.array([1, 2, 0, 2, 0, n])
    out = torch.full((n,), 77, dtype=torch.int64, device="cuda")
    edges = torch.full((6,), 77, dtype=torch.int32, device="cuda")
    rp = torch.from_numpy(rowptr).cuda()
    for cols in (bad, good):
        cl = torch.from_numpy(cols.astype(np.int32)).cuda()
        torch.cuda.synchronize()
        args = (n, 6, rp.data_ptr(), cl.data_ptr())
        if cols is good:
            assert engine.count_vertices_device(*args, out.data_ptr())[0] == 1
            assert out[:4].tolist() == [1, 1, 1, 0] and int(out.sum()) == 3
            continue
        for call in (lambda: engine.count_vertices_device(*args, out.data_ptr()),
                     lambda: engine.count_device(*args, edge_counts_ptr=edges.data_ptr(), edge_capacity=6)):
            with pytest.raises(tc.TCError) as e:
                call()
            assert e.value.status == 2
        assert bool((out == 77).all()) and bool((edges == 77).all())
