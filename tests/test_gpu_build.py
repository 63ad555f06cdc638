"""The CSR builder on both sides of the size where it sorts edges once as
(min, max) keys instead of twice as directed ones, against the CPU oracle."""
import time

import numpy as np
import pytest

import hetegeneous_parallel_programming_gb300 as tc
from oracle import oracle

pytestmark = pytest.mark.gpu
HALF = 1 << 18


@pytest.fixture(scope="module")
def engine():
    with tc.Engine(0) as eng:
        yield eng


def random_edges(n, m, seed):
    rng = np.random.default_rng(seed)
    s = (n * rng.random(m) ** 3).astype(np.int32)  # skewed: duplicates, loops and hubs
    return n, s, rng.integers(0, n, m).astype(np.int32)


CASES = {
    "below": lambda: random_edges(5000, HALF - 1, 1),
    "at": lambda: random_edges(5000, HALF, 2),
    "ragged": lambda: random_edges(4097, HALF + 4096 * 3 + 17, 3),
    "two_vertices": lambda: random_edges(2, HALF, 4),
    "one_vertex": lambda: random_edges(1, HALF, 5),  # only loops
    "one_edge_repeated": lambda: (900, np.full(HALF, 17, np.int32), np.full(HALF, 899, np.int32)),
    "wide_ids": lambda: random_edges((1 << 25) + 3, HALF + 5, 6),
    "power_of_two_ids": lambda: random_edges(1 << 16, 1 << 20, 7),
    "past_one_tile_a_block": lambda: random_edges(70001, 4096 * 608 + 4097, 8),
    "complete": lambda: (700, *(np.tile(x, 2).astype(np.int32) for x in np.triu_indices(700, 1))),
}


@pytest.mark.parametrize("name", CASES)
def test_csr_from_edges(engine, name):
    n, s, d = CASES[name]()
    want_row, want_col = oracle.csr_from_edges(n, s, d)
    row, col = engine.csr_from_edges(n, s, d)
    assert np.array_equal(row, want_row) and np.array_equal(col, want_col)


def test_bad_ids_are_dropped(engine):
    n, s, d = random_edges(3000, HALF + 100, 9)
    good = oracle.csr_from_edges(n, s, d)
    s2 = np.concatenate([s, [-1, 5, n, 7]]).astype(np.int32)
    d2 = np.concatenate([d, [4, -7, 3, n + 9]]).astype(np.int32)
    row, col = engine.csr_from_edges(n, s2, d2)
    assert np.array_equal(row, good[0]) and np.array_equal(col, good[1])


MANY = 1 << 20  # half keys from here on, while the vertices are no more than the samples
LONG = {
    "one_below": lambda: random_edges(5000, MANY - 1, 10),
    "at": lambda: random_edges(5000, MANY, 11),
    "as_many_vertices": lambda: random_edges(MANY, MANY, 12),
    "one_vertex_more": lambda: random_edges(MANY + 1, MANY, 13),
    "one_vertex": lambda: random_edges(1, MANY, 14),
    "two_vertices": lambda: random_edges(2, MANY, 15),
    "one_edge_repeated": lambda: (900, np.full(MANY, 17, np.int32), np.full(MANY, 899, np.int32)),
    "ragged_wide_ids": lambda: random_edges((1 << 22) + 3, (1 << 22) + 4096 * 3 + 17, 16),
}


@pytest.mark.parametrize("name", LONG)
def test_csr_from_long_lists(engine, name):
    n, s, d = LONG[name]()
    want_row, want_col = oracle.csr_from_edges(n, s, d)
    row, col = engine.csr_from_edges(n, s, d)
    assert np.array_equal(row, want_row) and np.array_equal(col, want_col)


@pytest.mark.parametrize("m", [1 << 18, 1 << 20])
def test_one_sample_more_is_no_jump_with_many_vertices(engine, m):
    """2^26 vertices: the sample that reaches the size of another method must not multiply the time (it was 3 x)."""
    torch = pytest.importorskip("torch")
    n = 1 << 26
    s, d = (torch.randint(n, (m,), dtype=torch.int32, device="cuda") for _ in range(2))
    row = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    col = torch.empty(2 * m, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    best = {}
    for k in (m - 1, m):
        for _ in range(8):
            t = time.perf_counter()
            engine.csr_from_edges_device(n, k, s.data_ptr(), d.data_ptr(), row.data_ptr(), col.data_ptr(), col.numel())
            best[k] = min(best.get(k, 1e9), time.perf_counter() - t)
    assert best[m] < 1.8 * best[m - 1], best
