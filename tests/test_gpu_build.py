"""The CSR builder on both sides of the size where it sorts edges once as
(min, max) keys instead of twice as directed ones, against the CPU oracle."""
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
