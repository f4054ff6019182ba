"""The sweep's host staging against a plain loop: small batches take one, large ones
whole columns; both have to give the same arrays and refuse the same edges."""
import numpy as np
import pytest

from aleph_b200 import abi
from aleph_b200.backend import _stage_graphs


def plain(graphs):
    sets, pool = [], []
    for nq, edges in graphs:
        sets.append((nq, len(edges), len(pool) // 2))
        for (i, j) in edges:
            pool += [int(i), int(j)]
    return sets, np.asarray(pool, dtype=np.uint32)


def forms(edges):
    yield edges
    yield [list(e) for e in edges]
    yield np.array(edges, dtype=np.int32).reshape(-1, 2)
    yield [(float(i), np.uint8(j)) for i, j in edges]


@pytest.mark.parametrize("count", [0, 1, 4, 5, 40])
def test_staged_graphs_are_a_plain_loops(count):
    rng = np.random.default_rng(count)
    graphs = []
    for k in range(count):
        n = int(rng.integers(3, 20))
        edges = [(int(i), int(j)) for i, j in (rng.choice(n, 2, replace=False) for _ in range(int(rng.integers(0, 30))))]
        graphs.append((n if k % 2 else np.int64(n), list(forms(edges))[k % 4]))
    sets, edges = _stage_graphs(graphs)
    want, pool = plain(graphs)
    assert edges.dtype == np.uint32 and np.array_equal(edges, pool)
    assert [(sets[k].num_qubits, sets[k].num_edges, sets[k].edge_offset) for k in range(count)] == want
    assert isinstance(sets[0] if count else abi.QaoaSet(), abi.QaoaSet)


@pytest.mark.parametrize("count", [1, 6])
@pytest.mark.parametrize("edge,error", [((0, -1), OverflowError), ((0, 1 << 32), OverflowError), ((0, 1, 2), ValueError),
                                        ((0,), ValueError)])
def test_edges_that_are_no_pairs_of_qubits_are_refused(edge, error, count):
    with pytest.raises(error):
        _stage_graphs([(4, [(0, 1), edge])] * count)


@pytest.mark.parametrize("count", [1, 6])
def test_edges_may_be_any_iterables_of_two(count):
    sets, edges = _stage_graphs([(4, [iter((0, 1)), map(int, "23")]) for _ in range(count)])
    assert edges.tolist() == [0, 1, 2, 3] * count
