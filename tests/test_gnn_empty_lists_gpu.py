"""Caller graphs whose list of a node ends before it begins: the node has no
neighbours, whatever entries lie between, and lists may then share entries.
Outputs and gradients are those of the graph with every list of its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def inputs(n, edges, seed=5):
    rng = np.random.default_rng(seed)
    f = lambda *s: rng.normal(size=s).astype(np.float32)
    return f(n, 14), f(edges, 4), f(n, 3), np.ones(n, np.float32), np.abs(f(edges))


def network(pdg):
    w = pdg.WarmStart(seed=1)
    p = w.get_params()
    p[-195:] = np.random.default_rng(2).uniform(-0.2, 0.2, 195)   # a decoder that is not zero
    w.set_params(p)
    w.set_smoothness(0.3)
    return w


# (ptr, adj, the entries of each list one after another, the plain ptr):
# a first node whose list starts at the end; a middle node between two that
# share their entries; two such nodes in a row
CASES = [([2, 0, 1, 2], [2, 1], [0, 1], [0, 0, 1, 2]),
         ([0, 2, 0, 2, 4, 6], [3, 4, 0, 2, 0, 2], [0, 1, 0, 1, 2, 3, 4, 5], [0, 2, 2, 4, 6, 8]),
         ([0, 2, 1, 0, 2, 4, 6], [4, 5, 0, 3, 0, 3], [0, 1, 0, 1, 2, 3, 4, 5], [0, 2, 2, 2, 4, 6, 8])]


@pytest.mark.parametrize("ptr,adj,order,plain", CASES)
@pytest.mark.parametrize("weighted", [False, True])
def test_lists_that_end_before_they_begin_are_empty(pdg, ptr, adj, order, plain, weighted):
    x, ef, target, free, ew = inputs(len(ptr) - 1, len(adj))
    w = network(pdg)
    got = w.eval(x, np.array(ptr, np.int32), np.array(adj, np.int32), ef, target, free, ew if weighted else None)
    want = w.eval(x, np.array(plain, np.int32), np.array(adj, np.int32)[order], ef[order], target, free,
                  ew[order] if weighted else None)
    assert np.array_equal(got[0], want[0]) and got[1] == want[1] and np.array_equal(got[2], want[2])


# an edge without a reverse beside such a list; a list that leaves the entries
@pytest.mark.parametrize("ptr,adj", [([2, 0, 1, 2], [2, 0]), ([0, 3, 0, 1, 2], [2, 1]), ([0, -1, 1, 2], [1, 1])])
def test_bad_graphs_with_such_lists_are_refused(pdg, ptr, adj):
    x, ef, target, free, _ = inputs(len(ptr) - 1, len(adj))
    w = network(pdg)
    with pytest.raises(pdg.PDGError) as e:
        w.eval(x, np.array(ptr, np.int32), np.array(adj, np.int32), ef, target, free)
    assert e.value.code == pdg.ERR_ARG
