"""Gradients of the warm-start network where the weight-gradient kernel's tiling
changes (around 16- and 32-row tiles, one tile per block and several), graphs
of changing size on one network, and adjacencies that are refused.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def path_problem(n, seed):
    """A path of n vertices (a vertex without edges for n = 1)."""
    import gnn_oracle as G
    rng = np.random.default_rng(seed)
    pairs = [(i, j) for i in range(n) for j in (i - 1, i + 1) if 0 <= j < n]
    dst = np.array([p[0] for p in pairs], np.int64)
    src = np.array([p[1] for p in pairs], np.int64)
    deg = np.bincount(dst, minlength=n) if n > 1 else np.zeros(1, np.int64)
    ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    f = lambda *s: rng.normal(size=s).astype(np.float32)
    p = {k: rng.normal(scale=0.25, size=s) for k, s in G.shapes()}
    return G, p, f(n, G.NF), f(len(src), G.EF), src, dst, deg, f(n, 3), np.ones(n, np.float32), ptr, src.astype(np.int32)


# R disjoint copies of a graph have the gradients of one copy: the loss is a
# mean, and with R a power of two every value behind the sums is the copy's
# scaled by an exact 1/R (bf16 roundings included).  What differs is the order
# of the fp32 sums: chains of at most 64 additions of 2^-24 each (4e-6), with
# some room for cancellation between a copy's rows.
@pytest.mark.parametrize("n,copies", [(1, 16), (1, 32), (3, 8), (5, 4), (5, 16), (17, 2), (17, 64), (19, 512), (31, 1024),
                                      (33, 1), (1025, 16)])
def test_gradients_of_copies_are_those_of_one(pdg, n, copies):
    G, p, x, e, src, dst, deg, target, free, ptr, adj = path_problem(n, n)
    w = pdg.WarmStart(seed=1)
    w.set_params(G.flatten(p).astype(np.float32))
    one = G.unflatten(w.eval(x, ptr, adj, e, target, free)[2])
    rep = lambda a: np.tile(a, (copies,) + (1,) * (a.ndim - 1))
    ptr_r = np.concatenate([[0], np.cumsum(np.tile(deg, copies))]).astype(np.int32)
    adj_r = (np.tile(adj, copies) + n * np.repeat(np.arange(copies), len(adj))).astype(np.int32)
    args = (rep(x), ptr_r, adj_r, rep(e), rep(target), rep(free))
    flat = w.eval(*args)[2]
    assert np.array_equal(flat, w.eval(*args)[2])   # a fixed order
    many = G.unflatten(flat)
    for name, _ in G.shapes():
        a, b = one[name].reshape(-1), many[name].reshape(-1)
        assert np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(a) + 1e-12, name


def test_growing_and_shrinking_graphs_on_one_network(pdg):
    # the buffers of one network serve graphs of any size, in any order
    fresh = {}
    w = pdg.WarmStart(seed=1)
    for n in (33, 9729, 16, 1, 257, 9729, 33):
        G, p, x, e, src, dst, deg, target, free, ptr, adj = path_problem(n, n)
        flat = G.flatten(p).astype(np.float32)
        w.set_params(flat)
        got = w.eval(x, ptr, adj, e, target, free)
        if n not in fresh:
            w2 = pdg.WarmStart(seed=1)
            w2.set_params(flat)
            fresh[n] = w2.eval(x, ptr, adj, e, target, free)
        assert all(np.array_equal(a, b) for a, b in zip((got[0], got[2]), (fresh[n][0], fresh[n][2])))


@pytest.mark.parametrize("bad", ["asymmetric", "past the end", "negative"])
def test_bad_adjacency_is_refused(pdg, bad):
    G, p, x, e, src, dst, deg, target, free, ptr, adj = path_problem(33, 1)
    adj = adj.copy()
    adj[5] = {"asymmetric": 20, "past the end": 33, "negative": -1}[bad]
    w = pdg.WarmStart(seed=1)
    with pytest.raises(pdg.PDGError) as err:
        w.eval(x, ptr, adj, e, target, free)
    assert err.value.code == pdg.ERR_ARG
    G, p, x, e, src, dst, deg, target, free, ptr, adj = path_problem(33, 1)
    w.eval(x, ptr, adj, e, target, free)   # and the network is usable afterwards
