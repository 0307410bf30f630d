"""Gradients of the warm-start network where the weight-gradient kernel's tiling
changes: around 16- and 32-row tiles, one tile per block and several, no rows
left for some blocks.  The bounds are those of the 30x30 comparison (bf16).
"""
import numpy as np
import pytest

from test_gnn_gpu import bf16_round

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


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 257, 9728, 9729, 19500])
def test_gradients_at_tile_edges_match_oracle(pdg, n):
    G, p, x, e, src, dst, deg, target, free, ptr, adj = path_problem(n, n)
    flat = G.flatten(p).astype(np.float32)
    w = pdg.WarmStart(seed=1)
    w.set_params(flat)
    out, loss, grads = w.eval(x, ptr, adj, e, target, free)
    again = w.eval(x, ptr, adj, e, target, free)[2]
    assert np.array_equal(grads, again)   # a fixed order
    pb = dict(G.unflatten(flat))
    for k in pb:
        if k[0] in "WABU":
            pb[k] = bf16_round(pb[k]).astype(np.float64)
    lo, go, oo = G.loss_and_grad(pb, bf16_round(x).astype(np.float64), e.astype(np.float64), src, dst, deg,
                                 target.astype(np.float64), free.astype(np.float64))
    assert abs(loss - lo) <= 2e-2 * lo
    assert np.linalg.norm(out - oo) <= 2e-2 * np.linalg.norm(oo)
    gg = G.unflatten(grads)
    for name, _ in G.shapes():
        a, b = gg[name].reshape(-1), go[name].reshape(-1)
        assert np.linalg.norm(a - b) <= 6e-2 * np.linalg.norm(b) + 1e-6, name


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
