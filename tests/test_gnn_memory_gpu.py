"""What a network holds on the device: the partial sums of its gradients belong
to the backward pass, so a network that only infers has none, and they grow with
the graph without a trace in the results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ring(n, seed):
    """A closed chain of n nodes and random inputs on it."""
    rng = np.random.default_rng(seed)
    f = lambda *s: rng.normal(size=s).astype(np.float32)
    ptr = np.arange(0, 2 * n + 1, 2, dtype=np.int32)
    adj = np.stack([(np.arange(n) - 1) % n, (np.arange(n) + 1) % n], 1).astype(np.int32).ravel()
    return f(n, 14), ptr, adj, f(2 * n, 4), f(n, 3), np.ones(n, np.float32)


def network(pdg):
    w = pdg.WarmStart(seed=1)
    p = w.get_params()
    p[-195:] = np.random.default_rng(2).uniform(-0.2, 0.2, 195)   # a decoder that is not zero
    w.set_params(p)
    return w


def test_networks_without_a_backward_pass_stay_small(pdg):
    import torch
    first = network(pdg)
    before = torch.cuda.mem_get_info()[0]
    nets = [network(pdg) for _ in range(16)]
    # parameters, Adam's state and the bf16 copies: 0.8 MB each, in 2 MB pages
    assert before - torch.cuda.mem_get_info()[0] <= 16 * 4 * 2 ** 20
    del nets, first


# one block of the sums, the full number of blocks (9,728 rows and more), fewer again
def test_partial_sums_grow_with_the_graph(pdg):
    w = network(pdg)
    for n, seed in [(3, 1), (500, 2), (9729, 3), (40, 4), (12001, 5)]:
        g = ring(n, seed)
        got, want = w.eval(*g), network(pdg).eval(*g)
        assert np.array_equal(got[0], want[0]) and got[1] == want[1] and np.array_equal(got[2], want[2])
        assert np.abs(got[2]).max() > 0
