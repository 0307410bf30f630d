"""A frame after one whose bounded waits ran out, from another state than the
failed frame's: nothing that frame left behind (offsets published to the
neighbours under tags that come again) is read.  Fixed sweep counts, a
tolerance, the caller's state moved by the frame, and a streaming plan whose
sweeps run in one launch, against the graph kernel, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 57


def cloth(pdg, kern, tol, nt=0):
    m = pdg.Mesh.hanging(N, 1.0, mtype=1, jitter=1e-4, seed=6)
    c = pdg.Constraints(m).build_stretch(5.0).build_bend(1e-3).pin_corners(N)
    return pdg.Solver(pdg.Config.default(max_iterations=20, rho=0.9, dt=1 / 60, gravity=-9.81, kernel=kern, tolerance=tol,
                                         block_threads=nt), m, c), m.arrays()["rest"]


def state(rest, seed):
    rng = np.random.default_rng(seed)
    wave = np.sin(rest[:, :1] * rng.uniform(3, 9, 3) + rest[:, 1:2] * rng.uniform(3, 9, 3)).astype(np.float32)
    return (rest + 0.01 * wave).astype(np.float32), rng.normal(0.0, 0.1, rest.shape).astype(np.float32)


# a budget of one cycle ends the first wait that is not over at once; 3,000
# cycles (a sweep or so) let the blocks publish some sweeps before they give up
@pytest.mark.parametrize("plan", [("RESIDENT", 0), ("RESIDENT", 256), ("RESIDENT", 512), ("STREAM", 0), ("STREAM", 128)])
@pytest.mark.parametrize("tol", [0.0, 0.3])
@pytest.mark.parametrize("budget", [1, 3000])
def test_frame_after_a_timeout_from_another_state(pdg, plan, tol, budget):
    g, rest = cloth(pdg, pdg.KERNEL_GRAPH, tol)
    s, _ = cloth(pdg, getattr(pdg, "KERNEL_" + plan[0]), tol, plan[1])
    for round in range(6):
        s.set_state(*state(rest, 2 * round))
        s.set_wait_budget(budget)
        try:
            s.step(1)
            assert budget > 1   # one cycle never suffices
        except pdg.PDGError as e:
            assert e.code == pdg.ERR_TIMEOUT
        s.set_wait_budget(2_000_000_000)
        x0, v0 = state(rest, 2 * round + 1)
        for k in (s, g):
            k.set_state(x0, v0)
        a, b = g.step(1)[0], s.step(1)[0]
        assert (a["iterations"], a["status"]) == (b["iterations"], b["status"])
        if plan[0] == "RESIDENT" and round % 2:   # and the caller's state moved by the frame itself
            x, v = np.empty_like(x0), np.empty_like(v0)
            s.step_host(x0, v0, x, v)
        else:
            x, v = s.get_state()
        assert np.array_equal(x, g.get_state()[0]) and np.array_equal(v, g.get_state()[1])
