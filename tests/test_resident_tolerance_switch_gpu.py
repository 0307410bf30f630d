"""A tolerance that comes and goes on one live solver.  The resident kernel's
frames alternate between two sets of sums and arrival counts, with a tolerance
or without: the frame that takes a tolerance up again must not see the counts of
the last one that had it.  Frames of both kinds in any order against the graph
kernel, bit for bit, sweep counts included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 0.3


def run(pdg, kern, nt, frames):
    m = pdg.Mesh.hanging(40, 0.5, mtype=1, jitter=1e-4, seed=3, ncols=37)
    c = pdg.Constraints(m).build_stretch(5.0).build_bend(1e-3).pin_corners(37)
    s = pdg.Solver(pdg.Config.default(max_iterations=60, rho=0.9, dt=1 / 60, gravity=-9.81, kernel=kern, tolerance=TOL,
                                      block_threads=nt), m, c)
    assert s.launch_info()["kernel"] == kern
    out, now = [], True
    for tol in frames:
        if tol != now:
            s.set_tolerance(TOL if tol else 0.0)
            now = tol
        st = s.step(1)[0]
        out.append((st["iterations"], st["status"], st["converged"], *s.get_state()))
    return out


# one tolerance frame or two, then 1, 2 and 3 fixed ones, twice over
@pytest.mark.parametrize("first", [1, 2])
@pytest.mark.parametrize("between", [1, 2, 3])
@pytest.mark.parametrize("nt", [0, 256, 512])
def test_tolerance_switched_off_and_on_matches_graph(pdg, first, between, nt):
    frames = ([True] * first + [False] * between) * 2 + [True] * 3
    g = run(pdg, pdg.KERNEL_GRAPH, 0, frames)
    r = run(pdg, pdg.KERNEL_RESIDENT, nt, frames)
    assert any(f[0] < 60 for f in g) and any(f[0] == 60 for f in g)   # both ends are met
    for a, b in zip(g, r):
        assert a[:3] == b[:3]
        assert np.array_equal(a[3], b[3]) and np.array_equal(a[4], b[4])
