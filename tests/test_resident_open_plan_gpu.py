"""The resident plan where the caller leaves it open: patches of up to 96 vertices
(160 with a tolerance) in 256-thread blocks, one per SM, then two per SM up to 160
and from 193 to 220, else the 512-thread blocks.  Same bits as the per-patch graph
kernel whatever the plan chose, for one cloth and for uneven ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(pdg, kern, shapes, tol, **plan):
    ms = [pdg.Mesh.hanging(r, 1.0, mtype=t, jitter=1e-4, seed=r, ncols=c) for r, c, t in shapes]
    cs = [pdg.Constraints(m).build_stretch(50.0).build_bend(1e-3).pin_corners(c) for m, (_, c, _) in zip(ms, shapes)]
    cfg = [pdg.Config.default(max_iterations=9, rho=0.9, dt=1 / 60, gravity=-9.81, kernel=kern, tolerance=tol, **plan)
           for _ in ms]
    s = pdg.Solver(cfg, ms, cs)
    st = s.step(2)
    states = [s.get_state(i) for i in range(len(ms))] if len(ms) > 1 else [s.get_state()]
    return states, [f["iterations"] for f in st], s.launch_info()


# 81 and 3,025 vertices (24 per patch), 9,409 (64, one per SM), 14,592 (96, one),
# 15,377 with cell centres (51, two; with a tolerance 104, one), 22,500 (75, two;
# 152, one), 46,000 (152, two), 47,961 (158, two), 50,625 (one of 352), 66,049 (218,
# two), 66,564 (219, two; 304 patches), 68,121 (one of 480); uneven cloths with a
# small last patch each
@pytest.mark.parametrize("shapes,threads", [
    ([(9, 9, 1)], 256), ([(55, 55, 0)], 256), ([(97, 97, 1)], 256), ([(114, 128, 2)], 256), ([(150, 150, 1)], 256), ([(200, 230, 1)], 256),
    ([(219, 219, 1)], 256), ([(225, 225, 1)], 512), ([(257, 257, 1)], 256), ([(258, 258, 0)], 256), ([(261, 261, 1)], 512), ([(77, 101, 3)], 256),
    ([(33, 41, 1), (17, 17, 2), (60, 33, 0), (2, 2, 1)], 256)])
@pytest.mark.parametrize("tol", [0.0, 1e-3])
def test_open_resident_plan_matches_graph(pdg, shapes, threads, tol):
    r = solve(pdg, pdg.KERNEL_RESIDENT, shapes, tol)
    assert r[2]["kernel"] == pdg.KERNEL_RESIDENT
    assert r[2]["block_threads"] == threads
    g = solve(pdg, pdg.KERNEL_GRAPH, shapes, tol, patch_verts=64, block_threads=128)
    assert g[1] == r[1]
    for (gx, gv), (rx, rv) in zip(g[0], r[0]):
        assert np.array_equal(gx, rx) and np.array_equal(gv, rv)
