"""The streaming kernel with more patches than are resident at once (fewer run as
one launch of the resident kernel): its instances with constant strides and the
general one, full and ragged patches, valence above ten, and the patch size that
the plan chooses, against the per-patch graph kernel, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(pdg, kern, rows, cols, mtype, pv, nt, tol):
    m = pdg.Mesh.hanging(rows, 1.0, mtype=mtype, jitter=1e-4, seed=rows, ncols=cols)
    c = pdg.Constraints(m).build_stretch(50.0).build_bend(1e-3).pin_corners(cols)
    cfg = pdg.Config.default(max_iterations=7, rho=0.9, dt=1 / 60, gravity=-9.81, kernel=kern, tolerance=tol,
                             patch_verts=pv, block_threads=nt)
    s = pdg.Solver(cfg, m, c)
    l0 = s.launches
    st = [s.step(1)[0] for _ in range(2)]
    return s.get_state(), st, s.launches - l0, s.launch_info()


# (rows, cols, mesh type, patch vertices, block threads): 128-vertex patches of a
# regular grid, the last one of 80; 256, the last one of 41; 625 small patches,
# whose slot stride is not the constant; valence 8 with two hinges each (more
# than ten contributions); 512 threads
@pytest.mark.parametrize("rows,cols,mtype,pv,nt", [(300, 300, 1, 128, 128), (301, 349, 2, 256, 256),
                                                   (100, 100, 1, 16, 128), (200, 211, 3, 128, 128),
                                                   (300, 277, 3, 256, 256), (401, 399, 0, 512, 512)])
@pytest.mark.parametrize("tol", [0.0, 0.7])
def test_stream_instances_match_graph(pdg, rows, cols, mtype, pv, nt, tol):
    g = solve(pdg, pdg.KERNEL_GRAPH, rows, cols, mtype, pv, nt, tol)
    r = solve(pdg, pdg.KERNEL_STREAM, rows, cols, mtype, pv, nt, tol)
    assert r[2] == 2 * (4 + 8)   # a launch per sweep: not the resident kernel's range
    assert [f["iterations"] for f in g[1]] == [f["iterations"] for f in r[1]]
    assert np.array_equal(g[0][0], r[0][0]) and np.array_equal(g[0][1], r[0][1])
    # (the sums of the patches' residuals are added in any order)
    for a, b in zip(g[1], r[1]):
        assert abs(a["res_final"] - b["res_final"]) <= 1e-5 * abs(a["res_final"])


# all patches resident: 379 of 128 vertices (two rounds of 128 threads), and the
# open plan with one patch per SM (152 vertices), two (160) and two of 198
@pytest.mark.parametrize("rows,cols,pv,nt", [(220, 220, 128, 128), (150, 150, 0, 0), (220, 220, 0, 0), (240, 250, 0, 0)])
@pytest.mark.parametrize("tol", [0.0, 0.7])
def test_resident_stream_plans_match_graph(pdg, rows, cols, pv, nt, tol):
    r = solve(pdg, pdg.KERNEL_STREAM, rows, cols, 1, pv, nt, tol)
    assert r[2] == 2 * 5   # the sweeps in one launch
    g = solve(pdg, pdg.KERNEL_GRAPH, rows, cols, 1, 128, 128, tol)
    assert [f["iterations"] for f in g[1]] == [f["iterations"] for f in r[1]]
    assert np.array_equal(g[0][0], r[0][0]) and np.array_equal(g[0][1], r[0][1])


# the network's messages are summed in one order whatever the plan: a random
# network, its start always kept, on the open plan and on the 256-vertex one
def test_network_start_does_not_depend_on_the_plan(pdg):
    import scenes
    out = []
    for plan in ({}, dict(patch_verts=256, block_threads=256)):
        ms, cs, cfg, _ = scenes.batch(5, seed=11, n_range=(17, 49), max_iterations=6, tolerance=0.0,
                                      kernel=pdg.KERNEL_STREAM, init=pdg.INIT_WARMSTART_KEEP, **plan)
        s = pdg.Solver(cfg, ms, cs)
        w = pdg.WarmStart(seed=4)
        p = w.get_params()
        w.set_params((p + np.random.default_rng(3).normal(0.0, 0.02, p.shape)).astype(np.float32))
        w.attach(s)
        s.step(2)
        out.append((s.launch_info()["patch_verts"], [s.get_state(i)[0] for i in range(len(ms))]))
        s.close(); w.close()
    assert out[0][0] != 256
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)


# 333x500: 192 vertices fill the last wave of blocks better on 152 SMs; 512x513:
# 1,026 patches of 256 (2.25 waves) or 1,368 of 192 (three)
@pytest.mark.parametrize("rows,cols", [(333, 500), (512, 513)])
def test_open_patch_size_matches_graph(pdg, rows, cols):
    r = solve(pdg, pdg.KERNEL_STREAM, rows, cols, 1, 0, 0, 0.0)
    assert r[3]["patch_verts"] in (192, 256) and r[3]["block_threads"] == 256
    g = solve(pdg, pdg.KERNEL_GRAPH, rows, cols, 1, r[3]["patch_verts"], 256, 0.0)
    assert np.array_equal(g[0][0], r[0][0]) and np.array_equal(g[0][1], r[0][1])
