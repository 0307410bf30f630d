"""The resident kernel where its plan changes: patches whose records fit one
round of the block's threads (one local step per sweep) and patches that need
two, both block sizes, fixed sweep counts and tolerances, against the
per-patch graph kernel, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (rows, cols, mesh type, patch vertices, block threads): record counts below,
# around and above the 480 (block 512) and 224 (block 256) compute threads;
# ragged sides leave a small last patch; type 3 has valence 8
PLANS = [(33, 33, 1, 32, 0), (41, 29, 2, 96, 256), (41, 29, 2, 160, 256), (41, 29, 0, 224, 256),
         (65, 61, 1, 288, 0), (65, 61, 1, 352, 0), (65, 61, 1, 384, 0), (65, 61, 2, 480, 0), (40, 33, 3, 256, 0)]


@pytest.mark.parametrize("rows,cols,mtype,pv,nt", PLANS)
@pytest.mark.parametrize("cap,final", [(1, 1), (2, 1), (9, 1), (40, 1), (7, 0)])
def test_resident_plans_match_graph_bitwise(pdg, rows, cols, mtype, pv, nt, cap, final):
    m = pdg.Mesh.hanging(rows, 1.0, mtype=mtype, jitter=1e-4, seed=rows, ncols=cols)
    c = pdg.Constraints(m).build_stretch(1e3).build_bend(1e-2).set_pins([0, cols - 1])
    out = []
    for kern in (pdg.KERNEL_GRAPH, pdg.KERNEL_RESIDENT):
        cfg = pdg.Config.default(max_iterations=cap, rho=0.99, dt=1 / 60, gravity=-9.81, kernel=kern, wind=(0.3, 0, -0.2),
                                 compute_final_residual=final)
        if kern == pdg.KERNEL_RESIDENT:
            cfg.patch_verts, cfg.block_threads = pv, nt
        s = pdg.Solver(cfg, m, c)
        assert s.launch_info()["kernel"] == kern
        st = s.step(3)[0]
        out.append((s.get_state(), st))
    (g, sg), (r, sr) = out
    assert np.array_equal(g[0], r[0]) and np.array_equal(g[1], r[1])
    assert (sg["iterations"], sg["status"], sg["converged"]) == (sr["iterations"], sr["status"], sr["converged"])
    assert abs(sg["res_final"] - sr["res_final"]) <= 1e-5 * abs(sg["res_final"])


# Tolerances: the resident kernel takes its decision about sweep k before sweep
# k + 2 and steps back; iterates and sweep counts must be those of the graph
# kernel, which decides before every sweep.  2.0 stops at the start iterate;
# the caps end the frame before, at and after the lag.
@pytest.mark.parametrize("tol", [2.0, 0.5, 1e-1, 1e-2, 1e-4])
@pytest.mark.parametrize("cap", [0, 1, 2, 3, 4, 17, 400])
@pytest.mark.parametrize("nt", [0, 256])
def test_resident_tolerance_matches_graph(pdg, tol, cap, nt):
    m = pdg.Mesh.hanging(24, 0.5, mtype=1, jitter=1e-4, seed=3, ncols=21)
    c = pdg.Constraints(m).build_stretch(20.0).build_bend(1e-3).pin_corners(21)
    out = []
    for kern in (pdg.KERNEL_GRAPH, pdg.KERNEL_RESIDENT):
        cfg = pdg.Config.default(max_iterations=cap, rho=0.9, dt=1 / 60, gravity=-9.81, kernel=kern, tolerance=tol)
        if kern == pdg.KERNEL_RESIDENT:
            cfg.block_threads = nt
        s = pdg.Solver(cfg, m, c)
        st = [s.step(1)[0] for _ in range(3)]
        out.append((s.get_state(), st))
    (g, sg), (r, sr) = out
    assert [f["iterations"] for f in sg] == [f["iterations"] for f in sr]
    assert [f["converged"] for f in sg] == [f["converged"] for f in sr]
    assert np.array_equal(g[0], r[0]) and np.array_equal(g[1], r[1])
    for a, b in zip(sg, sr):
        assert abs(a["res_final"] - b["res_final"]) <= 1e-5 * abs(a["res_final"])


@pytest.mark.parametrize("final", [0, 1])
def test_resident_batch_of_caps_and_tolerances_matches_graph(pdg, final):
    # each cloth has its own cap and tolerance (0: none), the first one none:
    # with final = 0 the frame then has no residual sweep
    sizes, caps, tols = (9, 21, 33, 12, 17), (30, 7, 30, 1, 0), (0.0, 1e-2, 1e-3, 1e-1, 1e-2)
    ms = [pdg.Mesh.hanging(n, 0.5, mtype=1, jitter=1e-4, seed=n) for n in sizes]
    cs = [pdg.Constraints(m).build_stretch(20.0).build_bend(1e-3).pin_corners(n) for m, n in zip(ms, sizes)]
    out = []
    for kern in (pdg.KERNEL_GRAPH, pdg.KERNEL_RESIDENT):
        cfgs = [pdg.Config.default(max_iterations=k, rho=0.9, dt=1 / 60, gravity=-9.81, kernel=kern, tolerance=t,
                                   compute_final_residual=final) for k, t in zip(caps, tols)]
        s = pdg.Solver(cfgs, ms, cs)
        st = [s.step(1) for _ in range(3)]
        out.append((s.get_state_all(), [[f["iterations"] for f in r] for r in st], [[f["converged"] for f in r] for r in st]))
    (g, ig, cg), (r, ir, cr) = out
    assert ig == ir and cg == cr
    assert np.array_equal(g[0], r[0]) and np.array_equal(g[1], r[1])


def test_resident_tolerance_frame_that_fails_stops_like_graph(pdg):
    # a NaN in the state: the record says where, x is kept and v is zero
    m = pdg.Mesh.hanging(17, 1.0, mtype=1, jitter=1e-4, seed=3)
    c = pdg.Constraints(m).build_stretch(1e3).build_bend(1e-2).pin_corners(17)
    out = []
    for kern in (pdg.KERNEL_GRAPH, pdg.KERNEL_RESIDENT):
        cfg = pdg.Config.default(max_iterations=12, rho=0.99, dt=1 / 60, gravity=-9.81, kernel=kern, tolerance=1e-3)
        s = pdg.Solver(cfg, m, c)
        x = m.arrays()["rest"].copy()
        x[100, 1] = np.nan
        s.set_state(x, np.zeros_like(x))
        st = s.step(1)[0]
        out.append((s.get_state(), st["status"], st["iterations"]))
    assert out[0][1] == pdg.ERR_NUMERIC and out[0][1:] == out[1][1:]
    assert np.array_equal(out[0][0][0], out[1][0][0], equal_nan=True) and np.array_equal(out[0][0][1], out[1][0][1])


# Streaming plans whose patches are all resident at once run their sweeps in
# one launch of the resident kernel: the same matrix, with the three block
# sizes (patches of 64 and 128 vertices, 200, 256) and two launches around a
# judged start.
@pytest.mark.parametrize("pv,nt", [(64, 128), (128, 128), (200, 256), (256, 256)])
@pytest.mark.parametrize("cap,tol,final", [(0, 0.0, 1), (1, 0.0, 0), (1, 1e-2, 1), (2, 2.0, 1), (3, 1e-1, 1), (17, 1e-2, 1),
                                           (18, 0.0, 0), (400, 1e-4, 1)])
def test_stream_ranges_match_graph(pdg, pv, nt, cap, tol, final):
    m = pdg.Mesh.hanging(40, 0.5, mtype=1, jitter=1e-4, seed=3, ncols=37)
    c = pdg.Constraints(m).build_stretch(20.0).build_bend(1e-3).pin_corners(37)
    out = []
    for kern in (pdg.KERNEL_GRAPH, pdg.KERNEL_STREAM):
        cfg = pdg.Config.default(max_iterations=cap, rho=0.9, dt=1 / 60, gravity=-9.81, kernel=kern, tolerance=tol,
                                 compute_final_residual=final, patch_verts=pv, block_threads=nt)
        s = pdg.Solver(cfg, m, c)
        assert s.launch_info()["kernel"] == kern
        l0 = s.launches
        st = [s.step(1)[0] for _ in range(3)]
        out.append((s.get_state(), st, s.launches - l0))
    (g, sg, _), (r, sr, nl) = out
    assert nl == 3 * 5   # reset, prediction, sweeps, statistics, finalisation
    assert [f["iterations"] for f in sg] == [f["iterations"] for f in sr]
    assert [f["converged"] for f in sg] == [f["converged"] for f in sr]
    assert np.array_equal(g[0], r[0]) and np.array_equal(g[1], r[1])
    for a, b in zip(sg, sr):
        assert abs(a["res_final"] - b["res_final"]) <= 1e-5 * abs(a["res_final"])
        assert abs(a["res_inertial"] - b["res_inertial"]) <= 1e-5 * abs(a["res_inertial"])


@pytest.mark.parametrize("judge", [0, 1, 3])
@pytest.mark.parametrize("keep", [False, True])
def test_learned_batch_on_stream_ranges_matches_graph(pdg, judge, keep):
    sizes, caps, tols = (9, 21, 33, 12), (30, 7, 30, 1), (0.0, 1e-2, 1e-3, 1e-1)
    ms = [pdg.Mesh.hanging(n, 0.5, mtype=1, jitter=1e-4, seed=n) for n in sizes]
    cs = [pdg.Constraints(m).build_stretch(20.0).build_bend(1e-3).pin_corners(n) for m, n in zip(ms, sizes)]
    w = pdg.WarmStart(seed=3)
    p = w.get_params()
    p[-195:] = np.random.default_rng(1).uniform(-0.2, 0.2, 195)   # a decoder that is not zero
    out = []
    for kern in (pdg.KERNEL_GRAPH, pdg.KERNEL_STREAM):
        cfgs = [pdg.Config.default(max_iterations=k, rho=0.9, dt=1 / 60, gravity=-9.81, kernel=kern, tolerance=t,
                                   init=pdg.INIT_WARMSTART_KEEP if keep and i == 2 else pdg.INIT_WARMSTART,
                                   patch_verts=128, block_threads=128) for i, (k, t) in enumerate(zip(caps, tols))]
        s = pdg.Solver(cfgs, ms, cs)
        w = pdg.WarmStart(seed=3)
        w.set_params(p)
        w.set_judge_sweeps(judge)
        w.attach(s)
        st = [s.step(1) for _ in range(4)]
        out.append((s.get_state_all(), [[(f["iterations"], f["warm_start_used"], f["converged"]) for f in r] for r in st]))
    assert out[0][1] == out[1][1]
    assert np.array_equal(out[0][0][0], out[1][0][0]) and np.array_equal(out[0][0][1], out[1][0][1])
