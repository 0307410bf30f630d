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
