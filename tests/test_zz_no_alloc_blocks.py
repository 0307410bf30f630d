"""The allocation-free frame in each of its block sizes: cloths just above and
below the sizes where the launch takes more threads per block (152 blocks of
128, 256, 512, 640, 768 or 1,024 threads with one element each, then several
elements per thread), against the solver entry point; and where a tolerance ends
the sweeps.  Collected last, like the other tests of this entry point.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL_POS = 1e-5    # the bar of the other one-frame position comparisons
REL_VEL = 1e-3


def rel(a, b):
    a = np.asarray(a, np.float64).reshape(-1); b = np.asarray(b, np.float64).reshape(-1)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


def scene(pdg, n):
    m = pdg.Mesh.hanging(n, 1.0, mtype=1, jitter=1e-4, seed=n, ncols=n)
    c = pdg.Constraints(m).build_stretch(1e3)
    c.build_bend(1e-2)
    c.set_pins([0, n - 1])
    rng = np.random.default_rng(n)
    rest = m.arrays()["rest"]
    x0 = (rest + rng.normal(0.0, 1e-4, rest.shape)).astype(np.float32)
    v0 = rng.normal(0.0, 1e-2, rest.shape).astype(np.float32)
    return m, c, x0, v0


def frame(pdg, torch, cfg, m, c, x0, v0):
    a, ca = m.arrays(), c.arrays()
    dev = lambda t: torch.as_tensor(np.ascontiguousarray(t), device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr()) if t.numel() else None
    pos, vel = dev(x0), dev(v0)
    mass, diag, tris, dm, area, ks, quads, w, nr, kb, pins, tgt = [dev(t) for t in (
        a["mass"], c.jacobi_diag(cfg.dt), a["tris"], a["Dm_inv"], a["area"], ca["k_stretch"], ca["quads"], ca["w"],
        ca["n_rest"], ca["bend_k"], ca["pins"], ca["targets"])]
    torch.cuda.synchronize()
    st = pdg.FrameStats()
    rc = pdg.lib().pdg_step_noalloc(C.byref(cfg), m.N, ptr(pos), ptr(vel), ptr(mass), ptr(diag), m.T, ptr(tris),
                                    ptr(dm), ptr(area), ptr(ks), len(ca["bend_k"]), ptr(quads), ptr(w), ptr(nr),
                                    ptr(kb), len(ca["pins"]), ptr(pins), ptr(tgt), None, C.byref(st))
    assert rc == 0, pdg.lib().pdg_last_error_string()
    return pos.cpu().numpy(), vel.cpu().numpy(), st


# triangles and hinges: 17,287 (blocks of 128), 19,719 (256), 39,427 (512), 77,875
# (640), 97,720 (768), 116,739 and 154,528 (1,024), 156,291 (several per thread)
@pytest.mark.parametrize("n", [60, 64, 90, 126, 141, 154, 177, 178])
def test_noalloc_matches_the_solver_in_each_block_size(pdg, n):
    torch = pytest.importorskip("torch")
    m, c, x0, v0 = scene(pdg, n)
    cfg = pdg.Config.default(max_iterations=6, rho=0.99, dt=1 / 60, gravity=-9.81, kernel=pdg.KERNEL_GRAPH)
    s = pdg.Solver(cfg, m, c)
    s.set_state(x0, v0)
    ref = s.step(1)[0]
    x_ref, v_ref = s.get_state()
    pos, vel, st = frame(pdg, torch, cfg, m, c, x0, v0)
    assert st.status == 0 and st.iterations == 6
    assert rel(pos, x_ref) < REL_POS
    assert rel(vel, v_ref) < REL_VEL
    assert abs(st.res_final - ref["res_final"]) <= 1e-3 * ref["res_final"] + 1e-12


# where the tolerance ends the sweeps, the frame is that of a cap at that sweep
@pytest.mark.parametrize("n", [9, 64, 178])
def test_noalloc_stopped_by_its_tolerance_is_the_frame_of_that_cap(pdg, n):
    torch = pytest.importorskip("torch")
    m, c, x0, v0 = scene(pdg, n)
    kw = dict(dt=1 / 60, gravity=-9.81, kernel=pdg.KERNEL_GRAPH, use_chebyshev=0)
    pos, vel, st = frame(pdg, torch, pdg.Config.default(max_iterations=200, tolerance=0.5, **kw), m, c, x0, v0)
    assert st.status == 0 and st.converged == 1 and 0 < st.iterations < 200
    assert st.res_final <= 0.5 * st.res_inertial
    p2, v2, s2 = frame(pdg, torch, pdg.Config.default(max_iterations=st.iterations, **kw), m, c, x0, v0)
    assert s2.iterations == st.iterations
    assert rel(pos, p2) < REL_POS and rel(vel, v2) < REL_VEL
