"""The allocation-free frame at the sizes where its launch changes: one block,
blocks with idle threads, one element per thread at most (the constants stay
in registers), several elements per thread, and the vertex limit, against the
solver entry point.  Collected last, like the other tests of this entry point.
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


# (rows, cols, bend): 2x2 without and with its one hinge; 9x40; 129x200: 76,000
# elements on fewer threads than are resident; 181x240: 216,000 elements, more
# than the resident threads; 512x256 = the vertex limit
@pytest.mark.parametrize("rows,cols,bend", [(2, 2, 0.0), (2, 2, 1e-2), (9, 40, 1e-2), (129, 200, 1e-2),
                                            (181, 240, 1e-2), (512, 256, 1e-2)])
def test_noalloc_matches_the_solver_over_its_sizes(pdg, rows, cols, bend):
    torch = pytest.importorskip("torch")
    m = pdg.Mesh.hanging(rows, 1.0, mtype=1, jitter=1e-4, seed=rows, ncols=cols)
    c = pdg.Constraints(m).build_stretch(1e3)
    if bend:
        c.build_bend(bend)
    c.set_pins([0, cols - 1])
    cfg = pdg.Config.default(max_iterations=6, rho=0.99, dt=1 / 60, gravity=-9.81, kernel=pdg.KERNEL_GRAPH,
                             wind=(0.3, 0.0, -0.2))
    a, ca = m.arrays(), c.arrays()
    rng = np.random.default_rng(rows)
    x0 = (a["rest"] + rng.normal(0.0, 1e-4, a["rest"].shape)).astype(np.float32)
    v0 = rng.normal(0.0, 1e-2, a["rest"].shape).astype(np.float32)
    s = pdg.Solver(cfg, m, c)
    s.set_state(x0, v0)
    ref = s.step(1)[0]
    x_ref, v_ref = s.get_state()

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
    assert st.status == 0 and st.iterations == 6
    assert rel(pos.cpu().numpy(), x_ref) < REL_POS
    assert rel(vel.cpu().numpy(), v_ref) < REL_VEL
    assert abs(st.res_final - ref["res_final"]) <= 1e-3 * ref["res_final"] + 1e-12
