"""The reference-literal mode ignores a tolerance: it runs every sweep of the cap
and reports no residual, on every launch plan, whether the tolerance is there at
creation or comes later.  The iterates are the graph kernel's, bit for bit."""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def solver(pdg, kern, tol, nt=0):
    m = pdg.Mesh.hanging(33, 1.0, mtype=1, jitter=1e-4, seed=4, ncols=29)
    c = pdg.Constraints(m).build_stretch(1e3).build_bend(1e-2).pin_corners(29)
    return pdg.Solver(pdg.Config.default(max_iterations=6, rho=0.9, dt=1 / 60, gravity=-9.81, kernel=kern, tolerance=tol,
                                         mode=pdg.MODE_REFERENCE_LITERAL, block_threads=nt), m, c)


def frames(s):
    st = [s.step(1)[0] for _ in range(2)]
    return s.get_state(), [(f["iterations"], f["status"], f["converged"], f["res_final"]) for f in st]


@pytest.mark.parametrize("kern,nt", [("AUTO", 0), ("RESIDENT", 0), ("RESIDENT", 256), ("AUTOTUNE", 0), ("STREAM", 0)])
@pytest.mark.parametrize("tol,later", [(0.0, False), (1e-3, False), (1e-3, True)])
def test_literal_mode_runs_with_a_tolerance(pdg, kern, nt, tol, later):
    (xg, vg), sg = frames(solver(pdg, pdg.KERNEL_GRAPH, tol))
    assert [f[:3] for f in sg] == [(6, 0, 0)] * 2
    s = solver(pdg, getattr(pdg, "KERNEL_" + kern), 0.0 if later else tol, nt)
    if later:
        s.set_tolerance(tol)
    (x, v), st = frames(s)
    assert np.array_equal(x, xg) and np.array_equal(v, vg)
    assert st == sg


def test_command_line_takes_literal_with_a_tolerance(pdg):
    exe = os.path.join(ROOT, "cloth-cuda_gb300", "bin", "sim_cloth")
    p = subprocess.run([exe, "10", "10", "0.1", "--steps", "5", "--iter", "5", "--mode", "literal", "--tol", "1e-3",
                        "--pin", "corners"], stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True, timeout=120)
    assert p.returncode == 0, p.stderr
