"""A network that moves from one solver to another: who is attached to whom, in
every order of destruction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solver(pdg, n):
    m = pdg.Mesh.hanging(n, 1.0, mtype=1, jitter=1e-4, seed=n)
    c = pdg.Constraints(m).build_stretch(1e3).build_bend(1e-2).pin_corners(n)
    cfg = pdg.Config.default(max_iterations=6, rho=0.99, dt=1 / 60, gravity=-9.81, kernel=pdg.KERNEL_GRAPH,
                             init=pdg.INIT_WARMSTART_KEEP)
    return pdg.Solver(cfg, m, c)


def attached(pdg, w):
    """eval is refused while the network is attached."""
    z = np.zeros
    try:
        w.eval(z((1, 14)), np.zeros(2, np.int32), np.zeros(0, np.int32), z((0, 4)), z((1, 3)), np.ones(1))
        return False
    except pdg.PDGError as e:
        assert e.code == pdg.ERR_STATE
        return True


def test_closing_the_former_solver_leaves_the_network_attached(pdg):
    a, b = solver(pdg, 9), solver(pdg, 11)
    w = pdg.WarmStart(seed=1)
    w.attach(a)
    assert a.step(1)[0]["warm_start_used"] == 1
    w.attach(b)
    a.close()
    assert attached(pdg, w)
    assert b.step(1)[0]["warm_start_used"] == 1
    w.close()
    assert b.step(1)[0]["warm_start_used"] == 0
    b.close()


def test_the_former_solver_and_the_former_network_are_released(pdg):
    a, b = solver(pdg, 9), solver(pdg, 11)
    w, w2 = pdg.WarmStart(seed=1), pdg.WarmStart(seed=2)
    w.attach(a)
    w.attach(b)
    assert a.step(1)[0]["warm_start_used"] == 0   # a is on its own again
    w2.attach(b)                                  # b changes its network
    assert not attached(pdg, w) and attached(pdg, w2)
    w.close()
    assert b.step(1)[0]["warm_start_used"] == 1
    b.close()
    assert not attached(pdg, w2)
    a.close()
    w2.close()
