"""A training pair whose solvers left the patch size open: the streaming plan may
choose one for the deep solver that the trajectory's solver does not have.  The
step is then that of a pair with the size given, to the rounding of the deep
solve (its sums follow its own vertex order); sizes that differ because the
caller gave them are refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solvers(pdg, kern, traj_plan, deep_plan):
    m = pdg.Mesh.hanging(333, 1.0, mtype=2, jitter=1e-3, seed=3, ncols=500)
    c = pdg.Constraints(m).build_stretch(1e3).build_bend(1e-2).pin_corners(500)
    out = []
    for cap, k, init, plan in ((4, kern, pdg.INIT_WARMSTART, traj_plan), (12, pdg.KERNEL_STREAM, pdg.INIT_INERTIAL, deep_plan)):
        out.append(pdg.Solver([pdg.Config.default(max_iterations=cap, rho=0.99, dt=1 / 60, gravity=-9.81, kernel=k,
                                                  init=init, **plan)], [m], [c]))
    return out


# x of about 1 rounds to 1e-7, which the network's offset scale of 2.7e-3 makes
# 4e-5 of a target of order one: the loss agrees to a few times that
@pytest.mark.parametrize("kern", ["KERNEL_STREAM", "KERNEL_GRAPH"])
def test_pair_with_an_open_patch_size_trains_like_one_with_it_given(pdg, kern):
    given = dict(patch_verts=256, block_threads=256)
    runs = []
    for deep_plan in ({}, given):
        traj, deep = solvers(pdg, getattr(pdg, kern), {}, deep_plan)
        w = pdg.WarmStart(seed=2)
        w.attach(traj)
        loss = [w.train_pair(traj, deep, 1e-4) for _ in range(2)]
        runs.append((loss, w.get_params(), deep.launch_info()["patch_verts"], traj.get_state()[0]))
        traj.close(); deep.close(); w.close()
    assert runs[1][2] == 256
    if runs[0][2] == 256:
        pytest.skip("the plan keeps 256 vertices per patch on this device")
    assert np.array_equal(runs[0][3], runs[1][3])   # the trajectory has the same plan in both
    assert np.allclose(runs[0][0], runs[1][0], rtol=2e-4)
    a, b = runs[0][1].astype(np.float64), runs[1][1].astype(np.float64)
    assert np.linalg.norm(a - b) <= 1e-3 * np.linalg.norm(b)


def test_pair_with_different_given_patch_sizes_is_refused(pdg):
    traj, deep = solvers(pdg, pdg.KERNEL_STREAM, {}, dict(patch_verts=128, block_threads=128))
    w = pdg.WarmStart(seed=2)
    w.attach(traj)
    with pytest.raises(Exception):
        w.train_pair(traj, deep, 1e-4)
    traj.close(); deep.close(); w.close()
