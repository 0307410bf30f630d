"""The patch size of a streaming plan left open: 192 vertices only where they are
clearly the faster ones of the two, with few waves of blocks and with many (on 152
SMs)."""
import pytest

pytestmark = pytest.mark.gpu


# us per sweep at 192 / 256 vertices: 290x290 7.1 / 8.0 (one wave), 400x400 12.0 /
# 13.5, 333x500 11.7 / 13.5, 485x485 16.2 / 15.05 (2.02 waves of 256), 513x513 17.0 /
# 17.4 (within what the estimate is good for), 640x640 25.7 / 25.2, 768x768 37.0 /
# 32.0 (5.05 waves of 256, 6.7 of 192), 769x769 35.8 / 31.9
@pytest.mark.parametrize("rows,cols,size", [(290, 290, 192), (400, 400, 192), (333, 500, 192), (485, 485, 256), (513, 513, 256),
                                            (640, 640, 256), (768, 768, 256), (769, 769, 256)])
def test_open_patch_size_is_the_faster_one(pdg, rows, cols, size):
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("measured on 152 SMs")
    m = pdg.Mesh.hanging(rows, 1.0, mtype=1, jitter=1e-4, seed=1, ncols=cols)
    c = pdg.Constraints(m).build_stretch(1e3).build_bend(1e-2).pin_corners(cols)
    s = pdg.Solver(pdg.Config.default(max_iterations=5, kernel=pdg.KERNEL_STREAM), m, c)
    i = s.launch_info()
    assert (i["kernel"], i["patch_verts"], i["block_threads"]) == (pdg.KERNEL_STREAM, size, 256)


# many cloths: 5.2 and 14.5 waves of 256 vertices (96 cloths 34.4 us per sweep at 192, 32.6 at 256)
@pytest.mark.parametrize("count", [96, 256])
def test_open_patch_size_of_a_batch(pdg, count):
    import scenes
    ms, cs, cfg, _ = scenes.batch(count, 0, max_iterations=5, tolerance=0.0, kernel=pdg.KERNEL_STREAM)
    assert pdg.Solver(cfg, ms, cs).launch_info()["patch_verts"] == 256
