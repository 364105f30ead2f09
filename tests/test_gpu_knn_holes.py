"""Neighbours of pixels deep inside a hole of a dense image (inpainting),
where the ring search meets thousands of points at the hole's rim, and walks
at image edges, around the table's radius and with runs of several items per
warp, against the oracle."""
import numpy as np
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,hole,k,tiling", [(256, 128, (60, 14, 190, 114), 50, False),
                                               (200, 170, (5, 5, 180, 165), 8, True),
                                               (200, 170, (40, 30, 170, 150), 256, False),
                                               (128, 128, (0, 0, 128, 90), 20, True)])
def test_holes(ts, oracle, wl, w, h, hole, k, tiling):
    spec = wl.inpaint_session(3, side=32)
    spec["out_w"], spec["out_h"] = w, h
    spec["examples"] = [{"image": wl.texture(21, h, w)}]
    mask = np.full((h, w, 4), 255, np.uint8)
    mask[hole[1]:hole[3], hole[0]:hole[2], :3] = 0
    spec["inpaint_mask"] = mask
    spec["params"].update(nearest_neighbors=k, random_sample_locations=5, tiling_mode=tiling, backtrack_stages=3)
    got = ts.run_spec(spec)
    assert_same(got, oracle.run(spec, nthreads=8), "hole %s in %dx%d k %d" % (hole, w, h, k))


@pytest.mark.parametrize("w,h,tiling", [(320, 300, True), (512, 256, False)])
def test_runs_of_items(ts, oracle, wl, w, h, tiling):
    """Launches of more items than warps: each warp walks several."""
    spec = wl.config1(out=64, ex=24)
    spec["out_w"], spec["out_h"] = w, h
    spec["params"].update(nearest_neighbors=9, random_sample_locations=3, tiling_mode=tiling, backtrack_stages=2)
    got = ts.run_spec(spec)
    assert_same(got, oracle.run(spec, nthreads=8), "%dx%d" % (w, h))
