"""Neighbour lists over the short resolved lists of the sparse first steps,
against the oracle: fewer points than k, clustered points (inpainting with a
few locked pixels in a corner: the density says nothing of the distance),
tiling mirrors, large k, exact and inexact sums."""
import numpy as np
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,k,tiling", [(128, 128, 1, True), (300, 180, 50, True), (512, 64, 256, True),
                                          (257, 129, 100, False)])
def test_sparse_steps(ts, oracle, wl, w, h, k, tiling):
    spec = wl.config1(out=64, ex=24)
    spec["out_w"], spec["out_h"] = w, h
    spec["params"].update(nearest_neighbors=k, random_sample_locations=4, tiling_mode=tiling, random_init=7,
                          backtrack_stages=6)
    got = ts.run_spec(spec)
    assert_same(got, oracle.run(spec, nthreads=8), "%dx%d k %d" % (w, h, k))


@pytest.mark.parametrize("w,h,k", [(256, 64, 50), (150, 130, 20)])
def test_clustered_points(ts, oracle, wl, w, h, k):
    spec = wl.inpaint_session(3, side=32)
    spec["out_w"], spec["out_h"] = w, h
    spec["examples"] = [{"image": wl.texture(22, h, w)}]
    mask = np.zeros((h, w, 4), np.uint8)
    mask[:9, :7] = 255  # 63 locked pixels in a corner
    spec["inpaint_mask"] = mask
    spec["params"].update(nearest_neighbors=k, random_sample_locations=4)
    got = ts.run_spec(spec)
    assert_same(got, oracle.run(spec, nthreads=8), "clustered %dx%d k %d" % (w, h, k))


def test_far_cluster_sums(ts, oracle, wl):
    """A locked block of 32 x 19 pixels at one end of the widest output: 19 of
    an item's neighbours fall to one lane, each up to 16383 columns away, so
    that their squared offsets pass 2^32 (19 * 15035^2).  The sample mask
    leaves the far items their random candidates, whose scores hold the
    weights (a neighbour's own candidate would match the block exactly)."""
    w, h, k = 16384, 32, 256
    spec = wl.inpaint_session(3, side=32)
    spec["out_w"], spec["out_h"] = w, h
    sample = np.zeros((h, w, 4), np.uint8)
    sample[:, :256] = 255
    spec["examples"] = [{"image": wl.texture(22, h, w), "sample": "image", "mask": sample}]
    mask = np.zeros((h, w, 4), np.uint8)
    mask[:19, :32] = 255
    spec["inpaint_mask"] = mask
    spec["params"].update(nearest_neighbors=k, random_sample_locations=2, backtrack_stages=0)
    got = ts.run_spec(spec, batch_divisor=1)
    assert got["stats"]["knn_chunks"] > 0
    assert_same(got, oracle.run(spec, batch_divisor=1, nthreads=16), "far cluster")
