"""The plain path's k-NN made ahead for outputs whose sides are not powers of
two (means by f64 chains, distances from the coordinate tables), against the
oracle: around the smallest such output, item counts around a mean block,
neighbours beyond the tables' radius, tiling mirrors, guides, inpainting."""
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,k,tiling,ahead", [(45, 45, 12, False, False), (46, 45, 12, True, True),
                                                (64, 65, 1, True, True), (97, 33, 65, True, True),
                                                (300, 7, 50, False, True), (71, 53, 256, False, True)])
def test_sizes(ts, oracle, wl, w, h, k, tiling, ahead):
    spec = wl.config1(out=32, ex=24)
    spec["out_w"], spec["out_h"] = w, h
    spec["params"].update(nearest_neighbors=k, random_sample_locations=9, tiling_mode=tiling)
    got = ts.run_spec(spec)
    assert_same(got, oracle.run(spec, nthreads=4), "%dx%d k %d" % (w, h, k))
    assert (got["stats"]["knn_chunks"] > 0) == ahead


@pytest.mark.parametrize("kind", ["guided", "inpaint", "sequential"])
def test_kinds(ts, oracle, wl, kind):
    spec = {"guided": wl.config2(out=60, ex=40), "inpaint": wl.inpaint_session(5, side=75),
            "sequential": wl.config0(out=47, ex=24)}[kind]
    divisor = 0 if kind == "sequential" else 8
    got = ts.run_spec(spec, batch_divisor=divisor)
    assert_same(got, oracle.run(spec, batch_divisor=divisor, nthreads=4), kind)
    assert got["stats"]["knn_chunks"] > 0
