"""The small-step resolve form (k up to 64) where its parts can go wrong,
against the oracle: one and two rounds of neighbours, random candidates beyond
the texels held per thread, many maps, masks, guides of another size, far
neighbours, steps that score every candidate and steps that stop early, and
lists made in the step chain."""
import numpy as np
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,m", [(1, 1), (5, 130), (31, 8), (32, 64), (33, 65), (63, 5), (64, 100)])
@pytest.mark.parametrize("full", [0, 1 << 30])
def test_k_m(ts, oracle, wl, k, m, full):
    spec = wl.config1(out=40, ex=24)
    spec["out_w"], spec["out_h"] = 64, 40
    spec["params"].update(nearest_neighbors=k, random_sample_locations=m)
    got = ts.run_spec(spec, team_max_batch=1 << 30, team_full_max_batch=full)
    assert_same(got, oracle.run(spec, nthreads=4), "k %d m %d full %d" % (k, m, full))


@pytest.mark.parametrize("kind", ["maps", "mask", "guide_size", "far", "translucent", "sequential"])
@pytest.mark.parametrize("full", [0, 1 << 30])
def test_kinds(ts, oracle, wl, kind, full):
    spec = wl.config2(out=64, ex=32) if kind == "guide_size" else wl.config1(out=64, ex=32)
    spec["params"].update(nearest_neighbors=20, random_sample_locations=30)
    divisor = 8
    if kind == "maps":
        spec["examples"] = [{"image": wl.texture(400 + i, 11, 9 + i % 4)} for i in range(20)]
    elif kind == "mask":
        m = np.zeros((32, 32, 4), np.uint8)
        m[3:20, 5:30, 0] = 255
        spec["examples"][1].update(sample="image", mask=m)
    elif kind == "guide_size":
        spec["examples"][0]["guide"] = wl.example_guide(9, 24, 40, sigma=2.0)
    elif kind == "far":
        spec["out_w"], spec["out_h"] = 256, 64  # sparse first steps: neighbours beyond the padding
    elif kind == "translucent":
        spec["examples"][0]["image"][..., 3] = 90
    else:
        spec["out_w"], spec["out_h"], divisor = 48, 48, 0
    got = ts.run_spec(spec, batch_divisor=divisor, team_max_batch=1 << 30, team_full_max_batch=full)
    assert_same(got, oracle.run(spec, batch_divisor=divisor, nthreads=4), "%s full %d" % (kind, full))


def test_lone_request(ts, oracle, wl):
    """The served form's lone requests run it with lists made in the chain."""
    spec = wl.config0(out=64, ex=32)
    with ts.Server() as server:
        g, _ = server.wait(server.submit(ts.builder_from_spec(spec).build()))
        assert_same(ts.generated_outputs(g), oracle.run(spec, nthreads=4), "lone request")
