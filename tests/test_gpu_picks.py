"""The pick chain on the device, against the oracle: lists of few and many
pixels, random init (a list that is not identity), inpainting (a list of masked
pixels), no and many backtrack stages, stages that pick everything or nothing,
and the batched form."""
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def small(spec, **params):
    spec["params"].update({"nearest_neighbors": 5, "random_sample_locations": 3, **params})
    return spec


@pytest.mark.parametrize("w,h,params", [(1, 1, {}), (3, 2, {"random_init": 6}), (256, 128, {}),
                                        (181, 182, {"random_init": 500}), (151, 217, {"nearest_neighbors": 0}),
                                        (256, 256, {"backtrack_stages": 0}), (200, 200, {"backtrack_percent": 1.0}),
                                        (200, 201, {"backtrack_percent": 0.0}),
                                        (190, 190, {"backtrack_stages": 9, "random_init": 1, "seed": 7})])
def test_picks(ts, oracle, wl, w, h, params):
    spec = small(wl.config1(out=32, ex=24), **{"random_init": None, "tiling_mode": False, **params})
    spec["out_w"], spec["out_h"] = w, h
    assert_same(ts.run_spec(spec), oracle.run(spec, nthreads=8), "%dx%d %s" % (w, h, params))


@pytest.mark.parametrize("init", [None, 40])
def test_inpaint(ts, oracle, wl, init):
    spec = small(wl.inpaint_session(17, side=400), random_init=init)
    assert_same(ts.run_spec(spec), oracle.run(spec, nthreads=8), "inpaint")


@pytest.mark.parametrize("graph", [False, True])
def test_batched(ts, oracle, wl, graph):
    specs = [small(wl.config0(out=182, ex=24)), small(wl.config1(out=256, ex=24)), small(wl.config0(out=60, ex=20)),
             small(wl.inpaint_session(18, side=380))]
    batch = ts.Batch(graph=graph)
    for s in specs:
        batch.add(ts.builder_from_spec(s).build())
    for g, s in zip(batch.run(), specs):
        assert_same(ts.generated_outputs(g), oracle.run(s, nthreads=8), s["name"])


@pytest.mark.parametrize("kind", ["plain", "inpaint", "served"])
def test_many_random_init(ts, oracle, wl, kind):
    """More random-init pixels than a 64th: the unresolved list is kept whole."""
    spec = wl.inpaint_session(19, side=96) if kind == "inpaint" else wl.config0(out=90, ex=24)
    spec = small(spec, random_init=700)
    if kind == "served":
        server = ts.Server()
        got = ts.generated_outputs(server.wait(server.submit(ts.builder_from_spec(spec).build()))[0])
    else:
        got = ts.run_spec(spec)
    assert_same(got, oracle.run(spec, nthreads=8), kind)
