"""Batched sessions whose neighbour lists are made ahead, against the oracle:
more sessions than streams, outputs above and below the size that makes its
lists ahead, power-of-two sides, no neighbours, guides, tiling, inpainting,
random init, no backtracking."""
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def specs_of(wl):
    def sized(spec, w, h, **params):
        spec["out_w"], spec["out_h"] = w, h
        spec["params"].update({"nearest_neighbors": 6, "random_sample_locations": 4, **params})
        return spec

    c = [sized(wl.config0(out=32, ex=20), 32, 32), sized(wl.config0(out=32, ex=20), 64, 64),
         sized(wl.config0(out=32, ex=24), 47, 44), sized(wl.config1(out=32, ex=24), 101, 33, nearest_neighbors=9),
         sized(wl.config1(out=32, ex=24), 20, 20), sized(wl.config0(out=32, ex=20), 60, 60, nearest_neighbors=0),
         sized(wl.config0(out=32, ex=20), 75, 75, random_init=200), sized(wl.config0(out=32, ex=20), 90, 51, backtrack_stages=0),
         sized(wl.config0(out=32, ex=20), 80, 80, nearest_neighbors=40)]
    g = wl.config2(out=60, ex=40)
    g["params"].update({"nearest_neighbors": 7, "random_sample_locations": 5})
    i = wl.inpaint_session(5, side=75)
    i["params"].update({"nearest_neighbors": 7, "random_sample_locations": 5})
    return c + [g, i]


@pytest.mark.parametrize("graph", [False, True])
def test_batch(ts, oracle, wl, graph):
    specs = specs_of(wl)
    batch = ts.Batch(graph=graph)
    for s in specs:
        batch.add(ts.builder_from_spec(s).build())
    for q, (g, s) in enumerate(zip(batch.run(), specs)):
        assert_same(ts.generated_outputs(g), oracle.run(s, nthreads=8), "session %d" % q)


def test_served(ts, oracle, wl):
    specs = specs_of(wl)
    server = ts.Server()
    tickets = [server.submit(ts.builder_from_spec(s).build()) for s in specs]
    for q, (t, s) in enumerate(zip(tickets, specs)):
        assert_same(ts.generated_outputs(server.wait(t)[0]), oracle.run(s, nthreads=8), "request %d" % q)


@pytest.mark.parametrize("n", [3, 90])
def test_guided_beside_unguided(ts, wl, n):
    """Steps whose guided and unguided sessions share a launch, and steps of
    more blocks than one launch takes (90 sessions of 64^2)."""
    specs = []
    for q in range(n):
        spec = wl.config2(out=64, ex=24) if q % 2 else wl.config0(out=64, ex=24)
        spec["params"].update({"nearest_neighbors": 4, "random_sample_locations": 2, "seed": q})
        specs.append(spec)
    batch = ts.Batch()
    for s in specs:
        batch.add(ts.builder_from_spec(s).build())
    for q, (g, s) in enumerate(zip(batch.run(), specs)):
        assert_same(ts.generated_outputs(g), ts.run_spec(s), "session %d" % q)
