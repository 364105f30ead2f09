"""Initial state of inpainting runs, against the oracle: rows of less than,
exactly and more than a mask word, masks that leave everything, nothing or
every other pixel to synthesise, random init on top, tiling mirrors; the plain
and the served form."""
import numpy as np
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def spec_of(wl, side, mask, tiling, init):
    spec = wl.inpaint_session(21, side=side)
    m = np.full((side, side, 4), 255, np.uint8)
    open_px = {"all": np.ones((side, side), bool), "none": np.zeros((side, side), bool),
               "checker": np.indices((side, side)).sum(0) % 2 == 0}[mask]
    m[open_px, :3] = 0
    spec["inpaint_mask"] = m
    spec["params"].update({"nearest_neighbors": 6, "random_sample_locations": 4, "tiling_mode": tiling,
                           "random_init": init})
    return spec


CASES = [(17, "all", False, None), (31, "checker", True, None), (32, "checker", False, 7), (33, "checker", True, 3),
         (33, "all", True, 20), (40, "none", False, None), (65, "checker", True, 64)]


@pytest.mark.parametrize("side,mask,tiling,init", CASES)
def test_inpaint_init(ts, oracle, wl, side, mask, tiling, init):
    spec = spec_of(wl, side, mask, tiling, init)
    assert_same(ts.run_spec(spec), oracle.run(spec, nthreads=8), "%d %s" % (side, mask))


def test_served(ts, oracle, wl):
    server = ts.Server()
    specs = [spec_of(wl, *c) for c in CASES]
    tickets = [server.submit(ts.builder_from_spec(s).build()) for s in specs]
    for t, s in zip(tickets, specs):
        assert_same(ts.generated_outputs(server.wait(t)[0]), oracle.run(s, nthreads=8), "served")
