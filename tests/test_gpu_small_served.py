"""Bursts of small requests, served and batched: the time of a burst against
one request's, and the results against the oracle where a run's picks are one
launch (few items, up to eight stages) and around that limit."""
import time

import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def _inpaint(wl, side, k, m, seed, stages=5, init=None):
    spec = wl.inpaint_session(seed, side=side)
    spec["params"].update(nearest_neighbors=k, random_sample_locations=m, backtrack_stages=stages, random_init=init)
    return spec


def test_candidates_side_by_side(ts, wl):
    """Sixteen requests whose candidates are long chains of draws (m = 200):
    side by side they take a few times one's time (on one stream after another
    fourteen times)."""
    sp = [_inpaint(wl, 64, 50, 200, 20 + i) for i in range(16)]
    ms = {}
    with ts.Server() as server:
        for n in (1, 16):
            v = []
            for _ in range(7):
                sessions = [ts.builder_from_spec(s).build() for s in sp[:n]]
                t0 = time.perf_counter()
                for t in [server.submit(s) for s in sessions]:
                    server.wait(t)
                v.append(time.perf_counter() - t0)
            ms[n] = sorted(v)[3] * 1e3
    assert ms[16] <= 7 * ms[1], ms


def _synth(wl, w, h, k, m, stages=5, init=None):
    spec = wl.config0(out=16, ex=16)
    spec["out_w"], spec["out_h"] = w, h
    spec["params"].update(nearest_neighbors=k, random_sample_locations=m, backtrack_stages=stages, random_init=init)
    return spec


def specs(wl):
    return [_inpaint(wl, 33, 8, 5, 3), _inpaint(wl, 48, 20, 9, 4, stages=7), _inpaint(wl, 40, 6, 4, 5, stages=9),
            _inpaint(wl, 40, 6, 4, 6, init=17), _synth(wl, 45, 40, 7, 5), _synth(wl, 40, 45, 0, 3),
            _synth(wl, 32, 32, 9, 4, init=30), _synth(wl, 46, 45, 7, 5, stages=7), _synth(wl, 47, 45, 7, 5),
            _synth(wl, 1, 1, 3, 2), _synth(wl, 16, 8, 5, 3, stages=0, init=100)]


def test_served_burst(ts, oracle, wl):
    server = ts.Server()
    sp = specs(wl) * 2
    sessions = [ts.builder_from_spec(s).build() for s in sp]
    tickets = [server.submit(s) for s in sessions]
    got = [ts.generated_outputs(server.wait(t)[0]) for t in tickets]
    for i, s in enumerate(sp):
        assert_same(got[i], oracle.run(s, nthreads=8), "served %d" % i)


@pytest.mark.parametrize("graph", [False, True])
def test_batch(ts, oracle, wl, graph):
    sp = specs(wl)
    batch = ts.Batch(graph=graph)
    for s in sp:
        batch.add(ts.builder_from_spec(s).build())
    for i, g in enumerate(batch.run()):
        assert_same(ts.generated_outputs(g), oracle.run(sp[i], nthreads=8), "batched %d" % i)
