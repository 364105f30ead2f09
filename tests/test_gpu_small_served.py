"""Bursts of small requests, served: the time of a burst against one
request's."""
import time

import pytest

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
