"""The warp resolve form where its parts can go wrong, against the oracle:
repeats found with 32-bit keys (up to 16 maps) and with 64-bit keys, neighbour
counts around a warp's rounds, distances of equal and unequal power-of-two
sides, and steps with fewer blocks than item counters."""
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ex,k,m,w,h", [(1, 1, 1, 16, 16), (16, 33, 9, 64, 16), (17, 32, 33, 32, 32),
                                          (3, 64, 65, 37, 21), (2, 65, 20, 32, 64)])
def test_warp_form(ts, oracle, wl, n_ex, k, m, w, h):
    spec = wl.config1(out=32, ex=20)
    spec["out_w"], spec["out_h"] = w, h
    spec["examples"] = [{"image": wl.texture(300 + i, 9 + i % 5, 12 + i % 3)} for i in range(n_ex)]
    spec["params"].update(nearest_neighbors=k, random_sample_locations=m, random_init=3)
    got = ts.run_spec(spec, team_max_batch=0, team_full_max_batch=0)
    assert_same(got, oracle.run(spec, nthreads=4), "warp form %d maps k %d m %d %dx%d" % (n_ex, k, m, w, h))


@pytest.mark.parametrize("k", [32, 33])
def test_default_forms(ts, oracle, wl, k):
    """Steps of 1024 to 2048 items with the thresholds left alone, on both
    sides of the neighbour count from which they take the warp form."""
    spec = wl.config0(out=128, ex=24)
    spec["params"].update(nearest_neighbors=k, random_sample_locations=3)
    ref = oracle.run(spec, nthreads=8)
    assert_same(ts.run_spec(spec), ref, "k = %d" % k)
    assert_same(ts.run_spec(spec, team_max_batch=2048), ref, "k = %d, thresholds set" % k)


@pytest.mark.parametrize("k", [9, 10, 11, 15, 16, 17, 21])
def test_guided_chunks(ts, oracle, wl, k):
    """Neighbour counts around the guided loop's chunks (4, then six at a time)."""
    spec = wl.config2(out=48, ex=40)
    spec["params"].update(nearest_neighbors=k, random_sample_locations=12)
    assert_same(ts.run_spec(spec, team_max_batch=0, team_full_max_batch=0), oracle.run(spec, nthreads=8), "k = %d" % k)
