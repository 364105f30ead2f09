"""Device memory that runs take and keep, from the driver's counters of the
default stream-ordered pool."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RESERVED_CURRENT, USED_CURRENT, USED_HIGH = 5, 7, 8  # CUmemPool_attribute


class DevMem:
    def __init__(self):
        self.cu = C.CDLL("libcuda.so.1")
        dev, ctx, self.pool = C.c_int(), C.c_void_p(), C.c_void_p()
        self._check(self.cu.cuInit(0))
        self._check(self.cu.cuDeviceGet(C.byref(dev), 0))
        self._check(self.cu.cuDevicePrimaryCtxRetain(C.byref(ctx), dev))
        self._check(self.cu.cuCtxSetCurrent(ctx))
        self._check(self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), dev))

    @staticmethod
    def _check(rc):
        assert rc == 0, "CUDA driver status %d" % rc

    def pool_bytes(self, attr):
        v = C.c_uint64()
        self._check(self.cu.cuMemPoolGetAttribute(self.pool, attr, C.byref(v)))
        return v.value

    def peak(self, run):
        """Most pool bytes that run() adds to those in use."""
        self._check(self.cu.cuCtxSynchronize())
        zero = C.c_uint64(0)
        self._check(self.cu.cuMemPoolSetAttribute(self.pool, USED_HIGH, C.byref(zero)))
        before = self.pool_bytes(USED_CURRENT)
        run()
        return self.pool_bytes(USED_HIGH) - before

    def leaving(self, keep, run):
        """run() with all but `keep` bytes of the device taken."""
        self._check(self.cu.cuCtxSynchronize())
        self._check(self.cu.cuMemPoolTrimTo(self.pool, C.c_size_t(0)))
        free, total, p = C.c_size_t(), C.c_size_t(), C.c_uint64()
        self._check(self.cu.cuMemGetInfo_v2(C.byref(free), C.byref(total)))
        self._check(self.cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(free.value - keep)))
        try:
            return run()
        finally:
            self._check(self.cu.cuMemFree_v2(p))


@pytest.fixture(scope="module")
def mem():
    return DevMem()


def test_sequential_schedule(ts, wl, mem):
    """One item a step: what the run holds more than one of larger steps is a
    few words a step (a fallback counter, the table of the steps' trees), not
    the warp resolve's 512 bytes of counters, which such steps never read."""
    spec = wl.config0(out=64, ex=16)
    spec["params"].update(nearest_neighbors=4, random_sample_locations=2)
    stats = {}

    def run(divisor):
        stats[divisor] = ts.run_spec(spec, batch_divisor=divisor)["stats"]

    run(8)
    few, many = mem.peak(lambda: run(8)), mem.peak(lambda: run(0))
    steps = stats[0]["batches"] - stats[8]["batches"]
    assert steps > 4096
    assert many - few <= 64 * steps, (few, many, steps)


def test_lists_ahead_leave_room(ts, wl, mem):
    """4.1 GB of neighbour lists with 4 GB of the device free: the run, which
    needs a quarter of that without them, makes them per step instead."""
    spec = wl.config0(out=64, ex=64)
    spec["out_w"], spec["out_h"] = 2000, 1001
    spec["params"].update(nearest_neighbors=256, random_sample_locations=1)
    tight = mem.leaving(4 << 30, lambda: ts.run_spec(spec))
    assert tight["stats"]["knn_chunks"] == 0
    free = ts.run_spec(spec)
    assert free["stats"]["knn_chunks"] > 0
    for key in ("image", "coord", "id", "resolved", "scores"):
        assert np.array_equal(tight[key], free[key]), key


def test_served_requests_share_a_tight_budget(ts, wl):
    """Four equal requests under a budget of four of them run side by side:
    what could be made ahead does not take the next ones' room."""
    spec = wl.config0(out=512, ex=64)
    with ts.Server(hbm_budget=1, max_active=4) as srv:  # alone, nothing made ahead
        alone = srv.wait(srv.submit(ts.builder_from_spec(spec).build()))[0].into_image()
        one = srv.stats()["peak_bytes"]
    sessions = [ts.builder_from_spec(spec).build() for _ in range(4)]
    with ts.Server(hbm_budget=4 * one, max_active=4) as srv:
        tickets = [srv.submit(s) for s in sessions]
        images = [srv.wait(t)[0].into_image() for t in tickets]
        stats = srv.stats()
    assert stats["peak_active"] == 4, stats
    assert stats["peak_bytes"] <= 4 * one
    assert all(np.array_equal(im, alone) for im in images)


def test_pool_is_given_back(ts, wl, mem):
    """A run of some 18 GB of buffers leaves at most 16 GiB in the pool."""
    spec = wl.config0(out=2048, ex=64)
    spec["params"].update(nearest_neighbors=256, random_sample_locations=129)
    assert mem.peak(lambda: ts.run_spec(spec)) > 16 << 30
    assert mem.pool_bytes(RESERVED_CURRENT) <= 16 << 30
