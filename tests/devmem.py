"""Device memory of the tests' process through the driver API: the default
stream-ordered pool's counters, and a fill that leaves a given amount free."""
import ctypes as C

RESERVED_CURRENT, USED_CURRENT, USED_HIGH = 5, 7, 8  # CUmemPool_attribute


def _check(rc):
    assert rc == 0, "CUDA driver status %d" % rc


class DevMem:
    def __init__(self, device=0):
        self.cu = C.CDLL("libcuda.so.1")
        _check(self.cu.cuInit(0))
        dev, ctx, self.pool = C.c_int(), C.c_void_p(), C.c_void_p()
        _check(self.cu.cuDeviceGet(C.byref(dev), device))
        _check(self.cu.cuDevicePrimaryCtxRetain(C.byref(ctx), dev))
        _check(self.cu.cuCtxSetCurrent(ctx))
        _check(self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), dev))

    def trim(self):
        """Gives the pool's idle memory back to the device."""
        _check(self.cu.cuCtxSynchronize())
        _check(self.cu.cuMemPoolTrimTo(self.pool, C.c_size_t(0)))

    def pool_bytes(self, attr):
        v = C.c_uint64()
        _check(self.cu.cuMemPoolGetAttribute(self.pool, attr, C.byref(v)))
        return v.value

    def peak_of(self, run):
        """(run's result, most pool bytes in use at once during it)."""
        zero = C.c_uint64(0)
        _check(self.cu.cuMemPoolSetAttribute(self.pool, USED_HIGH, C.byref(zero)))
        got = run()
        return got, self.pool_bytes(USED_HIGH)

    def free_bytes(self):
        free, total = C.c_size_t(), C.c_size_t()
        _check(self.cu.cuMemGetInfo_v2(C.byref(free), C.byref(total)))
        return free.value

    def leaving(self, keep, run):
        """run() with all but `keep` bytes of the device taken."""
        self.trim()
        p = C.c_uint64()
        _check(self.cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(self.free_bytes() - keep)))
        try:
            return run()
        finally:
            _check(self.cu.cuMemFree_v2(p))
