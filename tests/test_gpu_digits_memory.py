"""Device memory of the fixed-point digits (the FP64 and tier 3 kernels' inputs): held for one apply, not for a
call of the library that runs many."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

USED_HIGH = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH


class Pool:
    """The device's default memory pool (driver API: the library's context is the device's primary one)."""

    def __init__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.pool = ctypes.c_void_p()
        dev = ctypes.c_int()
        assert self.cu.cuInit(0) == 0 and self.cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), dev) == 0

    def most(self, f):
        """The most that was in use at once during f()."""
        v = ctypes.c_uint64(0)  # sets the high-water mark back to what is in use now
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_HIGH, ctypes.byref(v)) == 0
        f()
        assert self.cu.cuMemPoolGetAttribute(self.pool, USED_HIGH, ctypes.byref(v)) == 0
        return v.value


def batch(engine, order, n, prec):
    mra = engine.MultiResolutionAnalysis(order)
    fs = [engine.project(prec, engine.FunctionTree(mra), [(1.0, 2.0 + i, (0.1 * i, -0.2, 0.3), (0, 0, 0))])
          for i in range(n)]
    Hs = [engine.HelmholtzOperator(mra, 0.5 + 0.1 * i, prec) for i in range(n)]
    return mra, fs, Hs, [engine.FunctionTree(mra) for _ in fs]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_autotuner_holds_the_digits_of_one_apply(engine, precision):
    n, prec = 3, 1e-4
    mra, fs, Hs, outs = batch(engine, 5, n, prec)
    pool = Pool()
    # grows the outputs' trees to their final size first: what is left is the apply's own memory
    engine.apply_batch([prec] * n, outs, Hs, fs, precision=precision)

    def one():
        for o in outs:
            o.clear()
        engine.apply_batch([prec] * n, outs, Hs, fs, precision=precision)

    single = pool.most(one)
    tuned = pool.most(lambda: engine.autotune_batch([prec] * n, outs, Hs, fs, precision=precision, repeats=2))
    # the digits' 1.8 times the inputs of some 40 applies, were they held, against the same for one
    assert tuned <= 1.25 * single, (tuned, single)
