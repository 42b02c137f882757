"""A handle's calls on a device without spare memory: once the handle exists,
its uploads, evaluations and results need none, and give the same bits.

The device's current memory pool, from which a call's staging memory would
come, is replaced by one of bounded size that is full."""
import ctypes as C

import numpy as np
import pytest

from rich_problems import rich_problem
from texo_gb300 import abi
from texo_gb300.placer import Placer, default_params

pytestmark = pytest.mark.gpu


class Location(C.Structure):
    _fields_ = [("type", C.c_int), ("id", C.c_int)]


class PoolProps(C.Structure):
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("location", Location), ("security", C.c_void_p),
                ("max_size", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


class FullPool:
    """Makes a pool of 2 MiB, filled, the device's current one."""

    def __enter__(self):
        self.cuda = C.CDLL("libcuda.so.1")
        self.pool, self.before, self.taken = C.c_void_p(), C.c_void_p(), []
        props = PoolProps(alloc_type=1, location=Location(1, 0), max_size=2 << 20)
        assert self.cuda.cuDeviceGetMemPool(C.byref(self.before), 0) == 0
        assert self.cuda.cuMemPoolCreate(C.byref(self.pool), C.byref(props)) == 0
        full = False
        for size in (1 << 20, 1 << 9):   # the least block that a pool gives out is 512 bytes
            for _ in range(4096):
                p = C.c_uint64()
                full = self.cuda.cuMemAllocFromPoolAsync(C.byref(p), C.c_size_t(size), self.pool, None) != 0
                if full:
                    break
                self.taken.append(p)
        assert full
        assert self.cuda.cuDeviceSetMemPool(0, self.pool) == 0
        return self

    def __exit__(self, *a):
        assert self.cuda.cuDeviceSetMemPool(0, self.before) == 0
        for p in self.taken:
            assert self.cuda.cuMemFreeAsync(p, None) == 0
        assert self.cuda.cuStreamSynchronize(None) == 0
        assert self.cuda.cuMemPoolDestroy(self.pool) == 0


def calls(g):
    c, _, _ = g.initial()
    e = g.evaluate(c, 4.0)
    part = g.evaluate(c, 4.0, arrays=False)
    t, x, _ = g.run(3, allow_nonconverged=True)
    g.reset()
    phys, fill = g.scatter(x)
    return [e["wirelength"], part["wirelength"], e["wa_gradient"], e["field_gradient"], e["density"], e["potential"], t, x,
            phys, fill, np.array(g.hpwl(x))]


@pytest.mark.parametrize("engine", [abi.ENGINE_HOST, abi.ENGINE_DEVICE])
@pytest.mark.parametrize("fields", [1, 2])
def test_calls_without_spare_memory_give_the_same(engine, fields):
    prob = rich_problem(fields=fields)
    with Placer(prob, default_params(engine=engine, best_effort=1, max_iterations=20)) as g:
        spare = calls(g)
        g.reset()
        with FullPool():
            none = calls(g)
    assert all(np.array_equal(a, b) for a, b in zip(spare, none))
