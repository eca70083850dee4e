"""Which kernel a direct sum runs, seen from its time: each call against another of
the same sums, so that the device's clock drops out. The bounds lie halfway between
the ratio with the right kernel and with the wrong one."""
import ctypes as C
import time

import numpy as np
import pytest

from fastlinkingnumbers_b200 import Engine
from fastlinkingnumbers_b200 import _native as N

pytestmark = pytest.mark.gpu


def walks(sizes, seed, spread):
    """Closed Gaussian walks about centres in a cube of side `spread`."""
    rng = np.random.default_rng(seed)
    out = []
    for n in sizes:
        s = rng.normal(size=(n, 3))
        p = np.cumsum(s - s.mean(axis=0), axis=0)
        out.append(p - p.mean(axis=0) + spread * rng.uniform(size=3))
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64), np.concatenate(out)


def all_pairs(n):
    return np.stack(np.triu_indices(n, 1), axis=1).astype(np.int32)


class Calls:
    """Device-array calls of one set of loops and pairs; time() is the best of many."""

    def __init__(self, off, xyz, pairs):
        import torch
        self.torch, self.engine, self.lib = torch, Engine(0), N.load()
        self.n, self.nloops = len(pairs), len(off) - 1
        self.d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (xyz, off, pairs)]
        self.lk = torch.zeros(self.n, dtype=torch.float64, device="cuda")

    def allocating(self, precision, **params):
        self.engine.linking_numbers_device(self.d[0].data_ptr(), self.d[1].data_ptr(), self.nloops,
                                           self.d[2].data_ptr(), self.n, self.lk.data_ptr(), method="directsum",
                                           precision=precision, **params)

    def noalloc(self, precision):
        st = self.lib.fln_linking_numbers_direct_noalloc(
            C.c_void_p(self.d[0].data_ptr()), C.c_void_p(self.d[1].data_ptr()), self.nloops,
            C.c_void_p(self.d[2].data_ptr()), self.n, precision, C.c_void_p(self.lk.data_ptr()), None)
        assert st == 0, self.lib.fln_last_error()

    def time(self, call, *args, **params):
        best = 1e9
        for _ in range(25):
            self.torch.cuda.synchronize()
            t = time.perf_counter()
            call(*args, **params)
            self.torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best


@pytest.mark.parametrize("loops,steps", [(5, 998), (8, 2000)])
def test_allocation_free_call_of_few_items(loops, steps):
    """The allocation-free mixed call runs the kernel of few items as the allocating one does (times
    of 0.95 of its; with the kernel of many 2.4 and 1.4)."""
    c = Calls(*walks([steps] * loops, 3, 10.0), all_pairs(loops))
    assert c.time(c.noalloc, N.PREC_MIXED) < 1.2 * c.time(c.allocating, N.PREC_MIXED)


@pytest.mark.parametrize("loops,steps,most", [(10, 60, 2.6), (20, 100, 4.4), (20, 130, 4.8), (100, 60, 3.4)])
def test_mixed_sum_of_near_loops(loops, steps, most):
    """Loops on one spot, nearly all segment pairs near ones: the mixed sum evaluates them in FP64
    about as fast as lanes can (2.0, 2.1, 2.3 and 2.4 times the FP64 sum; it was 3.2, 6.8, 7.0
    and 4.3 when a warp looked for every pair's owner in turn)."""
    c = Calls(*walks([steps] * loops, 5, 1.0), all_pairs(loops))
    assert c.time(c.allocating, N.PREC_MIXED) < most * c.time(c.allocating, N.PREC_FP64)


@pytest.mark.parametrize("sizes", [(200000, 20), (200000, 300), (10000, 8572)])
def test_long_lone_pair(sizes):
    """A lone FP64 pair with a long loop runs the general kernel: the times of another tile shape,
    which always does (with the lone pairs' kernel 2.8, 1.8 and 2.3 times as long)."""
    c = Calls(*walks(sizes, 7, 5.0), all_pairs(2))
    general = c.time(c.allocating, N.PREC_FP64, direct_tile=1)
    assert c.time(c.allocating, N.PREC_FP64) < 1.4 * general


def test_few_items_are_spread_over_the_chip():
    """120 items on device arrays, where the grid does not know their number, against a grid of 120
    CTAs (1.05 times its time; 1.6 when the items met on some SMs)."""
    c = Calls(*walks([5000] * 3, 9, 200.0), all_pairs(3))
    assert c.time(c.allocating, N.PREC_MIXED) < 1.3 * c.time(c.noalloc, N.PREC_MIXED)
