"""Direct sums of curves whose coordinates are very large or very small.

Linking numbers do not depend on the unit of length: a Hopf link has the same
one at every scale at which a segment pair's term (a product of six
differences of coordinates) is a number of the arithmetic that forms it.
"""
import ctypes as C

import numpy as np
import pytest

from fastlinkingnumbers_b200 import Engine
from fastlinkingnumbers_b200 import _native as N

pytestmark = pytest.mark.gpu


def hopf(n, m, scale):
    """Two rings of radius `scale`, linked once (linking number -1), with n and m vertices."""
    a, b = 2 * np.pi * np.arange(n) / n, 2 * np.pi * np.arange(m) / m
    first = np.stack([np.cos(a), np.sin(a), 0 * a], axis=1)
    second = np.stack([1 + np.cos(b), 0 * b, np.sin(b)], axis=1)
    return np.array([0, n, n + m], dtype=np.int64), np.concatenate([first, second]) * scale


def sums(off, xyz, npairs, precision):
    """The sums of `npairs` times the pair (0, 1) by the allocating and the allocation-free call."""
    import torch
    d_xyz, d_off = torch.from_numpy(xyz).cuda(), torch.from_numpy(off).cuda()
    d_pairs = torch.tensor([[0, 1]] * npairs, dtype=torch.int32, device="cuda")
    out = torch.zeros(2, npairs, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    Engine(0).linking_numbers_device(d_xyz.data_ptr(), d_off.data_ptr(), 2, d_pairs.data_ptr(), npairs,
                                     out[0].data_ptr(), method="directsum", precision=precision)
    L = N.load()
    st = L.fln_linking_numbers_direct_noalloc(C.c_void_p(d_xyz.data_ptr()), C.c_void_p(d_off.data_ptr()), 2,
                                              C.c_void_p(d_pairs.data_ptr()), npairs, precision,
                                              C.c_void_p(out[1].data_ptr()), None)
    assert st == 0, L.fln_last_error()
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("sizes", [(7, 9), (64, 60), (129, 301)])
@pytest.mark.parametrize("scale", [1e-50, 1e-45, 1e-30, 1e-25, 1e-23, 1e-21, 1.0, 1e22, 1e24, 1e26, 1e30, 1e45, 1e50])
def test_fp64_sums_at_every_scale(sizes, scale):
    off, xyz = hopf(*sizes, scale)
    for npairs in (1, 3):  # the lone pair's kernel and the batched one
        # A term's rounding is a few 1e-16 and the 40,000 terms add up to one turn: below 1e-11 in all.
        np.testing.assert_allclose(sums(off, xyz, npairs, N.PREC_FP64), -1.0, rtol=0, atol=1e-11)


@pytest.mark.parametrize("sizes", [(64, 60), (300, 200)])  # two segments per thread, and one
@pytest.mark.parametrize("scale", [1e-17, 1e-12, 1e-9, 1e-8, 1e-7, 3e-7, 1e-6, 3e-6, 1e-5, 3e-5, 1e-4, 1e5])
def test_mixed_sums_at_small_scales(sizes, scale):
    """Terms of 64 d^6 that are subnormal in FP32, or 0, or small enough that their parts are."""
    off, xyz = hopf(*sizes, scale)
    np.testing.assert_allclose(sums(off, xyz, 3, N.PREC_MIXED), -1.0, rtol=0, atol=1e-5)
