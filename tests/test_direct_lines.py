"""Direct sums on both sides of the lines where the plan changes the kernel or cuts
curve 2, against the oracle or against whole walks (the allocation-free call)."""
import numpy as np
import pytest

from fastlinkingnumbers_b200 import _native as N
from oracle import pyoracle
from test_direct_speed import Calls, all_pairs, walks

pytestmark = pytest.mark.gpu


# A lone FP64 pair: up to 2 x 148 items of 32 segments for its own kernel, the general one above.
@pytest.mark.parametrize("sizes", [(9472, 321), (9473, 321), (65, 9473), (40000, 33), (40001, 2)])
def test_lone_pair(sizes):
    off, xyz = walks(sizes, 11, 5.0)
    ref, _, _, _ = pyoracle.Oracle().set_polylines(off, xyz).eval_pairs(pyoracle.DIRECT_FAST, all_pairs(2))
    c = Calls(off, xyz, all_pairs(2))
    c.allocating(N.PREC_FP64)
    np.testing.assert_allclose(c.lk.cpu().numpy(), ref, rtol=0, atol=1e-9)
    assert c.engine.stats()["segment_pairs"] == float(sizes[0]) * sizes[1]
    host, _, _ = c.engine.linking_numbers(xyz, off, all_pairs(2), "directsum", precision=N.PREC_FP64)
    assert host[0] == c.lk.cpu().numpy()[0]  # the host knows the sizes there: the same kernel


# Mixed sums are cut along curve 2 from 2^30 segment pairs on: 32,768 x 32,768 is the first.
@pytest.mark.parametrize("sizes", [(32768, 32767), (32768, 32768), (33001, 32999), (200000, 6001)])
def test_large_mixed_sum(sizes):
    c = Calls(*walks(sizes, 13, 20.0), all_pairs(2))
    c.noalloc(N.PREC_MIXED)
    whole = c.lk.cpu().numpy().copy()
    c.allocating(N.PREC_MIXED, fp64_margin=0.0)
    # The same FP32 runs of 32 terms: only the order of the FP64 additions differs.
    np.testing.assert_allclose(c.lk.cpu().numpy(), whole, rtol=0, atol=1e-9)
    c.allocating(N.PREC_FP64)
    np.testing.assert_allclose(c.lk.cpu().numpy(), whole, rtol=0, atol=1e-5)


# Mixed plans with fewer items than CTAs: around the numbers of SMs (148) and of the few-items
# kernel's CTAs (592), by it (curve 2 of 300 segments) and by the packed one (30).
@pytest.mark.parametrize("other", [30, 300])
@pytest.mark.parametrize("items", [1, 2, 147, 148, 149, 296, 591, 592, 593, 1183, 1184, 1185])
def test_few_items(items, other):
    c = Calls(*walks((128 * items - 5, other), items, 5.0), all_pairs(2))
    c.noalloc(N.PREC_MIXED)  # a grid of as many CTAs as items
    ref = c.lk.cpu().numpy().copy()
    for _ in range(3):
        c.lk.fill_(7.0)
        c.torch.cuda.synchronize()
        c.allocating(N.PREC_MIXED, fp64_margin=-1.0)
        assert c.lk.cpu().numpy()[0] == ref[0]
    c.allocating(N.PREC_FP64)
    np.testing.assert_allclose(c.lk.cpu().numpy(), ref, rtol=0, atol=1e-5)
