"""Sums do not depend on timing where rounds are cut short: on a call whose exact
lists reach their limit (which input a round leaves to the next then follows the
warps' timing), and on one that ends in rounds of short budgets, repeated calls
and calls with the exact list on the same stream agree bit for bit."""
import numpy as np
import pytest

from fastlinkingnumbers_b200 import Engine, Model, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("n_loops,n_steps,cube", [(1000, 20_000, 504.0), (60, 4_000, 100.0)])
def test_sums_do_not_depend_on_what_a_round_left_over(n_loops, n_steps, cube):
    engine = Engine(0)
    off, xyz = workloads.polymer(seed=3, n_loops=n_loops, n_steps=n_steps, cube=cube)
    counts = -np.diff(off).astype(np.int32)
    poff, pxyz, pairs, _ = Model().SetCurves(3, counts, xyz).Prepare(True, engine=engine)
    # (The first call sizes the frontier's buffer; pairs without room retry from the roots.)
    engine.linking_numbers(pxyz, poff, pairs, "barneshut", bh_bucket=10)
    runs = [engine.linking_numbers(pxyz, poff, pairs, "barneshut", bh_bucket=10, bh_exact_serial=serial)
            for serial in (0, 1, 0, 1)]
    for lk, err, flags in runs[1:]:
        assert np.array_equal(lk.view(np.uint64), runs[0][0].view(np.uint64))
        assert np.array_equal(err.view(np.uint64), runs[0][1].view(np.uint64))
        np.testing.assert_array_equal(flags, runs[0][2])
