"""The mixed direct sum of few items runs one segment per thread, that of many two
packed ones: the same pairs, alone and repeated often enough to change the kernel,
have the same sums bit for bit."""
import numpy as np
import pytest

from fastlinkingnumbers_b200 import Engine, Model, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("n_loops,n_steps,repeat", [(2, 129, 900), (4, 257, 200), (5, 998, 20), (7, 1500, 6)])
def test_few_items_sum_as_many(n_loops, n_steps, repeat):
    engine = Engine(0)
    off, xyz = workloads.polymer(seed=29, n_loops=n_loops, n_steps=n_steps, cube=10.0)
    poff, pxyz, pairs, _ = Model().SetCurves(3, -np.diff(off).astype(np.int32), xyz).Prepare(True, engine=engine)
    assert len(pairs) > 0
    lk, _, _ = engine.linking_numbers(pxyz, poff, pairs, "directsum", precision=1, fp64_margin=-1.0)
    many, _, _ = engine.linking_numbers(pxyz, poff, np.tile(pairs, (repeat, 1)), "directsum", precision=1, fp64_margin=-1.0)
    assert np.array_equal(many.reshape(repeat, -1).view(np.uint64), np.tile(lk.view(np.uint64), (repeat, 1)))
