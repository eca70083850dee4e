"""The node-pair walk of Discretize hands its stacks on sooner when a launch has
few batches. The marks are flags, so neither the pieces nor the round count may
depend on it: a single curve pair, and counts of overlapping curve pairs on both
sides of the line (four batches per resident warp), against the host path bit
for bit."""
import numpy as np
import pytest

from fastlinkingnumbers_b200 import Engine, Model, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("n_loops,n_steps", [(2, 30_000), (150, 400), (240, 400)])
def test_refinement_does_not_depend_on_the_budget(n_loops, n_steps):
    off, xyz = workloads.polymer(seed=17, n_loops=n_loops, n_steps=n_steps, cube=20.0)
    counts = -np.diff(off).astype(np.int32)
    off_h, xyz_h, pairs_h, rounds_h = Model().SetCurves(3, counts, xyz).Prepare(True)
    off_d, xyz_d, pairs_d, rounds_d = Model().SetCurves(3, counts, xyz).Prepare(True, engine=Engine(0))
    assert rounds_d == rounds_h and len(pairs_h) > 0.9 * n_loops * (n_loops - 1) / 2
    assert np.array_equal(off_d, off_h) and np.array_equal(pairs_d, pairs_h)
    assert np.array_equal(xyz_d.view(np.uint64), xyz_h.view(np.uint64))
