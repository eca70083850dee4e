"""Curve-order tree build at the edges of its blocks and groups: loops of a
few segments, around the 16-segment groups and the 1,024-segment block, and of
several blocks, against the oracle's FP64 restatement of the same trees and
traversal."""
import numpy as np
import pytest

from fastlinkingnumbers_b200 import Engine
from oracle import pyoracle

# 2..17: one group and its shapes, or two; 33, 65, 130: nodes of 16 segments
# beside nodes of 17; 1023..1025: one block or two; the rest: several.
SIZES = [2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17, 31, 32, 33, 34, 65, 130, 257, 511, 513, 1023, 1024, 1025, 2047, 2049, 5000,
         20011]


@pytest.mark.gpu
@pytest.mark.parametrize("bucket", [1, 8])
def test_block_edges_match_oracle(bucket):
    rng = np.random.default_rng(17)
    loops = []
    for n in [700] + SIZES:
        steps = rng.normal(size=(n, 3))
        steps -= steps.mean(axis=0)
        p = np.cumsum(steps, axis=0)
        loops.append((p - p.mean(axis=0)) * 20.0 / np.sqrt(max(n, 16)))
    off = np.concatenate([[0], np.cumsum([len(x) for x in loops])]).astype(np.int64)
    xyz = np.concatenate(loops).astype(np.float32).astype(np.float64)
    pairs = np.array([(0, k + 1) for k in range(len(SIZES))] + [(k, k + 1) for k in range(1, len(SIZES))], dtype=np.int32)
    o = pyoracle.Oracle().set_polylines(off, xyz)
    lk_o, err_o, far_o, ex_o = o.eval_curve_bh(pairs, beta=2.0, bucket=bucket)
    engine = Engine(0)
    lk, err, _ = engine.linking_numbers(xyz, off, pairs, "barneshut", bh_bucket=bucket, target_error=1e30,
                                        bh_escalations=0, fp64_margin=0.0, bh_err_limit=1e30)
    s = engine.stats()
    # FP32 moments, far field and exact terms: 2e-5 on a sum, 1e-3 on an
    # estimate; the node pairs are the same except on the opening boundary.
    np.testing.assert_allclose(lk, lk_o, rtol=0, atol=2e-5)
    np.testing.assert_allclose(err, err_o, rtol=1e-3, atol=1e-9)
    assert abs(s["bh_far_evals"] - float(far_o.sum())) <= 1e-5 * float(far_o.sum()) + 2
    assert abs(s["bh_leaf_evals"] - float(ex_o.sum())) <= 1e-5 * float(ex_o.sum()) + 64
