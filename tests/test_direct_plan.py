"""The direct sum's device plan: items along both loops, calls of few and of many
pairs, a plan that outgrows its room, and bad input, against the oracle."""
import numpy as np
import pytest

from fastlinkingnumbers_b200 import Engine, FlnError
from fastlinkingnumbers_b200 import _native as N
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _loops(sizes, seed, scale=3.0):
    rng = np.random.default_rng(seed)
    out = []
    for n in sizes:
        s = rng.normal(size=(n, 3))
        s -= s.mean(axis=0)
        p = np.cumsum(s, axis=0)
        out.append((p - p.mean(axis=0)) * scale / np.sqrt(max(n, 8)) + rng.normal(size=3) * 0.3)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    return off, np.concatenate(out).astype(np.float32).astype(np.float64)


def _all_pairs(n):
    i, j = np.triu_indices(n, 1)
    return np.stack([i, j], axis=1).astype(np.int32)


# Sizes around the block (64, 128, 256 segments), the 32-segment runs and spans
# and the 256-vertex tile, both ways round.
CASES = {
    "one small pair": ([33, 31], [(0, 1)]),
    "edges": ([2, 3, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 513, 1000], None),
    "long against short": ([20011, 3, 40, 300], None),
    "long pair": ([7001, 6007], [(1, 0)]),
    # A lone pair's tiles of 42 steps (four to a staged stretch) and items of 32 segments.
    "lone 2 x 2": ([2, 2], [(0, 1)]),
    "lone 43 x 42": ([43, 42], [(0, 1)]),
    "lone 129 x 41": ([41, 129], [(0, 1)]),
    "lone 337 x 169": ([337, 169], [(0, 1)]),
    "more items than room": ([20000] + [3] * 130, [(k + 1, 0) for k in range(130)]),
    "many pairs": (list(range(2, 72)), None),
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("prec,tol", [(N.PREC_FP64, 1e-9), (N.PREC_MIXED, 1e-5)])
def test_plan_matches_oracle(name, prec, tol):
    sizes, pairs = CASES[name]
    off, xyz = _loops(sizes, 5)
    pairs = _all_pairs(len(sizes)) if pairs is None else np.array(pairs, dtype=np.int32)
    ref, _, _, _ = pyoracle.Oracle().set_polylines(off, xyz).eval_pairs(pyoracle.DIRECT_FAST, pairs)
    eng = Engine(0)  # a new engine: no room left by other calls
    for tile in range(6):
        lk, err, flags = eng.linking_numbers(xyz, off, pairs, "directsum", precision=prec, direct_tile=tile,
                                             fp64_margin=0.0)
        np.testing.assert_allclose(lk, ref, rtol=0, atol=tol)
        assert not err.any() and not flags.any()
    s = eng.stats()
    n = np.diff(off)
    assert s["segment_pairs"] == float((n[pairs[:, 0]] * n[pairs[:, 1]]).sum()) and s["pairs"] == len(pairs)
    # The margin check on the device: every pair below an impossible margin.
    lk, _, flags = eng.linking_numbers(xyz, off, pairs, "directsum", precision=prec, fp64_margin=0.75)
    np.testing.assert_allclose(lk, ref, rtol=0, atol=1e-9)
    want = N.PAIR_FP64_RECOMPUTED if prec == N.PREC_MIXED else 0
    assert (flags == want).all() and eng.stats()["fp64_recomputed"] == (len(pairs) if want else 0)


@pytest.mark.parametrize("npairs", [3, 5000])
def test_bad_device_input_is_refused(npairs):
    torch = pytest.importorskip("torch")
    off, xyz = _loops([12, 9, 1, 20], 7)
    eng = Engine(0)
    d_xyz = torch.from_numpy(xyz).cuda()
    good = np.tile(np.array([[0, 1]], dtype=np.int32), (npairs, 1))
    for word, bad_pair, bad_off in (("out of range", (0, 4), None), ("out of range", (-1, 1), None),
                                    ("two vertices", (0, 2), None), ("different", (3, 3), None),
                                    ("start at 0", None, [1, 12, 21, 22, 42]),
                                    ("non-decreasing", None, [0, 12, 21, 20, 42])):
        pairs = good.copy()
        if bad_pair:
            pairs[npairs // 2] = bad_pair
        o = torch.tensor(off.tolist() if bad_off is None else bad_off, dtype=torch.int64, device="cuda")
        d_pairs = torch.from_numpy(pairs).cuda()
        lk = torch.full((npairs,), 7.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        with pytest.raises(FlnError) as e:
            eng.linking_numbers_device(d_xyz.data_ptr(), o.data_ptr(), 4, d_pairs.data_ptr(), npairs, lk.data_ptr(),
                                       method="directsum")
        assert e.value.status == 1 and word in str(e.value)
        torch.cuda.synchronize()
        assert bool((lk == 7.0).all())
