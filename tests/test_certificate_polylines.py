"""The polylines of a certificate computed on the GPU come to the model beside the
sums, on a stream and a thread of their own: they are those of Prepare, for small
and large models, and also when the sums fail."""
import ctypes as C

import numpy as np
import pytest

from fastlinkingnumbers_b200 import Engine, FlnError, LinkingNumberCertificate, Model, workloads
from fastlinkingnumbers_b200 import _native as N

pytestmark = pytest.mark.gpu


def prepared(model):
    """The polylines a model holds: (offsets, vertices, pairs)."""
    L = N.load()
    nv, np_ = C.c_int64(), C.c_int64()
    N.check(L.fln_model_prepared_sizes(model.handle, C.byref(nv), C.byref(np_)))
    off = np.empty(model.num_curves() + 1, dtype=np.int64)
    xyz, pairs = np.empty((nv.value, 3)), np.empty((np_.value, 2), dtype=np.int32)
    N.check(L.fln_model_get_prepared(model.handle, off.ctypes.data_as(C.c_void_p), xyz.ctypes.data_as(C.c_void_p),
                                     pairs.ctypes.data_as(C.c_void_p)))
    return off, xyz, pairs


# 20 x 400 points go in one copy; 60 x 20,000 (above 16 MB) in pieces through pinned buffers.
@pytest.mark.parametrize("loops,steps,cube", [(20, 400, 12.0), (60, 20000, 200.0)])
@pytest.mark.parametrize("fail", [False, True])
def test_polylines_after_a_certificate(loops, steps, cube, fail):
    eng = Engine(0)
    off, xyz = workloads.polymer(seed=17, n_loops=loops, n_steps=steps, cube=cube)
    counts = -np.diff(off).astype(np.int32)
    want = Model().SetCurves(3, counts, xyz).Prepare(True, engine=eng)
    assert steps < 20000 or want[1].nbytes > 16 << 20
    m = Model().SetCurves(3, counts, xyz)
    if fail:
        with pytest.raises(FlnError, match="stack"):  # the traversal's bound, lowered
            LinkingNumberCertificate().ComputeFromModel(m, engine=eng, bh_spill_cap=1, barnes_hut_init_beta=9.0)
    else:
        LinkingNumberCertificate().ComputeFromModel(m, engine=eng)
    for got, ref in zip(prepared(m), want[:3]):
        assert np.array_equal(got, ref)
    # The next certificate starts from them.
    a = LinkingNumberCertificate().ComputeFromModel(m, engine=eng).text()
    assert a == LinkingNumberCertificate().ComputeFromModel(Model().SetCurves(3, counts, xyz), engine=eng).text()
