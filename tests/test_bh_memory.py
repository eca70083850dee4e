"""Device memory of a Barnes-Hut call on a GPU that other programs use as well."""
import numpy as np
import pytest

from fastlinkingnumbers_b200 import Engine, Model, workloads

pytestmark = pytest.mark.gpu


def test_first_frontier_takes_a_fifth_of_the_free_memory():
    torch = pytest.importorskip("torch")
    off, xyz = workloads.polymer(seed=31, n_loops=30, n_steps=60000, cube=150.0)
    maker = Engine(0)
    poff, pxyz, pairs, _ = Model().SetCurves(3, -np.diff(off).astype(np.int32), xyz).Prepare(True, engine=maker)
    maker.close()
    torch.cuda.empty_cache()
    room = 40 << 30
    taken = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
    held = {}
    for roots in (1, 0):  # without the frontier's buffer, and with it
        eng = Engine(0)
        free = torch.cuda.mem_get_info()[0]
        eng.linking_numbers(pxyz, poff, pairs, "barneshut", bh_retry_from_roots=roots)
        held[roots] = free - torch.cuda.mem_get_info()[0]
        eng.close()
    del taken
    torch.cuda.empty_cache()
    # A buffer is allocated with an eighth, 256 MB at most, to spare.
    assert 0 < held[0] - held[1] <= room // 5 + (257 << 20)
