"""A large geometry behind a batch of small ones, with the rest of the device
memory taken (a torch allocation; allocations fail, nothing faults): the memory
that the batch's slots hold is given back for it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_slots_of_an_earlier_batch_make_room():
    import torch

    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    items = [sy.cluster(300, seed=40 + k) for k in range(8)]
    geos, sts = [g for g, _ in items], [s for _, s in items]
    geo, st = sy.cluster(600, seed=3)
    with Engine(0) as eng:
        ref = eng.energy(geo, st, "plain")
    with Engine(0) as eng:
        before = torch.cuda.mem_get_info()[0]
        refs = eng.energy_batch(geos, sts, "mixed")
        free = torch.cuda.mem_get_info()[0]
        assert before - free > 2000 * MB              # eight slots of 300 MB
        left = 300 * MB                               # the large one's matrices and factors: 600 MB in one buffer
        block = torch.empty(free - left, dtype=torch.uint8, device="cuda")
        try:
            res = eng.energy(geo, st, "plain")
        finally:
            del block
            torch.cuda.empty_cache()
        again = eng.energy_batch(geos, sts, "mixed")
    assert res.status == ref.status == 0 and abs(res.energy - ref.energy) <= 1e-9
    np.testing.assert_allclose(res.alpha_iw, ref.alpha_iw, rtol=1e-9, atol=1e-12)
    for a, b in zip(again, refs):
        assert a.status == 0 and abs(a.energy - b.energy) <= 1e-9
