"""Mixed solves when device memory is short (a torch allocation takes the rest
of it; nothing faults, allocations fail): the FP64 factors that do not fit are
tried once per upload, not once per compute, and a batch whose slots were
planned while there was room is planned again with fewer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


class _OnlyLeft:
    """Leaves `left` bytes of device memory free while it is entered."""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        import torch
        free, _ = torch.cuda.mem_get_info()
        assert free > self.left
        self.block = torch.empty(free - self.left, dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        import torch
        del self.block
        torch.cuda.empty_cache()


def _check(results, refs):
    for r, ref in zip(results, refs):
        assert r.status == ref.status == 0
        assert abs(r.energy - ref.energy) <= 1e-6                        # the mixed mode's bar
        np.testing.assert_allclose(r.alpha_iw, ref.alpha_iw, rtol=1e-8, atol=1e-12)


def test_factors_that_do_not_fit_are_tried_once():
    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    geo, st = sy.cluster(800, seed=12)       # FP64 factors 1015 MB, the FP32 path's buffers 640 MB
    with Engine(0) as eng:
        ref = eng.energy(geo, st, "plain")
        eng.energy(*sy.cluster(30, seed=1), "mixed")
        assert eng.upload([geo], [st]) == 0
        with _OnlyLeft(820 * MB):
            for k in range(3):
                assert eng.compute("mixed") == 0
                assert eng.stats()["graph_replayed"] == (k > 0)
                code, res = eng.download()
                assert code == 0 and res[0].refine_iters > 1             # not the FP64 factors
                _check(res, [ref])
        assert eng.upload([geo], [st]) == 0                              # room again: the factors again
        assert eng.compute("mixed") == 0
        code, res = eng.download()
        assert code == 0 and res[0].refine_iters == 1
        _check(res, [ref])


def test_fewer_slots_when_memory_ran_out():
    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    items = [sy.cluster(300, seed=40 + k) for k in range(8)]             # 140 MB of matrices each, as much for the factors
    geos, sts = [g for g, _ in items], [s for _, s in items]
    with Engine(0) as eng:
        eng.energy(*sy.cluster(30, seed=1), "mixed")
        refs = eng.energy_batch(geos, sts, "plain")
        with _OnlyLeft(300 * MB):
            _check(eng.energy_batch(geos, sts, "mixed"), refs)
        _check(eng.energy_batch(geos, sts, "mixed"), refs)
