"""The block-CG phases that run in one cluster launch (3 N <= 2048 rows) at
the edges of their 64-row blocks, block pairs and 16-row tasks, from zero and
from a network, alone and side by side in a batch, against the direct FP64
solve (the learned mode's 1e-6 bar and its residual gate)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    eng = Engine(0)
    items = [sy.cluster(60, seed=90 + k) for k in range(6)]
    eng.learned_train([g for g, _ in items], [s for _, s in items], epochs=2, lr=2e-3, seed=1)
    yield eng
    eng.close()


def _check(a, b):
    assert a.status == b.status == 0
    assert a.refine_iters > 0 and a.err_est[0] <= 1e-10
    np.testing.assert_allclose(a.alpha_iw, b.alpha_iw, rtol=1e-6, atol=0)
    assert abs(a.energy - b.energy) <= 1e-6


@pytest.mark.parametrize("N", [3, 5, 21, 43, 64, 65, 86, 128, 150, 682, 683])
def test_one_cluster(engine, N):
    from mbd_b200 import synthetic as sy
    geo, st = sy.cluster(N, seed=500 + N)
    ref = engine.energy(geo, st, "plain")
    for net in (False, True):
        engine.use_network(net)
        _check(engine.energy(geo, st, "mixed_learned"), ref)


def test_side_by_side(engine):
    from mbd_b200 import synthetic as sy
    items = [sy.cluster(n, seed=30 + n) for n in (21, 43, 64, 100, 128, 150, 200, 250, 300, 11, 400)]
    geos, sts = [g for g, _ in items], [s for _, s in items]
    engine.use_network(True)
    refs = engine.energy_batch(geos, sts, "plain")
    for a, b in zip(engine.energy_batch(geos, sts, "mixed_learned"), refs):
        _check(a, b)
