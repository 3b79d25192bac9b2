"""The block-CG iterations above the one-launch size (3 N > 2048 rows), whose
FP32 matrix pass goes in 64 x 128 chunks: odd and even numbers of 64-row
blocks, full and ragged last blocks, from zero and from a network, against the
direct FP64 solve (the learned mode's 1e-6 bar and its residual gate)."""
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


@pytest.mark.parametrize("N", [683, 704, 705, 725, 726])   # 3 N = 2049, 2112, 2115, 2175, 2178; 64-row blocks 33, 33, 34, 34, 35
def test_large_cluster(engine, N):
    from mbd_b200 import synthetic as sy
    geo, st = sy.cluster(N, seed=700 + N)
    ref = engine.energy(geo, st, "plain")
    for net in (False, True):
        engine.use_network(net)
        got = engine.energy(geo, st, "mixed_learned")
        assert got.status == ref.status == 0
        assert got.refine_iters > 0 and got.err_est[0] <= 1e-10
        np.testing.assert_allclose(got.alpha_iw, ref.alpha_iw, rtol=1e-6, atol=0)
        assert abs(got.energy - ref.energy) <= 1e-6
