"""A relay solve whose residual is not a finite number misses the residual gate:
the learned mode started by a network of NaN or overflowing parameters gives
the direct FP64 solve's results (to rounding: the same code on the same
matrices), on both sides of the one-launch block CG's size limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [40, 700])
@pytest.mark.parametrize("value", [np.nan, 1e30])
def test_unusable_network(N, value):
    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    geo, st = sy.cluster(N, seed=N)
    with Engine(0) as eng:
        ref = eng.energy(geo, st, "plain")
        eng.set_learned_params(np.full(eng.lib.mbd_rsscs_learned_param_count(), value, dtype=np.float32))
        res = eng.energy(geo, st, "mixed_learned", check=False)
    assert ref.status == res.status == 0
    assert res.refine_iters == -1 and res.err_est[0] == np.inf
    assert abs(res.energy - ref.energy) <= 1e-9
    np.testing.assert_allclose(res.alpha_iw, ref.alpha_iw, rtol=1e-10, atol=0)
