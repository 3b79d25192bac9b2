"""The one-launch FP64 Cholesky of the relay matrices at the edges of its
64-wide block columns and 128-row tiles, through the plain mode's screened
polarizabilities against the FP64 oracle (held to the plain mode's 1e-9
relative bar; backward error of a Cholesky solve at these condition numbers
is below 1e-12).  n = 3 N rows: a matrix smaller than a block column, one row
short of and past one and two block columns, an odd and an even number of
tiles, a last block column of 1, 2 and 63 rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [3, 21, 22, 42, 43, 64, 65, 85, 107, 128])
def test_relay_factor_edges(N):
    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    from oracle import mbd_oracle as o
    geo, st = sy.cluster(N, seed=400 + N)
    ref = o.mbd_at_rsscs(o.Geometry(geo.names, geo.coords, geo.hirshfeld, geo.lattice, geo.n_periodic), o.Settings())
    assert ref.status == "ok"
    with Engine(0) as eng:
        res = eng.energy(geo, st, "plain")
    assert res.status == 0
    np.testing.assert_allclose(res.alpha_iw, ref.alpha_iw, rtol=1e-9, atol=0)
    np.testing.assert_allclose(res.c6_eff, ref.c6_eff, rtol=1e-9, atol=0)
    assert abs(res.energy - ref.energy) <= 1e-9
