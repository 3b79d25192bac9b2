"""A compute's results can be downloaded more than once: geometries whose
energy comes from the trace form, and geometries it refuses (chains of alkali
atoms with imaginary or soft modes), whose Hamiltonian the first download's
eigenvalue reduction uses up.  Every download against the oracle (1e-9 Ha, the
plain mode's bar) and bit-equal to the first; with the two-stage and the
one-stage reduction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _oracle(geo, st):
    from oracle import mbd_oracle as o
    return o.mbd_at_rsscs(o.Geometry(list(geo.names), geo.coords, geo.hirshfeld, geo.lattice, geo.n_periodic),
                          o.Settings(xc=st.xc))


def _chain(element, n, d):
    from mbd_b200 import Geometry, Settings
    return Geometry([element] * n, np.array([[d * i, 0.0, 0.0] for i in range(n)]), np.ones(n)), Settings(xc=1)


@pytest.mark.parametrize("two_stage", [True, False])
def test_repeated_downloads(two_stage, monkeypatch):
    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    if not two_stage:
        monkeypatch.setenv("MBD_B200_TWO_STAGE", "0")
        monkeypatch.setenv("MBD_B200_TRACE", "1")
    items = [_chain("K", 12, 3.0), sy.cluster(30, seed=5), _chain("Na", 12, 4.5), _chain("K", 40, 3.0)]
    refs = [_oracle(g, s) for g, s in items]
    assert any(r.nimag > 0 for r in refs) and any(r.nimag == 0 for r in refs)
    with Engine(0) as eng:
        assert eng.upload([g for g, _ in items], [s for _, s in items]) == 0
        for compute in range(2):
            assert eng.compute("plain") == 0
            code, first = eng.download()
            assert code == 0
            for r, ref in zip(first, refs):
                assert r.status == 0 and r.nimag == ref.nimag
                assert abs(r.energy - ref.energy) <= 1e-9
            for again in range(2):
                code, res = eng.download()
                assert code == 0
                for r, f in zip(res, first):
                    assert r.status == 0 and r.nimag == f.nimag and r.energy == f.energy
