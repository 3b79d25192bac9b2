"""A batch of geometries whose trace form is refused (chains of Na atoms with
imaginary modes, 12 to 120 rows, among clusters): each as the oracle has it,
and their eigenvalue stages share launches -- a batch issues one chase, one
bisection and one energy launch however many were refused, where a geometry by
itself needs the same three."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _oracle(geo, st):
    from oracle import mbd_oracle as o
    return o.mbd_at_rsscs(o.Geometry(list(geo.names), geo.coords, geo.hirshfeld, geo.lattice, geo.n_periodic),
                          o.Settings(xc=st.xc))


def _chain(n):
    from mbd_b200 import Geometry, Settings
    return Geometry(["Na"] * n, np.array([[4.5 * i, 0.0, 0.0] for i in range(n)]), np.ones(n)), Settings(xc=1)


def _tail_launches(eng, items):
    assert eng.upload([g for g, _ in items], [s for _, s in items]) == 0
    assert eng.compute("plain") == 0
    before = eng.stats()["launches"]
    code, res = eng.download()
    assert code == 0
    return eng.stats()["launches"] - before, res


@pytest.mark.parametrize("two_stage", [True, False])
def test_refused_geometries_share_their_launches(two_stage, monkeypatch):
    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    if not two_stage:
        monkeypatch.setenv("MBD_B200_TWO_STAGE", "0")
        monkeypatch.setenv("MBD_B200_TRACE", "1")
    sizes = [40, 33, 32, 31, 22, 21, 16, 11, 10, 5, 4]
    chains = [_chain(n) for n in sizes]
    with Engine(0) as eng:
        alone = [_tail_launches(eng, [c])[0] for c in chains]
        items = chains[:5] + [sy.cluster(25, seed=3), sy.cluster(70, seed=4)] + chains[5:]
        together, res = _tail_launches(eng, items)
    refused = sum(k > 0 for k in alone)
    assert refused >= 6
    # of a geometry's launches by itself at least two (bisection, energy) are shared
    assert 0 < together <= sum(alone) - 2 * (refused - 1)
    for r, (geo, st) in zip(res, items):
        ref = _oracle(geo, st)
        assert ref.status == "ok" and r.status == 0
        assert r.nimag == ref.nimag and abs(r.energy - ref.energy) <= 1e-9
