"""The energy from shifted Cholesky factors against the oracle's eigenvalues
(1e-9 Ha, the plain mode's bar): Hamiltonians around one and two block
columns, an isolated pair, a periodic sheet with a vacuum axis and a 2 x 2 x 2
supercell; and the geometries it must refuse -- chains of alkali atoms with
imaginary modes, or a mode so soft that the certificate fails -- whose
energies and counts of imaginary modes come from the eigenvalues."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from mbd_b200 import Engine
    eng = Engine(0)
    yield eng
    eng.close()


def _oracle(geo, st):
    from oracle import mbd_oracle as o
    return o.mbd_at_rsscs(
        o.Geometry(list(geo.names), geo.coords, geo.hirshfeld, geo.lattice, geo.n_periodic),
        o.Settings(xc=st.xc, mbd_supercell_cutoff=st.mbd_supercell_cutoff, mbd_cfdm_dip_cutoff=st.mbd_cfdm_dip_cutoff,
                   mbd_scs_dip_cutoff=st.mbd_scs_dip_cutoff, mbd_scs_vacuum_axis=st.mbd_scs_vacuum_axis))


def _chain(element, n, d):
    from mbd_b200 import Geometry, Settings
    return Geometry([element] * n, np.array([[d * i, 0.0, 0.0] for i in range(n)]), np.ones(n)), Settings(xc=1)


def _case(name):
    from mbd_b200 import synthetic as sy
    if name == "sheet":
        return sy.graphene_sheet(3)
    if name == "box":
        return sy.periodic_box(24, 3, scs_cut=50.0, cfdm_cut=30.0, sc_cut=9.0)
    return sy.cluster(int(name), seed=70 + int(name))


@pytest.mark.parametrize("mode", ["plain", "mixed_learned"])
@pytest.mark.parametrize("name", ["2", "21", "22", "43", "64", "86", "200", "sheet", "box"])
def test_energy_matches_eigenvalues(engine, name, mode):
    geo, st = _case(name)
    ref = _oracle(geo, st)
    engine.use_network(False)
    res = engine.energy(geo, st, mode)
    assert res.status == 0 and ref.status == "ok"
    assert engine.timings()["trace_form"] > 0.0
    assert res.nimag == 0 == ref.nimag
    assert abs(res.energy - ref.energy) <= (1e-9 if mode == "plain" else 1e-6)


@pytest.mark.parametrize("element,n,d", [("K", 4, 4.0), ("K", 12, 3.0), ("Na", 12, 4.5), ("Na", 12, 5.0), ("Na", 8, 5.0)])
def test_imaginary_and_soft_modes(engine, element, n, d):
    geo, st = _chain(element, n, d)
    ref = _oracle(geo, st)
    assert ref.status == "ok"
    res = engine.energy(geo, st, "plain")
    assert res.status == 0 and res.nimag == ref.nimag
    assert abs(res.energy - ref.energy) <= 1e-9


def test_refused_and_accepted_in_one_batch(engine):
    from mbd_b200 import synthetic as sy
    items = [sy.cluster(90, seed=1), _chain("K", 12, 3.0), sy.cluster(40, seed=2), _chain("K", 4, 4.0)]
    refs = [_oracle(g, s) for g, s in items]
    assert engine.upload([g for g, _ in items], [s for _, s in items]) == 0
    for replay in range(3):
        assert engine.compute("plain") == 0
        code, res = engine.download()
        assert code == 0
        assert engine.stats()["graph_replayed"] == (replay > 0)
        for r, ref in zip(res, refs):
            assert r.status == 0 and r.nimag == ref.nimag
            assert abs(r.energy - ref.energy) <= 1e-9
