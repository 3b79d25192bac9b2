"""The trace form's energy to rounding: against 0.5 sum sqrt(lambda) - 1.5 sum
omega from eigenvalues refined in extended precision, for the Hamiltonian of
the call's own polarizabilities.  Bound: 4e-16 of sum sqrt(lambda), a few
roundings of the sum -- the quadrature's truncation, which alone was up to 7e-16
of it with one node fewer, has to stay below them.  The eigenvalue path meets
the same bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _reference(geo, st, alpha, c6):
    from oracle import mbd_oracle as o
    H, _, _ = o.cfdm_hamiltonian(
        o._System(o.Geometry(list(geo.names), geo.coords, geo.hirshfeld, geo.lattice, geo.n_periodic),
                  o.Settings(xc=st.xc)), alpha, c6)
    H = np.tril(H) + np.tril(H, -1).T
    V = np.linalg.eigh(H)[1].astype(LD)
    lam = (V * H.astype(LD).dot(V)).sum(0) / (V * V).sum(0)          # Rayleigh quotients: errors squared
    omega = LD(4) / LD(3) * c6.astype(LD) / alpha.astype(LD) ** 2
    root = np.sqrt(lam).sum()
    return LD(0.5) * root - LD(1.5) * omega.sum(), root


# with one node fewer (40, 2) is off by 6.5e-16 of the sum
@pytest.mark.parametrize("N,k", [(12, 1), (12, 5), (20, 0), (40, 2), (61, 3), (100, 2), (200, 1)])
def test_energy_to_rounding(N, k, monkeypatch):
    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    geo, st = sy.cluster(N, seed=1000 + 10 * N + k)
    with Engine(0) as eng:
        res = eng.energy(geo, st, "plain")
        assert eng.timings()["trace_form"] > 0.0
    monkeypatch.setenv("MBD_B200_TRACE", "0")
    with Engine(0) as eng:
        eig = eng.energy(geo, st, "plain")
    assert np.array_equal(res.alpha_eff, eig.alpha_eff) and np.array_equal(res.c6_eff, eig.c6_eff)
    E, root = _reference(geo, st, res.alpha_eff, res.c6_eff)
    for r in (res, eig):
        assert abs(LD(r.energy) - E) * 2 <= LD(4e-16) * root
