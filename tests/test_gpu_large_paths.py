"""Relay paths that the size rules keep for large matrices.

* 3xTF32 factors with FP64 refinement (relay matrices above 5700 rows), forced
  for all sizes (MBD_B200_MIXED_DIRECT=0) at the edges of their 128-row panels
  and of the 64-row residual blocks, against the plain mode: the solve meets the
  residual gate of 1e-10, whose share in a polarizability is below 1e-7.
* The triangular solve of more than 8064 rows, a launch a step, in the plain
  mode, against the mixed mode's solve at that size: 2689 atoms, 8067 rows, the
  last block of either kernel ragged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(a, b):
    assert a.status == b.status == 0
    assert a.err_est[0] <= 1e-10 and a.refine_iters > 1     # refined, not the FP64 factors
    assert abs(a.energy - b.energy) <= 1e-6
    np.testing.assert_allclose(a.alpha_iw, b.alpha_iw, rtol=1e-7, atol=0)


@pytest.fixture(scope="module")
def refined():
    from mbd_b200 import Engine
    mp = pytest.MonkeyPatch()
    mp.setenv("MBD_B200_MIXED_DIRECT", "0")
    eng = Engine(0)
    yield eng
    eng.close()
    mp.undo()


@pytest.mark.parametrize("N", [2, 21, 22, 42, 43, 64, 85, 86, 128, 129, 171, 300])
def test_refinement_at_ragged_sizes(refined, N):
    from mbd_b200 import synthetic as sy
    geo, st = sy.cluster(N, seed=600 + N)
    _check(refined.energy(geo, st, "mixed"), refined.energy(geo, st, "plain"))


def test_refinement_in_a_batch(refined):
    from mbd_b200 import synthetic as sy
    items = [sy.cluster(n, seed=n) for n in (90, 43, 150, 21, 64, 200, 128, 33, 86)]
    geos, sts = [g for g, _ in items], [s for _, s in items]
    refs = refined.energy_batch(geos, sts, "plain")
    for a, b in zip(refined.energy_batch(geos, sts, "mixed"), refs):
        _check(a, b)


def test_triangular_solve_by_steps():
    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    geo, st = sy.cluster(2689, seed=5)
    with Engine(0) as eng:
        _check(eng.energy(geo, st, "mixed"), eng.energy(geo, st, "plain"))
