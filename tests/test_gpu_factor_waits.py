"""Waits of the Cholesky launches that run out (from the host: the first tiles
wait for a diagonal block that never comes, 50 ms limit) end with
MBD_ERR_TIMEOUT wherever these launches run: a plain compute, the FP64 re-run of
a solve that missed the residual gate, the labels of a training.  The context
then works again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MBD_ERR_TIMEOUT = 7


@pytest.fixture
def engine():
    from mbd_b200 import Engine
    with Engine(0) as eng:
        eng.set_option("wait_limit_s", 0.05)
        yield eng
        eng.set_option("wait_limit_s", 2.0)


def _items():
    from mbd_b200 import synthetic as sy
    return [sy.cluster(40, seed=6), sy.cluster(75, seed=7)]


def _split(items):
    return [g for g, _ in items], [s for _, s in items]


def _same(results, refs):
    for r, ref in zip(results, refs):
        assert r.status == ref.status == 0
        assert abs(r.energy - ref.energy) <= 1e-9
        np.testing.assert_allclose(r.alpha_iw, ref.alpha_iw, rtol=1e-8, atol=1e-12)


def test_plain_compute(engine):
    items = _items()
    refs = engine.energy_batch(*_split(items), "plain")
    engine.set_option("test_stall_wait", 2)
    assert engine.get_option("test_stall_wait") == 2.0
    for r in engine.energy_batch(*_split(items), "plain", check=False):
        assert r.status == MBD_ERR_TIMEOUT and np.isnan(r.energy)
    engine.set_option("test_stall_wait", 0)
    _same(engine.energy_batch(*_split(items), "plain"), refs)


@pytest.mark.parametrize("mode", ["mixed", "mixed_learned"])
def test_rerun_after_a_missed_gate(engine, mode):
    items = _items()
    refs = engine.energy_batch(*_split(items), "plain")
    engine.use_network(False)
    engine.set_option("residual_gate", 0.0)
    assert engine.upload(*_split(items)) == 0
    assert engine.compute(mode) == 0
    engine.set_option("test_stall_wait", 2)      # the compute ran without it
    code, res = engine.download()
    assert code == MBD_ERR_TIMEOUT
    assert res[0].status == MBD_ERR_TIMEOUT and np.isnan(res[0].energy)
    engine.set_option("test_stall_wait", 0)
    assert engine.compute(mode) == 0
    code, res = engine.download()
    assert code == 0 and all(r.refine_iters == -1 for r in res)
    _same(res, refs)


def test_training_labels(engine):
    from mbd_b200 import MbdError
    items = _items()
    engine.set_option("test_stall_wait", 2)
    with pytest.raises(MbdError) as e:
        engine.learned_train(*_split(items), epochs=1)
    assert e.value.code == MBD_ERR_TIMEOUT
    engine.set_option("test_stall_wait", 0)
    assert np.isfinite(engine.learned_train(*_split(items), epochs=1)).all()
