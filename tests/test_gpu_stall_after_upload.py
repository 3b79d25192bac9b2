"""The bulge chase's stalled wait (MBD_OPT_TEST_STALL_WAIT = 1) reaches a batch
that was uploaded before the option was set, as it does one uploaded after it:
the batch's energies then come from the eigenvalue path, whose chase times out;
with the option off again they come from the trace form."""
import pytest

pytestmark = pytest.mark.gpu

MBD_ERR_TIMEOUT = 7


@pytest.mark.parametrize("computed_before", [False, True])
def test_option_set_after_the_upload(computed_before):
    from mbd_b200 import Engine
    from mbd_b200 import synthetic as sy
    geo, st = sy.cluster(50, seed=31)
    with Engine(0) as eng:
        ref = eng.energy(geo, st, "plain")
        assert eng.upload([geo], [st]) == 0
        for k in range(2 * computed_before):
            assert eng.compute("plain") == 0
            assert eng.download()[0] == 0
        eng.set_option("wait_limit_s", 0.05)
        eng.set_option("test_stall_wait", 1)
        try:
            assert eng.compute("plain") == 0
            code, res = eng.download()
            assert code == MBD_ERR_TIMEOUT and res[0].status == MBD_ERR_TIMEOUT
        finally:
            eng.set_option("test_stall_wait", 0)
            eng.set_option("wait_limit_s", 2.0)
        for k in range(3):
            assert eng.compute("plain") == 0
            code, res = eng.download()
            assert code == 0 and eng.timings()["trace_form"] > 0.0
            assert abs(res[0].energy - ref.energy) <= 1e-9
