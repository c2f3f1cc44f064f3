"""The sort's bounded wait between tiles, made to run out: a tile whose
predecessor never publishes its counts gives up, the next tile stops as well,
neither writes, and the handle's own sorts go on as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [1, 2, 1024])
def test_sort_wait_gives_up_and_fails_closed(rfmm_mod, polls):
    R = rfmm_mod
    from rfmm import scenes
    p = scenes.plummer(20000, seed=76)
    prm = R.default_params(gravity=1.0, softening=1e-3, dt=5e-4)
    with R.Solver(len(p), prm) as s:
        s.upload(p)
        assert s.check_sort_timeout(polls) == R.RFMM_ERR_TIMEOUT
        assert s.check_sort_timeout(0) == R.RFMM_ERR_INVALID
        assert s.check_sort_timeout((1 << 22) + 1) == R.RFMM_ERR_INVALID
        assert s.device_error() == (0, 0)  # the engine's own error word is untouched
        s.upload(p)  # sorts again
        s.step(3)
        got = s.particles()
    with R.Solver(len(p), prm) as ref:
        ref.upload(p)
        ref.step(3)
        assert np.array_equal(got.view(np.uint32), ref.particles().view(np.uint32))
