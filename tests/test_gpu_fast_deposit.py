"""The fast float variant deposits the exact contract's integers for every
fixed-point scale: what integrate deposits for the positions it has moved
equals the oracle's moments of those positions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1000.0, 30000.0, 32768.0])
@pytest.mark.parametrize("n", [65536, 700001])
def test_fast_deposit_is_exact_for_any_scale(rfmm_mod, oracle_mod, n, scale):
    """Scales that are not powers of two round the product: at 30,000 a product
    and bias rounded once instead of in turn differ for about 3 coordinates in
    10,000.  Whole numbers, so no tolerance."""
    O, R = oracle_mod, rfmm_mod
    from rfmm import scenes
    p = scenes.uniform(n, seed=71)
    kw = dict(gravity=1.0, softening=1e-3, dt=5e-4)
    with R.Solver(n, R.default_params(fixed_point_scale=scale, **kw)) as s:
        s.set_float_mode(R.FLOAT_FAST)
        s.upload(p)
        s.step(2)
        moved = s.particles()
        s.solve_fields()  # on the tree integrate deposited
        got = s.moments()
    st = O.OracleState(moved, O.make_params(n, scale=scale, **kw))
    st.solve_fields()
    assert np.array_equal(got.view(np.uint32), st.moments.view(np.uint32))
