"""Leaf assignment at and around cell boundaries, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [4, 5, 6])
def test_leaves_at_cell_boundaries_bit_exact(rfmm_mod, oracle_mod, depth):
    """Bodies on every cell boundary of an axis, 1 to 4,096 ulps to either side
    of it, beyond the grid's ends and at non-finite coordinates lie in the
    oracle's leaves (their moments are the oracle's)."""
    O, R = oracle_mod, rfmm_mod
    edge = ((np.arange((1 << depth) + 1, dtype=np.float64) * 2.0 / (1 << depth) - 1.0) * np.float32(1.6)).astype(np.float32)
    near = [edge]
    for ulps in (1, 2, 3, 8, 64, 1024, 4096):
        for sign in (-1, 1):
            x = edge.view(np.int32) + np.int32(sign * ulps)
            near.append(x.view(np.float32))
    x = np.concatenate(near + [np.float32([0.0, -0.0, 1e-30, -1e-30, 1.599984, -1.599984, 1.7, -1.7, 4e6, -4e6,
                                           1e9, -1e9, 3e38, -3e38, np.inf, -np.inf, np.nan])])
    x = np.where(np.abs(x) < 1e-37, np.float32(0.0), x)  # the steps of +-0 are subnormal or NaN patterns
    n = 3 * len(x)
    p = np.zeros(n, R.PARTICLE_DTYPE)
    p["pos"] = 0.3
    for axis in range(3):
        p["pos"][axis * len(x): (axis + 1) * len(x), axis] = x
    st = O.OracleState(p, O.make_params(n, gravity=1.0, softening=1e-3, dt=5e-4, depth=depth))
    st.solve_fields()
    with R.Solver(n, R.default_params(gravity=1.0, softening=1e-3, dt=5e-4, depth=depth)) as s:
        s.upload(p)
        s.solve_fields()
        assert np.array_equal(s.moments().view(np.uint32), np.asarray(st.moments).view(np.uint32))
