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


@pytest.mark.parametrize("scale", [2.0 ** 15, 2.0 ** 22])
@pytest.mark.parametrize("depth", [4, 6])
def test_steps_at_cell_and_wall_boundaries_bit_exact(rfmm_mod, oracle_mod, depth, scale):
    """Two steps of bodies at and around cell boundaries, the soft wall's band,
    the world's edge and half fixed-point units, slow and fast, at both ends of
    the deposit scale's range: every state and the last step's moments equal
    the oracle's."""
    O, R = oracle_mod, rfmm_mod
    rng = np.random.default_rng(depth)
    edge = np.concatenate([(np.arange((1 << depth) + 1) * 2.0 / (1 << depth) - 1.0) * 1.6,
                           [1.384, -1.384, 1.576, -1.576, 1.59, 1.599984, 1.7, 4e6, 0.0, -0.0],
                           (np.arange(-20, 20) + 0.5) / 2.0 ** 15]).astype(np.float32)
    x = [edge]
    for ulps in (1, 2, 64, 4096):
        for sign in (-1, 1):
            y = (edge.view(np.int32) + np.int32(sign * ulps)).view(np.float32)
            x.append(np.where(np.abs(y) >= 1e-37, y, np.float32(0.0)))
    x = np.concatenate(x)
    p = np.zeros(3 * len(x), R.PARTICLE_DTYPE)
    p["pos"] = rng.uniform(-1.5, 1.5, (len(p), 3))
    for axis in range(3):
        p["pos"][axis * len(x): (axis + 1) * len(x), axis] = x
    p["vel"] = np.where(np.arange(len(p))[:, None] % 2 == 0, np.float32(0.0), rng.normal(0.0, 2.0, (len(p), 3)))
    names = p.dtype.names
    for k in names:  # hue and excitation over their range and its ends
        if k not in ("pos", "vel"):
            p[k] = rng.choice(np.float32([0.0, 0.3, 0.5, 0.7, 0.70000005, 1.0, 0.99]), len(p))
    kw = dict(gravity=1.0, softening=1e-3, dt=5e-4, depth=depth)
    st = O.OracleState(p, O.make_params(len(p), scale=scale, **kw))
    st.step(2)
    with R.Solver(len(p), R.default_params(fixed_point_scale=scale, **kw)) as s:
        s.upload(p)
        s.step(2)
        assert np.array_equal(s.particles().view(np.uint32), st.particles.view(np.uint32))
        assert np.array_equal(s.moments().view(np.uint32), np.asarray(st.moments).view(np.uint32))


@pytest.mark.parametrize("n", [33, 255, 257, 4099])
@pytest.mark.parametrize("spread", [0.01, 0.2, 1.3])
def test_deposit_runs_bit_exact(rfmm_mod, oracle_mod, n, spread):
    """Steps without a re-sort between them, so that leaves hold one run, many
    short ones and single bodies, at odd counts that end inside a lane's pair:
    states and moments equal the oracle's."""
    O, R = oracle_mod, rfmm_mod
    rng = np.random.default_rng(n)
    p = np.zeros(n, R.PARTICLE_DTYPE)
    p["pos"] = rng.normal(0.0, spread, (n, 3))
    p["vel"] = rng.normal(0.0, 40.0 * spread, (n, 3))
    kw = dict(gravity=1.0, softening=1e-3, dt=5e-4, depth=4)
    st = O.OracleState(p, O.make_params(n, **kw))
    st.step(5)
    with R.Solver(n, R.default_params(**kw)) as s:
        s.upload(p)
        s.step(5)
        assert np.array_equal(s.particles().view(np.uint32), st.particles.view(np.uint32))
        assert np.array_equal(s.moments().view(np.uint32), np.asarray(st.moments).view(np.uint32))
