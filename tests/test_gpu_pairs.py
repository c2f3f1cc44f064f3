"""Integrate with two packed bodies per lane, the exact variant's form above 16
body tiles per SM, against the oracle bit for bit: scenes just below and above
that line, at counts that end inside a lane's pair."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def line(rfmm_mod):
    """The most bodies of one scene that still take one body per lane."""
    torch = pytest.importorskip("torch")
    return 16 * 256 * torch.cuda.get_device_properties(0).multi_processor_count


def _same(g, r, what):
    """Bit equality where the oracle is a number; NaN where it is NaN."""
    g, r = np.ascontiguousarray(g).view(np.uint32).ravel(), np.ascontiguousarray(r).view(np.uint32).ravel()
    nan = np.isnan(r.view(np.float32))
    assert np.array_equal(np.isnan(g.view(np.float32)), nan), what
    bad = np.nonzero(g[~nan] != r[~nan])[0]
    assert len(bad) == 0, "%s differs in %d of %d words" % (what, len(bad), len(g))


def _compare(R, O, p, steps, scale=0.0, tuning=(), near=0, **kw):
    kw = dict(dict(gravity=1.0, softening=1e-3, dt=5e-4), **kw)
    st = O.OracleState(p, O.make_params(len(p), scale=scale or None, near_mode=near, **kw))
    st.step(steps)
    with R.Solver(len(p), R.default_params(fixed_point_scale=scale, **kw)) as s:
        if near:
            s.set_near_mode(R.NEAR_P2P)
        if tuning:
            t = s.tuning()
            for k, v in tuning:
                setattr(t, k, v)
            s.set_tuning(t)
        s.upload(p)
        s.step(steps)
        _same(s.particles(), st.particles, "particles")
        assert np.array_equal(s.moments().view(np.uint32), st.moments.view(np.uint32)), "moments of the last step"


@pytest.mark.parametrize("more", [0, 1, 2, 255, 256, 257])
@pytest.mark.parametrize("spread", [0.01, 0.3])
def test_runs_at_odd_counts(rfmm_mod, oracle_mod, line, more, spread):
    """Fast bodies, no re-sort between five steps: leaves hold one run, many
    short ones and single bodies, and runs begin and end inside pairs."""
    rng = np.random.default_rng(more)
    n = line + more
    p = np.zeros(n, rfmm_mod.PARTICLE_DTYPE)
    p["pos"] = rng.normal(0.0, spread, (n, 3))
    p["vel"] = rng.normal(0.0, 40.0 * spread, (n, 3))
    _compare(rfmm_mod, oracle_mod, p, 5, tuning=(("integrate_dynamic", more % 2),))


@pytest.mark.parametrize("scale", [2.0 ** 15, 2.0 ** 22])
@pytest.mark.parametrize("depth", [4, 5, 6])
def test_cell_and_wall_boundaries(rfmm_mod, oracle_mod, line, depth, scale):
    """Bodies at and around cell boundaries, the soft wall's band, the world's
    edge, half fixed-point units and beyond the grid, non-finite ones among
    them, next to ordinary bodies in the same lane's pair."""
    rng = np.random.default_rng(depth)
    edge = np.concatenate([(np.arange((1 << depth) + 1) * 2.0 / (1 << depth) - 1.0) * 1.6,
                           [1.384, -1.384, 1.576, -1.576, 1.59, 1.599984, 1.7, 4e6, -4e6, 0.0, -0.0],
                           (np.arange(-20, 20) + 0.5) / 2.0 ** 15]).astype(np.float32)
    x = [edge]
    for ulps in (1, 2, 64, 4096):
        for sign in (-1, 1):
            y = (edge.view(np.int32) + np.int32(sign * ulps)).view(np.float32)
            x.append(np.where(np.abs(y) >= 1e-37, y, np.float32(0.0)))
    x = np.concatenate(x + [np.float32([1e9, -1e9, 3e38, -3e38, np.inf, -np.inf, np.nan])])
    n = line + 259
    p = np.zeros(n, rfmm_mod.PARTICLE_DTYPE)
    p["pos"] = rng.uniform(-1.5, 1.5, (n, 3))
    p["vel"] = np.where(np.arange(n)[:, None] % 2 == 0, np.float32(0.0), rng.normal(0.0, 2.0, (n, 3)))
    at = rng.permutation(n)[: 3 * len(x)]
    for axis in range(3):
        p["pos"][at[axis * len(x): (axis + 1) * len(x)], axis] = x
    for k in ("hue", "exc"):  # over their range and its ends
        p[k] = rng.choice(np.float32([0.0, 0.3, 0.5, 0.7, 0.70000005, 1.0, 0.99]), n)
    _compare(rfmm_mod, oracle_mod, p, 2, scale=scale, depth=depth)


@pytest.mark.parametrize("mode", [1.0, 2.0, 3.0])
def test_control_modes(rfmm_mod, oracle_mod, line, mode):
    from rfmm import scenes
    p = scenes.plummer(line + 1, seed=81)
    _compare(rfmm_mod, oracle_mod, p, 3, control_point=[0.45, 0.5, 0.55, 1.0], control_axis_mode=[0.3, 0.9, 0.2, mode])


def test_exact_pair_sums(rfmm_mod, oracle_mod, line):
    from rfmm import scenes
    _compare(rfmm_mod, oracle_mod, scenes.uniform(line + 1, seed=82), 2, near=1)


def test_batch_of_ragged_scenes(rfmm_mod, oracle_mod, line):
    """Scenes that change inside a CTA's tiles, each ending inside a pair."""
    O, R = oracle_mod, rfmm_mod
    from rfmm import scenes
    sizes = [line // 2 + 1, 1, 257, line // 2 - 513, 4099]
    kw = dict(gravity=1.0, softening=1e-3, dt=5e-4)
    ps = [scenes.make(("plummer", "uniform")[i % 2], n, 83 + i) for i, n in enumerate(sizes)]
    with R.Batch(sizes, [R.default_params(**kw)] * len(sizes)) as b:
        for i, p in enumerate(ps):
            b.upload(i, p)
        b.commit()
        b.step(20)  # over a re-sort
        got = [b.download(i) for i in range(len(ps))]
    for g, p in zip(got, ps):
        st = O.OracleState(p, O.make_params(len(p), **kw))
        st.step(20)
        _same(g, st.particles, "particles of %d" % len(p))
