"""A batch's tuning says what it launches: rules on the batch's size are
defaults, and explicit values are taken as they are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scenes_n,pdl", [((4096, 9000, 30000), 1), ((5 * 1048576, 65536), 0)])
def test_batch_defaults_and_explicit_values(rfmm_mod, scenes_n, pdl):
    """Both sides of 96 tiles per SM (3.7 million bodies on 152)."""
    R = rfmm_mod
    torch = pytest.importorskip("torch")
    from rfmm import scenes
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = sum((n + 255) // 256 for n in scenes_n)
    assert (tiles > 96 * sms) == (pdl == 0)
    ps = [scenes.uniform(n, seed=80 + i) for i, n in enumerate(scenes_n)]
    prm = R.default_params(gravity=1.0, softening=1e-3, dt=5e-4)
    want = None
    for change in (dict(), dict(pdl=1 - pdl), dict(m2l_ctas_per_sm=6), dict(integrate_ctas_per_sm=1)):
        with R.Batch(scenes_n, [prm] * len(ps)) as b:
            t = b.tuning()
            assert (t.pdl, t.m2l_ctas_per_sm) == (pdl, 4)
            for k, v in change.items():
                setattr(t, k, v)
            b.set_tuning(t)
            assert b.tuning().as_dict() == t.as_dict()
            for i, p in enumerate(ps):
                b.upload(i, p)
            b.commit()
            b.step(2)
            got = [b.download(i) for i in range(len(ps))]
        if want is None:
            want = got
        for g, w in zip(got, want):
            assert np.array_equal(g.view(np.uint32), w.view(np.uint32)), change


def test_plain_defaults(rfmm_mod):
    R = rfmm_mod
    with R.Solver(1 << 20) as s:
        assert (s.tuning().pdl, s.tuning().m2l_ctas_per_sm) == (1, 6)
