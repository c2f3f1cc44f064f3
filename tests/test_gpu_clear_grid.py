"""An upload's time follows the larger of its two jobs, the bodies' keys and
the tree's clearing."""
import pytest

pytestmark = pytest.mark.gpu


def test_small_plan_with_a_deep_tree_is_not_cleared_by_one_sm(rfmm_mod):
    """255 bodies in a forced depth-6 tree clear the same 19 MB as 300,000
    bodies do, and do less of everything else."""
    torch = pytest.importorskip("torch")
    R = rfmm_mod
    from rfmm import scenes
    stream = torch.cuda.Stream()
    best = {}
    for n in (255, 300000):
        p = torch.from_numpy(scenes.uniform(n, seed=73).view("f4").reshape(n, 8).copy()).cuda()
        torch.cuda.synchronize()
        with R.Solver(n, R.default_params(depth=6)) as s:
            s.set_stream(stream.cuda_stream)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            times = []
            for _ in range(30):
                a.record(stream)
                s.upload_device(p.data_ptr(), 32 * n)
                b.record(stream)
                b.synchronize()
                times.append(a.elapsed_time(b))
            best[n] = min(times[5:])
            s.set_stream(None)
    print("upload, ms: %s" % best)
    assert best[255] <= best[300000], best
