"""A step on a stream that is being captured is refused, whatever its length:
the handle's buffers alternate from step to step, so a captured step would
replay on stale ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 2, 17])
def test_step_under_capture_is_refused(rfmm_mod, steps):
    torch = pytest.importorskip("torch")
    R = rfmm_mod
    from rfmm import scenes
    p = scenes.plummer(5000, seed=72)
    prm = R.default_params(gravity=1.0, softening=1e-3, dt=5e-4)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    keep = torch.zeros(64, device="cuda")
    torch.cuda.synchronize()
    with R.Solver(len(p), prm) as s:
        s.set_stream(stream.cuda_stream)
        s.upload(p)
        s.sync()
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="thread_local")
            keep.add_(1.0)  # (a graph of its own)
            status = R.lib().rfmm_step(s.handle, steps)
            graph.capture_end()
        assert status == -2, status  # RFMM_ERR_CUDA
        s.step(3)  # the refused call changed nothing
        got = s.particles()
        s.set_stream(None)
    with R.Solver(len(p), prm) as s:
        s.upload(p)
        s.step(3)
        assert np.array_equal(got.view(np.uint32), s.particles().view(np.uint32))
