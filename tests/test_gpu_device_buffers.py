"""Device uploads and downloads give the host path's bodies whatever the
caller's buffer: 32-byte aligned (read and written in place) or not (copied)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 30001])
@pytest.mark.parametrize("offset", [0, 4, 16, 32])
def test_device_buffers_at_any_alignment(rfmm_mod, n, offset):
    torch = pytest.importorskip("torch")
    R = rfmm_mod
    from rfmm import scenes
    p = scenes.make("plummer", n, 61)
    with R.Solver(n) as s:
        s.upload(p)
        s.step(3)
        want = s.particles()
    raw = torch.zeros(32 * n + 96, dtype=torch.uint8, device="cuda")
    assert raw.data_ptr() % 32 == 0
    raw[offset: offset + 32 * n] = torch.from_numpy(p.view(np.uint8).copy()).cuda()
    out = torch.full((32 * n + 96,), 0xA5, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with R.Solver(n) as s:
        s.upload_device(raw.data_ptr() + offset, 32 * n)
        s.step(3)
        s.download_device(R.BUF_PARTICLES, out.data_ptr() + offset, 32 * n)
    got = out.cpu().numpy()
    assert np.array_equal(got[offset: offset + 32 * n], want.view(np.uint8))
    assert np.all(got[:offset] == 0xA5) and np.all(got[offset + 32 * n:] == 0xA5)
