"""A device buffer that is too short is refused, as the runtime's copies refuse
it, although full ones are read and written in place.

The short buffer is the lower of two neighbouring allocations that the test
owns, so not even a wrongly accepted call leaves mapped memory."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZE = 1 << 20


def _neighbours():
    """Two allocations of SIZE bytes, the second where the first ends, and all made."""
    rt = C.CDLL("libcudart.so.13")
    made = []
    for _ in range(16):
        p = C.c_void_p()
        assert rt.cudaMalloc(C.byref(p), C.c_size_t(SIZE)) == 0
        made.append(p.value)
        for low in made:
            if low + SIZE in made:
                return rt, low, made
    return rt, None, made


def test_short_device_buffer_is_refused_and_handle_stays_usable(rfmm_mod):
    torch = pytest.importorskip("torch")  # (the context; memory below is the runtime's)
    R = rfmm_mod
    from rfmm import scenes
    n = (SIZE + (1 << 16)) // 32
    p = scenes.plummer(n, seed=75)
    whole = torch.from_numpy(p.view(np.uint8).copy()).cuda()
    out = torch.zeros(32 * n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    rt, low, made = _neighbours()
    try:
        if low is None:
            pytest.skip("no two neighbouring allocations")
        for m in made:
            assert rt.cudaMemset(C.c_void_p(m), 0x5A, C.c_size_t(SIZE)) == 0
        assert rt.cudaDeviceSynchronize() == 0
        lib = R.lib()
        with R.Solver(n, R.default_params(gravity=1.0, softening=1e-3, dt=5e-4)) as s:
            s.upload_device(whole.data_ptr(), 32 * n)
            assert lib.rfmm_upload_particles_device(s.handle, low, 32 * n) == -2  # RFMM_ERR_CUDA
            assert lib.rfmm_download_device(s.handle, R.BUF_PARTICLES, low, 32 * n) == -2
            s.solve_fields()
            assert lib.rfmm_download_device(s.handle, R.BUF_FIELDS, low, 48 * s.cells) == -2
            s.download_device(R.BUF_PARTICLES, out.data_ptr(), 32 * n)  # the bodies of the good upload
            assert np.array_equal(out.cpu().numpy(), p.view(np.uint8))
            s.upload_device(whole.data_ptr(), 32 * n)
            s.step(2)
            s.sync()
        got = np.empty(SIZE, np.uint8)
        for m in made:
            assert rt.cudaMemcpy(C.c_void_p(got.ctypes.data), C.c_void_p(m), C.c_size_t(SIZE), 2) == 0
            assert np.all(got == 0x5A)
    finally:
        for m in made:
            rt.cudaFree(C.c_void_p(m))


@pytest.mark.parametrize("n", [257, 30001])
def test_managed_buffers_are_taken(rfmm_mod, n):
    """Managed memory goes the way of device memory, whatever its size."""
    pytest.importorskip("torch")
    R = rfmm_mod
    from rfmm import scenes
    p = scenes.plummer(n, seed=77)
    with R.Solver(n) as s:
        s.upload(p)
        s.step(2)
        want = s.particles()
    rt, at = C.CDLL("libcudart.so.13"), C.c_void_p()
    assert rt.cudaMallocManaged(C.byref(at), C.c_size_t(32 * n), C.c_uint(1)) == 0
    try:
        C.memmove(at.value, p.ctypes.data, 32 * n)
        with R.Solver(n) as s:
            s.upload_device(at.value, 32 * n)
            s.step(2)
            s.download_device(R.BUF_PARTICLES, at.value, 32 * n)
        got = np.frombuffer(C.string_at(at.value, 32 * n), np.uint8)
        assert np.array_equal(got, want.view(np.uint8))
    finally:
        rt.cudaFree(at)
