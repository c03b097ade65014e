"""Records that enter and leave through device memory: 16-byte aligned
buffers of the handle's GPU move straight between the caller's buffer and the
work state, anything else through the staged copy.  Both must hold the same
bits as the host path, before and after substeps, at counts around the 64
records one CTA stages."""
import ctypes as C

import numpy as np
import pytest

from helpers import GpuScene

pytestmark = pytest.mark.gpu


def _get(gpu, buf, ptr, n):
    gpu._lib.check(gpu.load().mpm_get_particles(buf.handle, C.c_void_p(ptr), n, 1), buf.handle)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000])
@pytest.mark.parametrize("offset", [0, 1])   # in floats: 1 is not 16-byte aligned
def test_device_records_equal_host_records(gpu, n, offset):
    import torch

    spec = gpu.scenes.parity_scene(kind="explicit", n_side=10)
    spec.particles = spec.particles[:n].copy()
    host = GpuScene(gpu, spec)
    dev = GpuScene(gpu, spec)
    words = torch.zeros(n * 48 + 4, device="cuda")
    words[offset:offset + n * 48] = torch.from_numpy(spec.particles.view(np.float32).reshape(-1).copy()).cuda()
    out = torch.full((n * 48 + 4,), 7.0, device="cuda")
    torch.cuda.synchronize()
    for steps in (0, 2):
        dev.buf.write_particles_device(words.data_ptr() + 4 * offset, n)
        host.buf.write_particles(spec.particles)
        if steps:
            assert dev.step(steps) == 0 and host.step(steps) == 0
        want = host.particles()
        for dst_offset in (0, 1):
            _get(gpu, dev.buf, out.data_ptr() + 4 * dst_offset, n)
            dev.buf.sync()
            got = out[dst_offset:dst_offset + n * 48].cpu().numpy()
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32).reshape(-1)), (steps, dst_offset)
        part = (n + 1) // 2     # a leading part of the records
        _get(gpu, dev.buf, out.data_ptr(), part)
        dev.buf.sync()
        got = out[:part * 48].cpu().numpy()
        assert np.array_equal(got.view(np.uint32), want[:part].view(np.uint32).reshape(-1)), steps
        assert np.array_equal(dev.particles().view(np.uint32), want.view(np.uint32))
    host.close()
    dev.close()
