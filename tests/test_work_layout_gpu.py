"""The work state holds the records' values without their padding: records set
from device memory come back with the padding they had until a substep runs
(which zeroes it), at counts around the 64 records one CTA stages, with padding
in some of the stages only, in full, in part and on the host; and the deferred
passes, the collider and the first transfer alone see the same state as before."""
import ctypes as C

import numpy as np
import pytest

from helpers import GpuScene, compare_states, run_oracle

pytestmark = pytest.mark.gpu

PAD = [11, 15, 19, 23, 27, 31, 35, 39, 43, 47]


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 129, 1000])
@pytest.mark.parametrize("where", ["none", "all", "last", "second_stage"])
def test_padding_survives_until_a_substep(gpu, oracle_mod, n, where):
    import torch

    spec = gpu.scenes.parity_scene(kind="pbmpm", n_side=10, seed=51)
    spec.particles = spec.particles[:n].copy()
    rng = np.random.default_rng(n)
    words = spec.particles.view(np.float32).reshape(n, 48).copy()
    words[:, 3] = rng.normal(size=n)
    rows = {"none": [], "all": range(n), "last": [n - 1], "second_stage": range(64, min(n, 128))}[where]
    for r in rows:
        words[r, PAD] = rng.normal(size=10)
    src = torch.from_numpy(words).cuda()
    out = torch.full((n, 48), 7.0, device="cuda")
    lib = gpu.load()
    torch.cuda.synchronize()
    g = GpuScene(gpu, spec)

    def get(count):
        out.fill_(7.0)
        torch.cuda.synchronize()
        gpu._lib.check(lib.mpm_get_particles(g.buf.handle, C.c_void_p(out.data_ptr()), count, 1), g.buf.handle)
        g.buf.sync()
        return out[:count].cpu().numpy()

    assert g.step(1) == 0                       # leaves values in both work buffers
    g.buf.write_particles_device(src.data_ptr(), n)
    assert np.array_equal(get(n).view(np.uint32), words.view(np.uint32))
    assert np.array_equal(get((n + 1) // 2).view(np.uint32), words[: (n + 1) // 2].view(np.uint32))
    g.buf.write_particles_device(src.data_ptr(), n)
    assert g.p2g_only() == 0
    assert np.array_equal(g.particles().view(np.uint32).reshape(n, 48), words.view(np.uint32))
    assert np.array_equal(get(n).view(np.uint32), words.view(np.uint32))
    g.buf.write_particles_device(src.data_ptr(), n)
    assert g.step(1) == 0
    got = get(n)
    assert not got[:, PAD].any() and np.array_equal(got[:, 3], words[:, 3])
    o, want = run_oracle(oracle_mod, spec, particles=words.reshape(-1).view(gpu.PARTICLE_DTYPE).copy())
    o.close()
    compare_states(got.reshape(-1).view(gpu.PARTICLE_DTYPE), want)
    g.close()


@pytest.mark.parametrize("kind", ["explicit", "pbmpm"])
def test_substeps_with_collider_and_deferred_map(gpu, oracle_mod, kind):
    spec = gpu.scenes.parity_scene(kind=kind, n_side=13, seed=52, with_collider=True)
    lib = gpu.load()
    for deferred in (False, True):
        g = GpuScene(gpu, spec, tile_edge=8)
        if deferred:
            gpu._lib.check(lib.mpm_set_plasticity(g.buf.handle, 1, None, 0.0, 0.0, 0.0), g.buf.handle)
        assert g.step(3) == 0
        got = g.particles()
        g.close()
        o, want = run_oracle(oracle_mod, spec, n_steps=3)
        o.close()
        compare_states(got, want)
