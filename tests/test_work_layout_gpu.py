"""The work state holds the records' values without their padding: records set
from device memory come back with the padding they had until a substep runs
(which zeroes it), at counts around the 64 records one CTA stages, with padding
in some of the stages only, in full, in part and on the host; and the deferred
passes, the collider and the first transfer alone see the same state as before."""
import ctypes as C

import numpy as np
import pytest

from helpers import GpuScene, compare_states, make_params, run_oracle

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


def _scattered(gpu, kind, seed, n_side=13):
    spec = gpu.scenes.parity_scene(kind=kind, n_side=n_side, res=256, seed=seed)
    n = spec.particles.shape[0]
    rng = np.random.default_rng(seed)
    spec.particles["pos"] = rng.uniform(0.05, 0.95, (n, 3)).astype(np.float32)
    words = spec.particles.view(np.float32).reshape(n, 48)
    words[:, PAD] = rng.normal(size=(n, 10)).astype(np.float32)
    words[5 * 64:7 * 64, PAD] = 0.0
    return spec, words.view(np.uint32).copy()


def _check_kept(got, words, least=1000):
    """Every record is as it came, word for word, or advanced, with zero padding."""
    same = (got == words).all(1)
    moved = (got[:, :3] != words[:, :3]).any(1)
    assert same.sum() >= least and moved.sum() > 0
    assert not got[~same][:, PAD].any()


@pytest.mark.parametrize("kind", ["explicit", "pbmpm"])
@pytest.mark.parametrize("source", ["host", "device", "bound"])
def test_records_past_the_tile_storage_stay_as_they_came(gpu, kind, source):
    """Particles in tiles beyond the storage are left unchanged, padding and all,
    over several substeps and readbacks, however the records came in."""
    import torch

    spec, words = _scattered(gpu, kind, 53)
    n = words.shape[0]
    lib = gpu.load()
    dev = torch.from_numpy(words.view(np.float32).copy()).cuda()
    out = torch.full((n, 48), 7.0, device="cuda")
    buf = gpu.GpuMpmBufferManager(n_particles=n, tile_edge=8, max_tiles=40)
    pipe = gpu.GpuMpmPipelineManager(mpm_manager=buf, uniforms_manager=spec.uniforms,
                                     params=make_params(gpu, spec.params))
    torch.cuda.synchronize()
    if source == "host":
        buf.write_particles(spec.particles)
    elif source == "device":
        buf.write_particles_device(dev.data_ptr(), n)
    else:
        buf.bind_particles_device(dev.data_ptr(), n)
    for steps in (1, 2, 1):
        pipe.step(gpu.GpuSimulationMethodType(spec.method), steps)
        with pytest.raises(gpu.MpmError) as e:
            buf.sync()
        assert e.value.status == 0x2
        gpu._lib.check(lib.mpm_get_particles(buf.handle, C.c_void_p(out.data_ptr()), n, 1), buf.handle)
        torch.cuda.synchronize()
        _check_kept(out.cpu().numpy().view(np.uint32), words)
        if steps == 2:
            _check_kept(buf.read_particles().view(np.uint32).reshape(n, 48), words)
            part = buf.read_particles(n // 2).view(np.uint32).reshape(-1, 48)
            _check_kept(part, words[:n // 2], least=400)
    if source == "bound":
        _check_kept(dev.cpu().numpy().view(np.uint32), words)
    buf.close()


@pytest.mark.parametrize("kind", ["explicit", "pbmpm"])
def test_noalloc_leaves_records_past_its_tiles_as_they_came(gpu, kind):
    import torch

    spec, words = _scattered(gpu, kind, 54)
    n = words.shape[0]
    dev = torch.from_numpy(words.view(np.float32).copy()).cuda()
    torch.cuda.synchronize()
    ub, status, err = spec.uniforms.bytes(), C.c_uint32(0), C.create_string_buffer(256)
    params = make_params(gpu, spec.params)
    rc = gpu.load().mpm_step_noalloc(0, None, C.c_void_p(dev.data_ptr()), n, spec.method, ub, len(ub), C.byref(params),
                                     None, 0, 0, None, 0, C.byref(status), err, len(err))
    assert rc == -5 and status.value & 0x2
    torch.cuda.synchronize()
    _check_kept(dev.cpu().numpy().view(np.uint32), words)


def test_setting_and_getting_the_library_s_own_records(gpu):
    """The record buffer itself as source and destination, before and after a substep."""
    import torch

    spec = gpu.scenes.parity_scene(kind="explicit", n_side=10, seed=55)
    words = spec.particles.view(np.float32).reshape(-1, 48).copy()
    n = words.shape[0]
    words[:, PAD] = np.random.default_rng(5).normal(size=(n, 10))
    dev = torch.from_numpy(words).cuda()
    torch.cuda.synchronize()
    lib = gpu.load()
    lib.mpm_particles_device_ptr.restype = C.c_void_p
    g = GpuScene(gpu, spec)
    g.buf.write_particles_device(dev.data_ptr(), n)
    ptr = lib.mpm_particles_device_ptr(g.buf.handle)
    g.buf.write_particles_device(ptr, n)
    assert np.array_equal(g.particles().view(np.uint32).reshape(n, 48), words.view(np.uint32))
    assert g.step(2) == 0
    gpu._lib.check(lib.mpm_get_particles(g.buf.handle, C.c_void_p(ptr), n, 1), g.buf.handle)
    stepped = g.particles()
    g.buf.write_particles_device(ptr, n)
    assert np.array_equal(g.particles().view(np.uint8), stepped.view(np.uint8))
    g.close()
    other = GpuScene(gpu, spec)
    assert other.step(2) == 0
    compare_states(stepped, other.particles())
    other.close()
