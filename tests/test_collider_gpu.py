"""The collision pass against the oracle, bit for bit: snow inside the reach of
a bumpy surface whose mesh also holds triangles without area, slivers and
duplicates (equal distances), with paths too short for the swept test and long
enough for it, one scene and several in one handle."""
import numpy as np
import pytest

from helpers import GpuScene, compare_states, run_oracle

pytestmark = pytest.mark.gpu


def _scene(gpu, kind, speed, seed=50):
    spec = gpu.scenes.parity_scene(kind=kind, n_side=14, seed=seed)
    rng = np.random.default_rng(seed)
    v, f = gpu.scenes.fbm_terrain(20, 0.08, seed, base=0.3, axis_up=2)
    f = f.reshape(-1, 3)
    k = v.shape[0]
    extra = np.array([[0.5, 0.5, 0.3], [0.5, 0.5, 0.3], [0.5, 0.5, 0.3],            # a point
                      [0.3, 0.4, 0.31], [0.7, 0.4, 0.31], [0.5, 0.4, 0.31],         # a segment
                      [0.35, 0.6, 0.3], [0.65, 0.6, 0.3], [0.5, 0.6 + 1e-5, 0.3]],  # a sliver
                     np.float32)
    tris = np.concatenate([f, f[rng.integers(0, len(f), 40)], k + np.arange(9).reshape(3, 3)])
    spec.mesh = (np.concatenate([v, extra]), tris.astype(np.uint32).reshape(-1))
    u = gpu.scenes.make_uniforms([0, 0, 0], [1, 1, 1], spec.res, 1e-3 if kind == "pbmpm" else 2e-4, 2.0 ** 28,
                                 mesh=spec.mesh)
    spec.uniforms = u
    spec.particles["vel"] *= np.float32(speed)
    spec.particles["dxp"] *= np.float32(speed)
    return spec


@pytest.mark.parametrize("kind", ["explicit", "pbmpm"])
@pytest.mark.parametrize("speed", [0.05, 4.0])
def test_contact_with_degenerate_triangles_bit_exact(gpu, oracle_mod, kind, speed):
    spec = _scene(gpu, kind, speed)
    g = GpuScene(gpu, spec, tile_edge=8)
    assert g.step(4) == 0
    got = g.particles()
    g.close()
    free = GpuScene(gpu, _without_mesh(gpu, spec, kind), tile_edge=8)
    assert free.step(4) == 0
    assert not np.array_equal(free.particles()["pos"], got["pos"])     # the collider was touched
    free.close()
    o, want = run_oracle(oracle_mod, spec, n_steps=4)
    o.close()
    compare_states(got, want)


def _without_mesh(gpu, spec, kind):
    import dataclasses

    u = gpu.scenes.make_uniforms([0, 0, 0], [1, 1, 1], spec.res, 1e-3 if kind == "pbmpm" else 2e-4, 2.0 ** 28)
    return dataclasses.replace(spec, mesh=None, uniforms=u)


def test_contact_in_a_batch_bit_exact(gpu, oracle_mod):
    specs = [_scene(gpu, "explicit", s, seed=60 + i) for i, s in enumerate((0.05, 1.0, 4.0))]
    specs[1] = _without_mesh(gpu, specs[1], "explicit")
    b = gpu.GpuMpmBatch(specs)
    b.step(gpu.GpuSimulationMethodType.ExplicitMpm, 3)
    assert b.mpm.sync() == 0
    rec = b.mpm.read_particles()
    for i, spec in enumerate(specs):
        o, want = run_oracle(oracle_mod, spec, n_steps=3)
        o.close()
        compare_states(b.scene_particles(i, rec), want)
    b.close()
