"""The collision pass against the oracle, bit for bit: snow inside the reach of
a bumpy surface whose mesh also holds triangles without area, slivers and
duplicates (equal distances), with paths too short for the swept test and long
enough for it, one scene and several in one handle."""
import numpy as np
import pytest

from helpers import GpuScene, compare_states, make_params, run_oracle

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


@pytest.mark.parametrize("kind", ["explicit", "pbmpm"])
@pytest.mark.parametrize("extra", [1, 200])
def test_leaf_past_the_last_triangle_bit_exact(gpu, oracle_mod, kind, extra):
    """A caller's tree whose leaf reaches past the index words: the words after
    them (here vertex 0, whose bits name three more vertices) make further
    triangles, up to the end of the buffer, as in the oracle."""
    from types import SimpleNamespace

    spec = _without_mesh(gpu, gpu.scenes.parity_scene(kind=kind, n_side=14, seed=52), kind)
    verts = np.array([[0, 0, 0], [0.1, 0.1, 0.31], [0.9, 0.1, 0.31], [0.5, 0.9, 0.31],
                      [0.1, 0.1, 0.33], [0.9, 0.1, 0.325], [0.5, 0.9, 0.335]], np.float32)
    verts[0] = np.array([4, 5, 6], np.uint32).view(np.float32)
    idx = np.array([1, 2, 3], np.uint32)
    nodes = np.zeros((1, 8), np.uint32)
    nodes[0, 0:3] = np.full(3, -9, np.float32).view(np.uint32)
    nodes[0, 4:7] = np.full(3, 9, np.float32).view(np.uint32)
    nodes[0, 7] = 0x80000000 | (1 + extra)
    data = np.concatenate([idx, verts.reshape(-1).view(np.uint32)])
    spec.uniforms = gpu.scenes.make_uniforms([0, 0, 0], [1, 1, 1], spec.res, 1e-3 if kind == "pbmpm" else 2e-4,
                                             2.0 ** 28, mesh=(verts, idx))
    buf = gpu.GpuMpmBufferManager(n_particles=spec.particles.shape[0], tile_edge=8)
    buf.write_particles(spec.particles)
    pipe = gpu.GpuMpmPipelineManager(
        mpm_manager=buf, uniforms_manager=spec.uniforms, params=make_params(gpu, spec.params),
        collider_manager=SimpleNamespace(num_indices=3, collider_data=data, bvh_nodes=nodes))
    pipe.step(gpu.GpuSimulationMethodType(spec.method), 3)
    assert buf.sync() == 0
    got = buf.read_particles()
    buf.close()

    def run(nodes):
        p = spec.particles.copy()
        o = oracle_mod.Oracle(p.shape[0], max_blocks=200000, hash_size=2000003)
        o._col = oracle_mod.OrCollider(data.ctypes.data, data.size, nodes.ctypes.data, 1)
        for _ in range(3):
            o.step(spec.uniforms.bytes(), spec.params, p, spec.method)
        o.close()
        return p

    compare_states(got, run(nodes))
    within = nodes.copy()
    within[0, 7] = 0x80000001
    assert not np.array_equal(run(within)["pos"], got["pos"])      # the further triangle was touched
