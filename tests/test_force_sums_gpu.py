"""The PBMPM force sums that the first transfer forms for the iterations, against
the oracle, bit for bit: gravity along each single axis, several or none, the
interaction force in both modes, every tile edge, one to four iterations, and
scales that are and are not a power of two."""
import numpy as np
import pytest

from helpers import GpuScene, compare_states, make_params, run_oracle

pytestmark = pytest.mark.gpu


def _check(gpu, oracle_mod, spec, edge, steps=2):
    g = GpuScene(gpu, spec, tile_edge=edge)
    assert g.step(steps) == 0
    got = g.particles()
    g.close()
    o, want = run_oracle(oracle_mod, spec, n_steps=steps)
    o.close()
    compare_states(got, want)


@pytest.mark.parametrize("edge", [0, 8, 12, 14, 16])
@pytest.mark.parametrize("gravity,mode", [((-3.0, 0, 0), None), ((0, 4.0, 0), None), ((0, 0, 0), None),
                                          ((1.0, 0, -9.81), None), ((0, 0, -9.81), 0), ((2.0, 1.0, -9.81), 1)])
def test_force_directions(gpu, oracle_mod, edge, gravity, mode):
    # at tile_edge 0 a scene of 28^3 particles runs at edge 4
    spec = gpu.scenes.parity_scene(kind="pbmpm", n_side=28 if edge == 0 else 14, seed=41, interaction=mode is not None)
    spec.params["gravity"] = gravity
    if mode is not None:
        spec.uniforms.write_interaction_mode(mode)
    _check(gpu, oracle_mod, spec, edge)


@pytest.mark.parametrize("n_iter", [1, 2, 4])
@pytest.mark.parametrize("interaction", [False, True])
@pytest.mark.parametrize("scale", [2.0 ** 28, 2.5e8])
def test_iterations_and_scales(gpu, oracle_mod, n_iter, interaction, scale):
    spec = gpu.scenes.parity_scene(kind="pbmpm", n_side=14, seed=42, interaction=interaction, n_iter=n_iter)
    spec.uniforms.write_fixed_point_scale(scale)
    for edge in (8, 16):
        _check(gpu, oracle_mod, spec, edge)


def test_interaction_switched_on_and_off(gpu, oracle_mod):
    """The planes a handle needs change between substeps."""
    spec = gpu.scenes.parity_scene(kind="pbmpm", n_side=14, seed=43, interaction=True)
    g = GpuScene(gpu, spec, tile_edge=8)
    o, want = None, spec.particles.copy()
    for on in (False, True, True, False):
        spec.uniforms.write_is_interacting(on)
        assert g.step(1) == 0
        if o is not None:
            o.close()
        o, want = run_oracle(oracle_mod, spec, n_steps=1, particles=want)
        assert np.array_equal(g.grid(), o.dense_grid(spec.uniforms.bytes()))
    got = g.particles()
    g.close()
    o.close()
    compare_states(got, want)


def _capture_scene(gpu, kind, with_collider, n_iter=3):
    import torch

    spec = gpu.scenes.parity_scene(kind=kind, n_side=14, seed=44, with_collider=with_collider, n_iter=n_iter)
    stream = torch.cuda.Stream()
    buf = gpu.GpuMpmBufferManager(n_particles=spec.particles.shape[0], tile_edge=8, stream=stream.cuda_stream)
    buf.write_particles(spec.particles)
    pipe = gpu.GpuMpmPipelineManager(mpm_manager=buf, uniforms_manager=spec.uniforms,
                                     params=make_params(gpu, spec.params))
    gpu.load().mpm_use_graphs(buf.handle, 0)
    return spec, stream, buf, pipe


def _oracle_steps(oracle_mod, spec, methods, collider=None):
    p = spec.particles.copy()
    o = oracle_mod.Oracle(p.shape[0], max_blocks=200000, hash_size=2000003)
    for method, uniforms, col in methods:
        o.set_collider(*(spec.mesh if col else (None, None)))
        o.step(uniforms, spec.params, p, method, 0)
    o.close()
    return p


def test_first_pbmpm_step_of_a_handle_under_capture(gpu, oracle_mod):
    """A handle that has run explicit substeps only captures a PBMPM substep."""
    import torch

    spec, stream, buf, pipe = _capture_scene(gpu, "pbmpm", False)
    pipe.add_explicit_mpm_dispatches(n_particles=buf.n_particles)
    assert buf.sync() == 0
    u = spec.uniforms.bytes()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        gpu._lib.check(gpu.load().mpm_step(buf.handle, 1, 1), buf.handle)
    graph.replay()
    torch.cuda.synchronize()
    assert buf.sync() == 0
    got = buf.read_particles()
    del graph
    buf.close()
    compare_states(got, _oracle_steps(oracle_mod, spec, [(0, u, False), (1, u, False)]))


@pytest.mark.parametrize("kind,n_iter", [("pbmpm", 1), ("pbmpm", 3), ("explicit", 3)])
def test_captured_substep_follows_the_uniforms_and_the_collider(gpu, oracle_mod, kind, n_iter):
    """A caller's capture of a substep, replayed after the interaction force was
    switched on and a collider was set: the replay reads both, and its buffers
    are still there after further steps of the handle."""
    import torch

    spec, stream, buf, pipe = _capture_scene(gpu, kind, True, n_iter)
    u, method = spec.uniforms, spec.method
    u.write_interaction_pos([16.0, 16.0, 10.0])
    u.write_interaction_strength(50.0)
    u.write_interaction_radius(7.0)
    u.write_is_interacting(False)
    pipe.step(gpu.GpuSimulationMethodType(method), 2)        # sizes the storage; an even number of substeps
    assert buf.sync() == 0
    steps = [(method, u.bytes(), False)] * 2
    out = torch.zeros((4, 4, 4), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        gpu._lib.check(gpu.load().mpm_step(buf.handle, method, 2), buf.handle)
    graph.replay()
    torch.cuda.synchronize()
    steps += [(method, u.bytes(), False)] * 2
    col = gpu.GpuColliderBufferManager(vertices=spec.mesh[0], indices=spec.mesh[1])
    u.write_is_interacting(True)
    gpu._lib.check(gpu.load().mpm_set_collider(buf.handle, 0, col.collider_data.ctypes.data, col.collider_data.size,
                                               col.num_indices, col.bvh_nodes.ctypes.data, col.bvh_nodes.shape[0]),
                   buf.handle)
    pipe.push_uniforms()
    buf.calculate_density((4, 4, 4), out=out)                # uploads the scene
    buf.sync()
    graph.replay()
    torch.cuda.synchronize()
    steps += [(method, u.bytes(), True)] * 2
    pipe.step(gpu.GpuSimulationMethodType(method), 2)
    assert buf.sync() == 0
    steps += [(method, u.bytes(), True)] * 2
    graph.replay()
    torch.cuda.synchronize()
    steps += [(method, u.bytes(), True)] * 2
    got = buf.read_particles()
    del graph
    buf.close()
    want = _oracle_steps(oracle_mod, spec, steps)
    compare_states(got, want)
    free = _oracle_steps(oracle_mod, spec, [(m, b, False) for m, b, _ in steps])
    assert not np.array_equal(free["pos"], want["pos"])


def test_switching_the_interaction_allocates_nothing(gpu):
    import torch

    spec = gpu.scenes.parity_scene(kind="pbmpm", n_side=30, seed=45, interaction=True)
    spec.uniforms.write_is_interacting(False)
    g = GpuScene(gpu, spec, tile_edge=16)
    assert g.step(4) == 0
    free = torch.cuda.mem_get_info()[0]
    for on in (True, False, True):
        spec.uniforms.write_is_interacting(on)
        assert g.step(2) == 0
        # a graph is set up the first time; the planes of these tiles take 20 MB
        assert free - torch.cuda.mem_get_info()[0] < 8 << 20
    g.close()
