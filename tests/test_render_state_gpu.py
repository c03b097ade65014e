"""The renderer passes read the simulation's work state: splats of one scene of
a batch and of a single scene after substeps, after new device records without
a substep and after host records, on grids around the aggregation rule's line,
equal the splats of the read-back records; marching cubes on partial blocks
with a scale that is no power of two; a ray march captured in a CUDA graph and
replayed after the handle's workspace has grown."""
import ctypes as C

import numpy as np
import pytest

from helpers import GpuScene, run_oracle

pytestmark = pytest.mark.gpu


def _splat_equal(gpu, oracle_mod, buf, rec, scale, res_density, scene=0, part=slice(None)):
    got = buf.calculate_density(res_density, scene=scene).cpu().numpy().view(np.uint32)
    want = oracle_mod.splat("density", np.ascontiguousarray(rec[part]), [0, 0, 0], [1, 1, 1], res_density, scale)
    assert want.sum() > 0 and np.array_equal(got, want)


def _scale(spec):
    return float(np.frombuffer(spec.uniforms.bytes()[4:8], "<f4")[0])


@pytest.mark.parametrize("res", [(24, 20, 16), (5, 5, 5), (3, 4, 2)])
def test_splat_follows_the_work_state(gpu, oracle_mod, res):
    import torch

    spec = gpu.scenes.parity_scene(kind="explicit", n_side=16)
    g = GpuScene(gpu, spec)
    sc = _scale(spec)
    _splat_equal(gpu, oracle_mod, g.buf, spec.particles, sc, res)       # host records, no substep yet
    assert g.step(2) == 0
    got = g.buf.calculate_density(res).cpu().numpy().view(np.uint32)    # before anything reads the records back
    rec = g.particles()
    assert np.array_equal(got, oracle_mod.splat("density", rec, [0, 0, 0], [1, 1, 1], res, sc))
    moved = spec.particles.copy()
    moved["pos"] = moved["pos"][:, [1, 2, 0]]
    dev = torch.from_numpy(moved.view(np.float32).reshape(-1).copy()).cuda()
    torch.cuda.synchronize()
    g.buf.write_particles_device(dev.data_ptr(), moved.shape[0])
    _splat_equal(gpu, oracle_mod, g.buf, moved, sc, res)
    g.close()


def test_splat_of_one_scene_of_a_batch(gpu, oracle_mod):
    specs = gpu.scenes.c3_batched(n_scenes=3, seed=12, lo_count=300, hi_count=900)
    b = gpu.GpuMpmBatch(specs)
    b.step(gpu.GpuSimulationMethodType.ExplicitMpm, 2)
    grids = [b.mpm.calculate_density((16, 12, 14), scene=i).cpu().numpy().view(np.uint32) for i in range(3)]
    b.mpm.sync()
    rec = b.mpm.read_particles()
    for i, (first, n) in enumerate(b.ranges):
        want = oracle_mod.splat("density", np.ascontiguousarray(rec[first:first + n]), [0, 0, 0], [1, 1, 1],
                                (16, 12, 14), _scale(specs[i]))
        assert want.sum() > 0 and np.array_equal(grids[i], want)
    b.close()


@pytest.mark.parametrize("scale", [2.0 ** 28, 3.0e7, 2.0 ** 60])
@pytest.mark.parametrize("dres,mres", [((20, 31, 14), (41, 9, 17)), ((40, 8, 30), (11, 23, 16))])
def test_mc_scales_and_resolutions(gpu, oracle_mod, scale, dres, mres):
    import torch

    rng = np.random.default_rng(9)
    z, y, x = np.meshgrid(*(np.arange(r) for r in dres[::-1]), indexing="ij")
    inside = ((x / dres[0] - 0.5) ** 2 + (y / dres[1] - 0.5) ** 2 + (z / dres[2] - 0.5) ** 2) < 0.11
    dens = (inside * rng.uniform(0.2, 2.0, inside.shape) * min(scale, 1e9)).astype(np.uint32)
    spec = gpu.scenes.parity_scene(kind="pbmpm", n_side=4)
    spec.uniforms.write_fixed_point_scale(scale)
    g = GpuScene(gpu, spec)
    want, n_want = oracle_mod.marching_cubes(dens, [0, 0, 0], [1, 1, 1], scale, mres)
    max_v = n_want + 30
    out = torch.zeros((max_v, 6), dtype=torch.float32, device="cuda")
    d_dev = torch.from_numpy(dens.view(np.int32)).cuda()
    cnt, gen = C.c_uint32(0), C.c_uint32(0)
    torch.cuda.synchronize()
    for cap in (max_v, n_want // 2 + 1):
        gpu._lib.check(gpu.load().mpm_marching_cubes(
            g.buf.handle, 0, C.c_void_p(d_dev.data_ptr()), (C.c_uint32 * 3)(*dres), (C.c_uint32 * 3)(*mres),
            C.c_void_p(out.data_ptr()), cap, C.byref(cnt), C.byref(gen)), g.buf.handle)
        assert gen.value == n_want and cnt.value == min(n_want, cap)
        assert np.array_equal(out[:cnt.value].cpu().numpy().view(np.uint32), want[:cnt.value].view(np.uint32))
    g.close()


def test_captured_ray_march_replays_after_the_workspace_grows(gpu, oracle_mod):
    import torch

    spec = gpu.scenes.parity_scene(kind="explicit", n_side=12)
    w, h = 33, 21
    M = gpu.scenes.camera_inv_view_proj((0.5, -0.8, 0.9), (0.5, 0.5, 0.35), w, h)
    spec.uniforms.write_view_proj_inv_mat(M.reshape(4, 4))
    spec.uniforms.write_time(5)
    stream = torch.cuda.Stream()
    buf = gpu.GpuMpmBufferManager(n_particles=spec.particles.shape[0], stream=stream.cuda_stream)
    buf.write_particles(spec.particles)
    gpu.GpuMpmPipelineManager(mpm_manager=buf, uniforms_manager=spec.uniforms)
    vol = gpu.GpuVolumetricBufferManager(grid_resolution=spec.res, screen_dims=(w, h))
    vol.depth.fill_(-1.0)
    rp = gpu.GpuVolumetricRenderPipelineManager(mpm_manager=buf, volumetric_manager=vol)
    rp.add_mass_calculation_dispatch()      # uploads the scene: not capturable
    buf.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        rp.add_raymarch_dispatch()
    # a larger workspace on the same handle between capture and replay
    mc = gpu.GpuMarchingCubesBufferManager(grid_resolution=(64, 64, 64), max_vertices=1000)
    gpu.GpuMarchingCubesRenderPipelineManager(mpm_manager=buf, mc_manager=mc).add_mesh_generation_pass()
    graph.replay()
    torch.cuda.synchronize()
    sc = _scale(spec)
    grid = oracle_mod.splat("mass", spec.particles, [0, 0, 0], [1, 1, 1], spec.res, sc)
    rgba, depth, color = oracle_mod.raymarch(grid, [0, 0, 0], [1, 1, 1], sc, M, 5, w, h)
    assert np.array_equal(vol.color.cpu().numpy().view(np.uint32), color.view(np.uint32))
    assert np.array_equal(vol.output.cpu().numpy(), rgba)
    assert np.array_equal(vol.depth.cpu().numpy().view(np.uint32), depth.view(np.uint32))
    del graph
    buf.close()


@pytest.mark.parametrize("order", ["lattice", "random"])
@pytest.mark.parametrize("res", [(16, 16, 16), (17, 15, 18), (40, 11, 12), (3, 4, 2), (5000, 1, 1)])
def test_splat_groups_of_a_warp(gpu, oracle_mod, order, res):
    """Warps whose particles share base cells wholly, partly and not at all, with
    base cells off both ends of the grid, on grids on each side of the rules
    (cells against particles)."""
    import torch

    spec = gpu.scenes.parity_scene(kind="explicit", n_side=17, seed=71)
    p = spec.particles
    rng = np.random.default_rng(72)
    p["pos"][:600] = rng.uniform(0.0, 1.0, (600, 3))
    p["pos"][600:700, 0] = np.float32(1.0) - np.float32(2.0) ** -24
    p["pos"][700:760] = 0.0
    if order == "random":
        spec.particles = p[rng.permutation(len(p))]
    g = GpuScene(gpu, spec)
    out = torch.zeros(res[::-1], dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for steps in (0, 1):
        if steps:
            assert g.step(steps) == 0
        g.buf.calculate_density(res, out=out)
        g.buf.sync()
        rec = g.particles()
        want = oracle_mod.splat("density", rec, [0, 0, 0], [1, 1, 1], res, _scale(spec))
        assert want.sum() > 0 and np.array_equal(out.cpu().numpy().view(np.uint32), want)
    g.close()


def test_captured_ray_marches_do_not_share_a_workspace(gpu, oracle_mod):
    """Two captured ray marches of one handle, over snow and over an empty grid,
    replayed at the same time on two streams beside the handle's own marches."""
    import torch

    res, w, h = (128, 128, 128), 160, 90
    M = gpu.scenes.camera_inv_view_proj((1.5, -0.8, 1.2), (0.5, 0.5, 0.4), w, h)
    spec = gpu.scenes.parity_scene(kind="explicit", n_side=4)
    spec.uniforms.write_grid_resolution(res)
    spec.uniforms.write_view_proj_inv_mat(M.reshape(4, 4))
    spec.uniforms.write_time(5)
    stream = torch.cuda.Stream()
    buf = gpu.GpuMpmBufferManager(n_particles=spec.particles.shape[0], stream=stream.cuda_stream)
    buf.write_particles(spec.particles)
    gpu.GpuMpmPipelineManager(mpm_manager=buf, uniforms_manager=spec.uniforms)
    buf.calculate_grid_mass(res)                       # uploads the scene: not capturable
    buf.sync()
    k = (np.arange(128) + 0.5) / 128 - 0.5
    ball = (k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2) < 0.05
    sc = _scale(spec)
    grids = [np.where(ball, np.uint32(300.0 / 128 ** 3 * sc), 0).astype(np.uint32), np.zeros(res, np.uint32)]
    vols, views, graphs, want = [], [], [], []
    for grid in grids:
        vol = gpu.GpuVolumetricBufferManager(grid_resolution=res, screen_dims=(w, h))
        vol.mass_grid.copy_(torch.from_numpy(grid.view(np.int32)))
        vols.append(vol)
        views.append(gpu.GpuVolumetricRenderPipelineManager(mpm_manager=buf, volumetric_manager=vol))
        want.append(oracle_mod.raymarch(grid, [0, 0, 0], [1, 1, 1], sc, M, 5, w, h)[2])
    torch.cuda.synchronize()
    for view in views:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            view.add_raymarch_dispatch()
        graphs.append(g)
    other = gpu.GpuVolumetricBufferManager(grid_resolution=res, screen_dims=(w, h), mass_grid=vols[1].mass_grid)
    own = gpu.GpuVolumetricRenderPipelineManager(mpm_manager=buf, volumetric_manager=other)
    replay = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(30):
        for vol in vols:
            vol.color.zero_()
        torch.cuda.synchronize()
        for s, g in zip(replay, graphs):
            with torch.cuda.stream(s):
                g.replay()
        own.add_raymarch_dispatch()
        torch.cuda.synchronize()
        for vol, color in zip(vols, want):
            assert np.array_equal(vol.color.cpu().numpy().view(np.uint32), color.view(np.uint32))
    # buffers of captures that are gone are used again
    graphs.clear()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(100):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            views[0].add_raymarch_dispatch()
        del g
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 8 << 20
    buf.close()


def test_large_workspaces_are_given_back(gpu):
    """Marching cubes over 512^3 cells needs 1.5 GB for the call and keeps none of
    it; a small one keeps its buffer."""
    import torch

    spec = gpu.scenes.parity_scene(kind="explicit", n_side=12)
    g = GpuScene(gpu, spec)
    assert g.step(1) == 0
    counts = []
    for m in (64, 512, 64):
        mc = gpu.GpuMarchingCubesBufferManager(grid_resolution=(64, 64, 64), mc_grid_resolution=(m,) * 3,
                                               max_vertices=100000)
        view = gpu.GpuMarchingCubesRenderPipelineManager(mpm_manager=g.buf, mc_manager=mc)
        mc.density_grid[9:14, 7:19, 8:12] = int(4 * _scale(spec))
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        counts.append(view.add_mesh_dispatches())
        torch.cuda.synchronize()
        assert free - torch.cuda.mem_get_info()[0] < 160 << 20
    assert counts[0] == counts[2] > 0 and counts[1] > 0
    g.close()


@pytest.mark.parametrize("bound", [True, False])
def test_splat_reads_what_the_caller_wrote_to_current_records(gpu, oracle_mod, bound):
    """Records that are up to date are the caller's to change: a bound buffer after
    a step, the library's after mpm_particles_device_ptr."""
    import torch

    spec = gpu.scenes.parity_scene(kind="explicit", n_side=12)
    n = spec.particles.shape[0]
    g = GpuScene(gpu, spec)
    own = torch.from_numpy(spec.particles.view(np.float32).reshape(-1).copy()).cuda()
    torch.cuda.synchronize()
    if bound:
        g.buf.bind_particles_device(own.data_ptr(), n)
    assert g.step(2) == 0
    lib, out = gpu.load(), torch.zeros((16, 20, 24), dtype=torch.int32, device="cuda")
    lib.mpm_particles_device_ptr.restype = C.c_void_p
    ptr = lib.mpm_particles_device_ptr(g.buf.handle)
    g.buf.sync()
    rec = g.particles()
    rec["pos"] = rec["pos"][:, [1, 2, 0]]
    src = torch.from_numpy(rec.view(np.float32).reshape(-1).copy()).cuda()
    if bound:
        own.copy_(src)
    else:
        # the buffer of another handle is as good as any way to write there
        writer = gpu.GpuMpmBufferManager(n_particles=n)
        writer.write_particles(rec)
        gpu._lib.check(lib.mpm_get_particles(writer.handle, C.c_void_p(ptr), n, 1), writer.handle)
        writer.sync()
        writer.close()
    torch.cuda.synchronize()
    g.buf.calculate_density((24, 20, 16), out=out)
    g.buf.sync()
    g.close()
    want = oracle_mod.splat("density", rec, [0, 0, 0], [1, 1, 1], (24, 20, 16), _scale(spec))
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)


def test_splats_of_every_scene_of_a_batch(gpu, oracle_mod):
    """More scenes than are looked up in the work state, twice over, with a step
    between and a set of device records at the end."""
    import torch

    specs = gpu.scenes.c3_batched(n_scenes=7, seed=13, lo_count=200, hi_count=500)
    b = gpu.GpuMpmBatch(specs)
    outs = [torch.zeros((14, 12, 16), dtype=torch.int32, device="cuda") for _ in specs]
    torch.cuda.synchronize()
    for part in range(3):
        if part < 2:
            b.step(gpu.GpuSimulationMethodType.ExplicitMpm, 1)
        else:
            rec = b.mpm.read_particles()[::-1].copy()
            rec["pos"] = rec["pos"][:, [2, 0, 1]]
            dev = torch.from_numpy(rec.view(np.float32).reshape(-1).copy()).cuda()
            torch.cuda.synchronize()
            b.mpm.write_particles_device(dev.data_ptr(), rec.shape[0])
        for i in range(7):
            b.mpm.calculate_density((16, 12, 14), scene=i, out=outs[i])
        b.mpm.sync()
        rec = b.mpm.read_particles()
        for i, (first, n) in enumerate(b.ranges):
            want = oracle_mod.splat("density", np.ascontiguousarray(rec[first:first + n]), [0, 0, 0], [1, 1, 1],
                                    (16, 12, 14), _scale(specs[i]))
            assert want.sum() > 0 and np.array_equal(outs[i].cpu().numpy().view(np.uint32), want)
    b.close()
