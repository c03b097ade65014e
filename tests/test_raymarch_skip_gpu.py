"""The ray march's shortcuts against the oracle, bit for bit: an empty grid, a
single occupied cell at a face, an edge and a corner of the grid, thin sheets
with gaps of a brick, resolutions that are no multiple of the brick, a scale
that is no power of two, very dense snow (exponents past the short polynomial),
non-cubic cells, image sizes around the CTA's tile."""
import numpy as np
import pytest

from helpers import GpuScene

pytestmark = pytest.mark.gpu


def _check(gpu, oracle_mod, grid, scale, eye, target, w, h, gmax=(1.0, 1.0, 1.0)):
    import torch

    res = grid.shape[::-1]
    spec = gpu.scenes.parity_scene(kind="pbmpm", n_side=4)
    u = spec.uniforms
    u.write_grid_resolution(res)
    u.write_grid_max_coords(gmax)
    u.write_fixed_point_scale(scale)
    M = gpu.scenes.camera_inv_view_proj(eye, target, w, h)
    u.write_view_proj_inv_mat(M.reshape(4, 4))
    u.write_time(991)
    g = GpuScene(gpu, spec)
    vol = gpu.GpuVolumetricBufferManager(grid_resolution=res, screen_dims=(w, h))
    vol.mass_grid.copy_(torch.from_numpy(grid.view(np.int32)))
    vol.depth.fill_(-1.0)
    torch.cuda.synchronize()
    gpu.GpuVolumetricRenderPipelineManager(mpm_manager=g.buf, volumetric_manager=vol).add_raymarch_dispatch()
    g.buf.sync()
    rgba, depth, color = oracle_mod.raymarch(grid, [0, 0, 0], list(gmax), scale, M, 991, w, h)
    assert np.array_equal(vol.color.cpu().numpy().view(np.uint32), color.view(np.uint32))
    assert np.array_equal(vol.output.cpu().numpy(), rgba)
    assert np.array_equal(vol.depth.cpu().numpy().view(np.uint32), depth.view(np.uint32))
    g.close()


def _fill(res, cells, density, scale):
    """Cells (z, y, x slices) filled to a density in kg/m^3 of the unit box."""
    grid = np.zeros(res[::-1], np.uint32)
    v = density / (res[0] * res[1] * res[2]) * scale
    for c in cells:
        grid[c] = np.uint32(min(v, 4e9))
    return grid


VIEW = ((1.5, -0.8, 1.2), (0.5, 0.5, 0.4))


@pytest.mark.parametrize("cells", [
    [], [(0, 0, 0)], [(-1, -1, -1)], [(-1, 7, 0)], [(0, slice(None), -1)],
    [(slice(None, None, 9), slice(None), slice(None))], [(slice(None), slice(2, 4), slice(None))]])
def test_sparse_grids(gpu, oracle_mod, cells):
    res = (22, 19, 27)
    _check(gpu, oracle_mod, _fill(res, cells, 500.0, 2.0 ** 28), 2.0 ** 28, *VIEW, 53, 37)


@pytest.mark.parametrize("density,scale", [(120.0, 2.0 ** 28), (3000.0, 2.0 ** 26), (4e5, 2.0 ** 20), (500.0, 3.0e8),
                                           (300.0, 0.75 * 2.0 ** 28)])
def test_densities_and_scales(gpu, oracle_mod, density, scale):
    res = (21, 24, 18)
    rng = np.random.default_rng(7)
    block = _fill(res, [(slice(3, 13), slice(5, 19), slice(4, 17))], density, scale)
    grid = (block * rng.uniform(0.0, 1.3, block.shape)).astype(np.uint32)
    _check(gpu, oracle_mod, grid, scale, *VIEW, 45, 33)


@pytest.mark.parametrize("w,h", [(1, 1), (16, 4), (17, 5), (15, 3), (31, 40)])
def test_image_sizes_and_non_cubic_cells(gpu, oracle_mod, w, h):
    res = (20, 13, 16)
    grid = _fill(res, [(slice(2, 9), slice(3, 10), slice(5, 15))], 400.0, 2.0 ** 28)
    _check(gpu, oracle_mod, grid, 2.0 ** 28, (1.9, -0.4, 0.9), (0.6, 0.4, 0.3), w, h, gmax=(1.3, 0.7, 1.1))


def test_axis_aligned_view(gpu, oracle_mod):
    res = (16, 16, 16)
    grid = _fill(res, [(slice(4, 12), slice(6, 8), slice(4, 12))], 400.0, 2.0 ** 28)
    _check(gpu, oracle_mod, grid, 2.0 ** 28, (0.5, -1.0, 0.5), (0.5, 1.0, 0.5), 33, 33)


@pytest.mark.parametrize("far,size,res", [(1.5e5, 20.0, 256), (2e5, 6.0, 128), (5e5, 3.0, 128), (3e3, 3.0, 128),
                                          (1.5e5, 6.0, 16)])
def test_cameras_far_from_the_grid(gpu, oracle_mod, far, size, res):
    """Parallel rays from so far off that the rounding of each step adds up to
    cells (and, last, from where it does not): no sample may be skipped by its
    number then."""
    import torch

    grid = np.zeros((res,) * 3, np.uint32)
    z, y, x = np.meshgrid(*(np.arange(res) + 0.5,) * 3, indexing="ij")
    scale = float(2.0 ** np.floor(np.log2(5e7 / (400 * (size / res) ** 3))))
    rng = np.random.default_rng(3)
    for _ in range(4):
        c, r = rng.uniform(0.2, 0.8, 3) * res, rng.uniform(0.08, 0.2) * res
        grid[((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) < r * r] = np.uint32(300 * (size / res) ** 3 * scale)
    d = np.array([0.7, -0.6, 0.39]) / np.linalg.norm([0.7, -0.6, 0.39])
    a1 = np.cross(d, [0, 0, 1])
    a1 /= np.linalg.norm(a1)
    M = np.zeros((4, 4))
    M[0, :3], M[1, :3], M[2, :3] = a1 * size * 0.5, np.cross(a1, d) * size * 0.5, -2 * d * far
    M[3, :3], M[3, 3] = size / 2 + d * far, 1
    M = M.astype(np.float32).reshape(-1)
    w, h = 31, 25
    spec = gpu.scenes.parity_scene(kind="pbmpm", n_side=4)
    u = spec.uniforms
    u.write_grid_resolution((res,) * 3)
    u.write_grid_max_coords([size] * 3)
    u.write_fixed_point_scale(scale)
    u.write_view_proj_inv_mat(M.reshape(4, 4))
    u.write_time(991)
    g = GpuScene(gpu, spec)
    vol = gpu.GpuVolumetricBufferManager(grid_resolution=(res,) * 3, screen_dims=(w, h))
    vol.mass_grid.copy_(torch.from_numpy(grid.view(np.int32)))
    vol.depth.fill_(-1.0)
    torch.cuda.synchronize()
    gpu.GpuVolumetricRenderPipelineManager(mpm_manager=g.buf, volumetric_manager=vol).add_raymarch_dispatch()
    g.buf.sync()
    rgba, depth, color = oracle_mod.raymarch(grid, [0, 0, 0], [size] * 3, scale, M, 991, w, h)
    g.close()
    assert (color[..., 3] > 0).sum() > 100
    assert np.array_equal(vol.color.cpu().numpy().view(np.uint32), color.view(np.uint32))
    assert np.array_equal(vol.output.cpu().numpy(), rgba)
    assert np.array_equal(vol.depth.cpu().numpy().view(np.uint32), depth.view(np.uint32))


@pytest.mark.parametrize("size,scale", [(2e-12, 2.0 ** 20), (3e7, 2.0 ** -60)])
def test_cells_at_the_ends_of_the_range(gpu, oracle_mod, size, scale):
    """Cells whose volume leaves the range of the divisions by way of a reciprocal;
    the camera of the large grid stands in the snow."""
    res = (14, 11, 12)
    grid = np.zeros(res[::-1], np.uint32)
    grid[2:9, 3:8, 4:11] = 4_000_000_000
    eye = (1.5 * size, -0.8 * size, 1.2 * size) if size < 1 else (0.5 * size, 0.45 * size, 0.5 * size)
    _check(gpu, oracle_mod, grid, scale, eye, (0.5 * size,) * 3, 33, 21, gmax=(size,) * 3)
