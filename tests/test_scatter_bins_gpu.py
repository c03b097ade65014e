"""The binned particle scatter against the oracle's loop over all triangles,
bit for bit, where the bins can go wrong: slivers (whose hit test is wide of
their projection), triangles without area or with a vertex that is not finite,
large triangles that overflow the bins' lists, a flat mesh box, counts around
one warp, and a second call with a larger mesh on the same handle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(gpu, oracle_mod, soups, n):
    buf = gpu.GpuMpmBufferManager(n_particles=n)
    for soup in soups:
        mesh = gpu.GpuMeshBufferManager(vertices=soup)
        finite = soup[np.isfinite(soup).all(1)]
        mesh.min_coords, mesh.max_coords = finite.min(0), finite.max(0)
        init = gpu.GpuParticleInitializePipelineManager(mpm_manager=buf, mesh_manager=mesh,
                                                        uniforms_manager=gpu.GpuUniformsBufferManager())
        init.add_dispatch(n_particles=n)
        got = buf.read_particles(n)
        want = oracle_mod.scatter(mesh.vertices, mesh.min_coords, mesh.max_coords, n)
        assert np.array_equal(got.view(np.uint8).reshape(n, 192), want)
    buf.close()


def _sphere(gpu, sub, r=0.2, c=(0.45, 0.55, 0.5)):
    v, f = gpu.scenes.icosphere(sub, r, c)
    return v[f.astype(np.int64)]


def test_slivers_degenerate_and_non_finite(gpu, oracle_mod):
    rng = np.random.default_rng(2)
    base = _sphere(gpu, 2).reshape(-1, 3, 3)
    a, d = rng.uniform(0.3, 0.7, (60, 3)), rng.normal(0, 0.2, (60, 3))
    width = 10.0 ** rng.uniform(-7, -3, (60, 1))
    slivers = np.stack([a, a + d, a + d * rng.uniform(0.1, 0.9, (60, 1)) + width * rng.normal(0, 1, (60, 3))], 1)
    point = np.repeat(a[:4, None], 3, 1)
    bad = base[:6].copy()
    bad[0, 0, 0], bad[1, 1, 1], bad[2, 2, 2], bad[3, 0, 1], bad[4, 1, 2], bad[5, 2, 0] = (
        np.nan, np.inf, -np.inf, np.nan, np.inf, np.inf)
    soup = np.concatenate([base, slivers, point, bad]).astype(np.float32).reshape(-1, 3)
    _run(gpu, oracle_mod, [soup], 1500)


def test_large_triangles_overflow_the_lists(gpu, oracle_mod):
    rng = np.random.default_rng(3)
    boxes = []
    for _ in range(70):
        v, f = gpu.scenes.box_mesh(rng.uniform(0.0, 0.2, 3), rng.uniform(0.8, 1.0, 3))
        boxes.append(v[f.astype(np.int64)])
    big = np.concatenate(boxes * 3)      # each box three times: odd parity stays inside
    _run(gpu, oracle_mod, [big], 400)


@pytest.mark.parametrize("n", [1, 31, 33, 129])
def test_counts_and_a_growing_mesh(gpu, oracle_mod, n):
    _run(gpu, oracle_mod, [_sphere(gpu, 0), _sphere(gpu, 4), _sphere(gpu, 1)], n)


def test_flat_mesh_box(gpu, oracle_mod):
    tri = np.array([[0.2, 0.5, 0.2], [0.8, 0.5, 0.2], [0.5, 0.5, 0.8]] * 7, np.float32)   # 7 triangles, no y extent
    _run(gpu, oracle_mod, [tri], 40)


def test_bin_lists_past_32_bits(gpu, oracle_mod):
    """2^18 triangles, each in all 128 x 128 bins, total 2^32 list entries: the
    total must read as too long for the lists, not as its low 32 bits (which,
    with the box's own entries, lie below the lists' capacity)."""
    v, f = gpu.scenes.box_mesh((0.2, 0.3, 0.25), (0.8, 0.7, 0.75))
    box = v[f.astype(np.int64)].reshape(-1, 3).astype(np.float32)
    cover = np.array([[0.5, -9.0, -9.0], [0.5, 30.0, -9.0], [0.5, -9.0, 30.0]], np.float32)
    n_cover = 1 << 18                        # an even number: the box's parity stays
    n_tris = n_cover + len(box) // 3
    wrapped = (n_cover * 128 * 128) % 2 ** 32 + (len(box) // 3) * 128 * 128
    assert n_cover * 128 * 128 >= 2 ** 32 and wrapped <= 32 * n_tris + 16384
    soup = np.concatenate([box, np.tile(cover, (n_cover, 1))])
    mesh = gpu.GpuMeshBufferManager(vertices=soup)
    mesh.min_coords, mesh.max_coords = box.min(0), box.max(0)
    n = 40
    buf = gpu.GpuMpmBufferManager(n_particles=n)
    gpu.GpuParticleInitializePipelineManager(mpm_manager=buf, mesh_manager=mesh,
                                             uniforms_manager=gpu.GpuUniformsBufferManager()).add_dispatch(n_particles=n)
    got = buf.read_particles(n)
    buf.close()
    want = oracle_mod.scatter(mesh.vertices, mesh.min_coords, mesh.max_coords, n)
    assert np.array_equal(got.view(np.uint8).reshape(n, 192), want)
