"""Performance cases: the work a user of this framework has it do.

A simulation pass takes the records of a scene that lie in GPU memory, advances
them some substeps and brings the advanced records back, in the caller's order
(`set`, `step`, `get` of the buffer and pipeline managers).  The other passes
are the particle scatter that fills a scene and the two renderers' passes over
a simulated state.  Inputs are procedural (jittered lattices of snow, tori,
terrain), made from the seed alone.

Case keys of a simulation: n particles, grid resolution res (cells per edge of
a cubic domain of edge `size`), particle spacing in cells, shape of the snow,
order of the records ("lattice": x fastest, "random": as the scatter leaves
them), n_iter PBMPM iterations, substeps of one pass, the constants ("config":
y up, grid boundary layer, xi = 10; "reference": z up, particle reflection
only), the collider, an interaction force, and the initial strain (standard
deviation of the entries of F_e, which makes the return map act).
"""
from __future__ import annotations

import ctypes
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("webgpu-mpm-based-snow-simulation_b200")

DENSITY = 400.0


def _sim(name, **over):
    c = dict(name=name, kind="step", method="explicit", n=32768, res=64, size=1.0, spacing=0.8, shape="block",
             order="lattice", n_iter=6, substeps=4, mode="config", collider="none", interaction=False, strain=0.0,
             dt=1e-4)
    c.update(over)
    return c


def listed():
    return [
        # the smallest call: one substep of a preview scene, a ragged particle count
        _sim("explicit_4k", n=4099, spacing=0.5, substeps=1, mode="reference"),
        # a cube of snow at 64^3, explicit, some substeps per frame
        _sim("explicit_32k", substeps=8),
        # the app's default scene: 300,000 scattered particles, 256^3 grid over a 10 m domain
        _sim("explicit_app_300k", n=300000, res=256, size=10.0, spacing=0.5, order="random", mode="reference",
             substeps=4, dt=1.0 / 192),
        # a large explicit scene with snow beyond its yield surface, ragged count
        _sim("explicit_1m", n=1000003, res=192, spacing=0.5, shape="slab", substeps=4, strain=0.01, dt=5e-5),
        # interactive PBMPM at the reference's constants with the user pushing the snow
        _sim("pbmpm_20k_touch", method="pbmpm", n=20011, res=64, spacing=0.5, n_iter=3, order="random",
             mode="reference", interaction=True, substeps=4),
        # two colliding snow balls inside a box with a sphere obstacle
        _sim("pbmpm_balls_262k", method="pbmpm", n=262144, res=128, spacing=0.6, shape="balls", collider="box",
             substeps=4, dt=2e-4),
        # snow lying on and sliding over a 130,050-triangle terrain
        _sim("pbmpm_terrain_512k", method="pbmpm", n=524288, res=256, spacing=0.7, shape="slab", collider="terrain",
             substeps=2, strain=0.005, dt=5e-5),
        # the large benchmark slab: 4,194,304 particles, 512^3 sparse grid
        _sim("pbmpm_slab_4m", method="pbmpm", n=4194304, res=512, spacing=1.6, shape="slab", substeps=1, dt=5e-5),
        # many independent scenes advanced by the same launches
        dict(name="batch_explicit_48", kind="batch", scenes=48, lo=2000, hi=60000, substeps=4, dt=1e-4),
        # one frame of the volumetric renderer: mass splat and ray march
        dict(name="volumetric_720p", kind="volumetric", n=300000, res=128, size=4.0, spacing=0.6, width=1280,
             height=720),
        # one frame of the surface renderer: density splat and marching cubes
        dict(name="surface_1m", kind="surface", n=1000000, res=256, size=10.0, spacing=1.0, mc_scale=1.0),
        # filling a closed mesh with particles (the start of every scene)
        dict(name="scatter_64k", kind="scatter", n=65536, u=64, v=40),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(n, spacing, shape):
    """Cells that the longest edge of the snow takes."""
    nx = _dims(n, shape)[0]
    return nx * spacing if shape != "balls" else 2.6 * nx * spacing


def draw(rng):
    kind = rng.choices(["explicit", "pbmpm", "noalloc", "batch", "volumetric", "surface", "scatter"],
                       [30, 34, 8, 7, 7, 7, 7])[0]
    if kind in ("explicit", "pbmpm", "noalloc"):
        small = kind == "noalloc"
        method = rng.choice(["explicit", "pbmpm"]) if small else kind
        spacing = rng.choice([0.5, 0.6, 0.7, 0.8] if small else [0.5, 0.6, 0.7, 0.8, 1.2, 1.6])
        n = _log_int(rng, 1000, 50000 if small else (2000000 if method == "explicit" else 1200000))
        shape = rng.choice(["block", "slab", "balls"])
        need = _cells(n, spacing, shape) / 0.75
        res = rng.choice([r for r in (48, 64, 96, 128, 160, 192, 256, 384, 512) if r >= need][:3])
        mode = rng.choice(["config", "reference"])
        c = _sim("", method=method, n=n, res=res, spacing=spacing, shape=shape,
                 order=rng.choice(["lattice", "random"]), n_iter=rng.choice([1, 2, 3, 4, 6]), mode=mode,
                 substeps=1 if small else rng.choice([1, 2, 4] if n > 200000 else [1, 2, 4, 8]),
                 interaction=method == "pbmpm" and rng.random() < 0.2, strain=rng.choice([0.0, 0.0, 0.005, 0.01]),
                 dt=rng.choice([5e-5, 1e-4]))
        if method == "pbmpm" and c["strain"]:
            # released strain throws PBMPM snow apart within a few substeps
            c.update(strain=0.005, substeps=min(c["substeps"], 2))
        if not small:
            c["collider"] = "none" if shape == "block" else ("box" if shape == "balls" else
                                                             rng.choice(["none", "terrain"]))
        else:
            c["kind"] = "noalloc"
        del c["name"]
        return c
    if kind == "batch":
        hi = _log_int(rng, 8000, 60000)
        return dict(kind="batch", scenes=rng.randint(3, 48), lo=rng.randint(1000, 4000), hi=hi,
                    substeps=rng.choice([1, 2, 4]), dt=1e-4)
    if kind == "volumetric":
        w = rng.randint(200, 1920)
        return dict(kind="volumetric", n=_log_int(rng, 20000, 600000), res=rng.choice([96, 128, 160, 192]), size=4.0,
                    spacing=rng.choice([0.5, 0.6, 0.7]), width=w, height=max(100, w * 9 // 16))
    if kind == "surface":
        return dict(kind="surface", n=_log_int(rng, 20000, 1500000), res=rng.choice([160, 192, 224, 256]), size=10.0,
                    spacing=rng.choice([0.8, 1.0]), mc_scale=rng.choice([0.75, 1.0, 1.5]))
    return dict(kind="scatter", n=_log_int(rng, 2000, 120000), u=rng.randint(6, 64), v=rng.randint(5, 40))


# ----------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------
def _dims(n, shape):
    if shape == "slab":
        a = max(1, math.ceil((n / 16.0) ** (1 / 3)))
        return 4 * a, max(1, math.ceil(n / (16.0 * a * a))), 4 * a
    if shape == "balls":
        m = math.ceil((n / 2 / (math.pi / 6)) ** (1 / 3)) + 2
        return m, m, m
    m = math.ceil(n ** (1 / 3))
    return m, m, max(1, math.ceil(n / (m * m)))


def _lattice(dims, gen):
    nx, ny, nz = dims
    i = torch.arange(nx * ny * nz, device="cuda")
    ijk = torch.stack([i % nx, (i // nx) % ny, i // (nx * ny)], 1).double()
    u = torch.rand(ijk.shape, generator=gen, device="cuda", dtype=torch.float64) - 0.5
    return ijk + 0.5 + u - torch.tensor([nx / 2, ny / 2, nz / 2], device="cuda", dtype=torch.float64)


def _positions(c, gen):
    """Particle positions in cells from the domain's centre, and the sign of a ball's velocity along x."""
    n, shape = c["n"], c.get("shape", "block")
    p = _lattice(_dims(n, shape), gen) * c["spacing"]
    sign = torch.zeros(n, device="cuda", dtype=torch.float64)
    if shape != "balls":
        return p[:n], sign
    near = torch.argsort((p * p).sum(1))          # the lattice points nearest the centre
    a, b = p[near[: n - n // 2]], p[near[: n // 2]]
    gap = torch.tensor([0.65 * _dims(n, shape)[0] * c["spacing"], 0.0, 0.0], device="cuda", dtype=torch.float64)
    sign[: n - n // 2] = 1.0
    sign[n - n // 2:] = -1.0
    return torch.cat([a - gap, b + gap]), sign


def _records(c, gen):
    """192-byte particle records as an f32 CUDA tensor [n, 48]."""
    n, dx, size = c["n"], c["size"] / c["res"], c["size"]
    p, sign = _positions(c, gen)
    ref = c.get("mode", "config") == "reference"
    centre = torch.full((3,), 0.5 * size, device="cuda", dtype=torch.float64)
    if c.get("collider") == "terrain":
        # the slab's lower side meets the terrain (heights 0.2 to 0.3 of the domain)
        centre[1] = 0.27 * size + 0.5 * _dims(n, "slab")[1] * c["spacing"] * dx
    rec = torch.zeros((n, 48), device="cuda")
    rec[:, 0:3] = (p * dx + centre).float()
    rec[:, 3] = 1.0
    vel = 0.05 * torch.randn((n, 3), generator=gen, device="cuda")
    vel[:, 2 if ref else 1] -= 1.0
    vel[:, 0] += 2.0 * sign.float()
    rec[:, 4:7] = vel
    rec[:, 7] = DENSITY * (c["spacing"] * dx) ** 3
    for k in (0, 5, 10):
        rec[:, 8 + k] = 1.0
        rec[:, 20 + k] = 1.0
    if c.get("strain", 0.0):
        for col in range(3):
            rec[:, 8 + 4 * col: 11 + 4 * col] += c["strain"] * torch.randn((n, 3), generator=gen, device="cuda")
    if c.get("method") == "pbmpm":
        rec[:, 32:35] = vel * c["dt"]             # PBMPM transfers the displacement
    if c.get("order") == "random":
        rec = rec[torch.randperm(n, generator=gen, device="cuda")]
    return rec.contiguous()


def _scale(dx):
    """Fixed-point scale: a power of two that leaves a factor 40 above a cell full of snow."""
    return 2.0 ** math.floor(math.log2(5e7 / (DENSITY * dx ** 3)))


def _mesh(c):
    size = c["size"]
    if c["collider"] == "terrain":
        v, f = pkg.scenes.fbm_terrain(256, 0.1, 2)
        return v * np.float32(size), f
    if c["collider"] == "box":
        s = pkg.scenes.icosphere(3, 0.1 * size, (0.5 * size, 0.1 * size, 0.5 * size))
        return pkg.scenes.merge_meshes(pkg.scenes.box_mesh((0, 0, 0), (size,) * 3), s)
    return None


def _constants(c):
    dx = c["size"] / c["res"]
    over = dict(n_iter=c["n_iter"], force_divisor=float(c["n_iter"]))
    return pkg.scenes.config_params(dx, **over) if c["mode"] == "config" else pkg.scenes.reference_params(**over)


def _touch(c):
    if not c["interaction"]:
        return None
    return {"pos": [0.5 * c["res"]] * 3, "strength": 40.0, "radius": 0.15 * c["res"], "mode": 0}


def _uniforms(c, mesh=None):
    return pkg.scenes.make_uniforms([0.0] * 3, [c["size"]] * 3, (c["res"],) * 3, c["dt"],
                                    _scale(c["size"] / c["res"]), mesh=mesh, interaction=_touch(c))


def _params(d):
    p = pkg.default_params()
    for k, v in d.items():
        if k == "gravity":
            p.gravity[:] = [float(x) for x in v]
        else:
            setattr(p, k, v)
    return p


def _batch_specs(c, seed):
    """Scenes of log-uniform particle counts, blocks and balls, two grid resolutions, each its own material."""
    rng = np.random.default_rng(1000 + c["scenes"] + c["lo"])     # the sizes are the case's, the state is the seed's
    out = []
    for _ in range(c["scenes"]):
        s = _sim("", n=int(math.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"])))),
                 res=int(rng.choice([64, 128])), spacing=0.5, shape=str(rng.choice(["block", "balls"])), dt=c["dt"],
                 substeps=c["substeps"])
        s["young"], s["theta_c"] = float(rng.uniform(5e4, 3e5)), float(rng.uniform(1.5e-2, 3.5e-2))
        if _cells(s["n"], 0.5, s["shape"]) > 0.75 * s["res"]:
            s["res"] = 128
        out.append(s)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return out, [_records(s, gen) for s in out]


def _torus(c, seed):
    rng = np.random.default_rng(seed)
    u, v = np.meshgrid(np.arange(c["u"]), np.arange(c["v"]), indexing="ij")
    big, small = 2.0 + 0.2 * rng.random(), 0.8 + 0.2 * rng.random()
    a, b = 2 * np.pi * u / c["u"], 2 * np.pi * v / c["v"]
    r = small * (1.0 + 0.15 * np.sin(3 * a + 6.0 * rng.random()))
    p = np.stack([(big + r * np.cos(b)) * np.cos(a), (big + r * np.cos(b)) * np.sin(a), r * np.sin(b)], -1)
    verts = p.reshape(-1, 3).astype(np.float32)
    i, j = u.ravel(), v.ravel()
    i1, j1 = (i + 1) % c["u"], (j + 1) % c["v"]
    q = [x * c["v"] + y for x, y in ((i, j), (i1, j), (i1, j1), (i, j1))]
    return verts, np.concatenate([np.stack([q[0], q[1], q[2]], 1), np.stack([q[0], q[2], q[3]], 1)]).astype(np.uint32)


def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if c["kind"] == "batch":
        sims, recs = _batch_specs(c, seed)
        specs = []
        for s, r in zip(sims, recs):
            prm = pkg.scenes.config_params(1.0 / s["res"], youngs_modulus=s["young"], theta_c=s["theta_c"])
            specs.append(pkg.scenes.SceneSpec("scene", _uniforms(s), prm, r.cpu().numpy().view(pkg.PARTICLE_DTYPE)
                                              .reshape(-1), 0, c["substeps"], None, (s["res"],) * 3))
        batch = pkg.GpuMpmBatch(specs)
        start = torch.cat(recs)
        state = dict(c=c, mpm=batch.mpm, pipe=batch, start=start, out=torch.empty_like(start),
                     method=pkg.GpuSimulationMethodType.ExplicitMpm)
        torch.cuda.synchronize()
        return state
    if c["kind"] == "scatter":
        verts, faces = _torus(c, seed)
        mpm = pkg.GpuMpmBufferManager(n_particles=c["n"])
        init = pkg.GpuParticleInitializePipelineManager(
            mpm_manager=mpm, mesh_manager=pkg.GpuMeshBufferManager(vertices=verts, indices=faces),
            uniforms_manager=pkg.GpuUniformsBufferManager())
        return dict(c=c, mpm=mpm, init=init, out=torch.empty((c["n"], 48), device="cuda"))
    if c["kind"] in ("volumetric", "surface"):
        c = _sim(**{"name": "", **c})
        start = _records(c, gen)
        u = _uniforms(c)
        u.write_time(seed & 0xFFFF)
        mpm = pkg.GpuMpmBufferManager(n_particles=c["n"])
        state = dict(c=c, mpm=mpm)
        if c["kind"] == "volumetric":
            s = c["size"]
            u.write_view_proj_inv_mat(pkg.scenes.camera_inv_view_proj(
                (1.6 * s, -0.5 * s, 0.9 * s), (0.5 * s, 0.5 * s, 0.3 * s), c["width"], c["height"]))
            vol = pkg.GpuVolumetricBufferManager(grid_resolution=(c["res"],) * 3,
                                                 screen_dims=(c["width"], c["height"]))
            state.update(vol=vol, view=pkg.GpuVolumetricRenderPipelineManager(mpm_manager=mpm, volumetric_manager=vol))
        else:
            m = int(c["res"] // 2 * c["mc_scale"])
            mc = pkg.GpuMarchingCubesBufferManager(grid_resolution=(c["res"],) * 3, mc_grid_resolution=(m,) * 3,
                                                   max_vertices=2_000_000)
            state.update(mc=mc, view=pkg.GpuMarchingCubesRenderPipelineManager(mpm_manager=mpm, mc_manager=mc))
        state["pipe"] = pkg.GpuMpmPipelineManager(mpm_manager=mpm, uniforms_manager=u, params=_params(_constants(c)))
        torch.cuda.synchronize()
        mpm.write_particles_device(start.data_ptr(), c["n"])
        mpm.sync()
        return state
    start = _records(c, gen)
    out = torch.empty_like(start)
    torch.cuda.synchronize()
    if c["kind"] == "noalloc":
        return dict(c=c, start=start, out=out, uniforms=_uniforms(c).bytes(), params=_params(_constants(c)),
                    method=0 if c["method"] == "explicit" else 1)
    mesh = _mesh(c)
    mpm = pkg.GpuMpmBufferManager(n_particles=c["n"])
    col = pkg.GpuColliderBufferManager(vertices=mesh[0], indices=mesh[1]) if mesh is not None else None
    pipe = pkg.GpuMpmPipelineManager(mpm_manager=mpm, uniforms_manager=_uniforms(c, mesh), collider_manager=col,
                                     params=_params(_constants(c)))
    t = pkg.GpuSimulationMethodType
    return dict(c=c, mpm=mpm, pipe=pipe, start=start, out=out,
                method=t.ExplicitMpm if c["method"] == "explicit" else t.Pbmpm)


# ----------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------
def _get(s):
    """The records into the caller's device buffer, on the handle's stream."""
    lib = pkg.load()
    pkg._lib.check(lib.mpm_get_particles(s["mpm"].handle, ctypes.c_void_p(s["out"].data_ptr()), s["out"].shape[0], 1),
                   s["mpm"].handle)
    return s["out"]


def run(s):
    kind = s["c"]["kind"]
    if kind in ("step", "batch"):
        s["mpm"].write_particles_device(s["start"].data_ptr(), s["start"].shape[0])
        s["pipe"].step(s["method"], s["c"]["substeps"])
        return _get(s)
    if kind == "noalloc":
        s["out"].copy_(s["start"])
        rc = pkg.load().mpm_step_noalloc(0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
                                         ctypes.c_void_p(s["out"].data_ptr()), s["c"]["n"], s["method"], s["uniforms"],
                                         len(s["uniforms"]), ctypes.byref(s["params"]), None, 0, 0, None, 0, None, None,
                                         0)
        if rc:
            raise RuntimeError(f"mpm_step_noalloc: {rc}")
        return s["out"]
    if kind == "scatter":
        s["init"].add_dispatch(n_particles=s["c"]["n"])
        return _get(s)
    if kind == "volumetric":
        s["view"].add_prerender_passes()
        v = s["vol"]
        return dict(mass=v.mass_grid, image=v.output, depth=v.depth, color=v.color)
    count = s["view"].add_mesh_generation_pass()
    return dict(density=s["mc"].density_grid, vertices=s["mc"].vertices[:count])


# ----------------------------------------------------------------------
# what one pass cannot do without
# ----------------------------------------------------------------------
def _flops(n, method, n_iter):
    """Operations of one substep: a 27-cell gather or scatter is about 27 x 25, a 3x3 inverse, product or polar
    step about 45 each."""
    if method == "explicit":
        return n * (2 * 27 * 30 + 1200)
    return n * ((n_iter + 1) * 27 * 50 + n_iter * 900)


def work(case):
    c = case
    if c["kind"] in ("step", "noalloc"):
        return dict(bytes=2 * 192.0 * c["n"], flops=float(_flops(c["n"], c["method"], c["n_iter"]) * c["substeps"]))
    if c["kind"] == "batch":
        rng = np.random.default_rng(1000 + c["scenes"] + c["lo"])
        mean = (c["hi"] - c["lo"]) / math.log(c["hi"] / c["lo"]) if c["hi"] > c["lo"] else c["lo"]
        n = mean * c["scenes"]
        return dict(bytes=2 * 192.0 * n, flops=float(_flops(n, "explicit", 0) * c["substeps"]))
    if c["kind"] == "volumetric":
        pixels = c["width"] * c["height"]
        return dict(bytes=16.0 * c["n"] + 4.0 * c["res"] ** 3 + 24.0 * pixels, flops=60.0 * c["n"] + 8000.0 * pixels)
    if c["kind"] == "surface":
        d = (c["res"] // 2) ** 3
        m = d * c["mc_scale"] ** 3
        return dict(bytes=16.0 * c["n"] + 4.0 * d, flops=60.0 * c["n"] + 20.0 * m)
    # scatter: a candidate and the triangles over its point, a jitter of 18 noise values
    return dict(bytes=192.0 * c["n"] + 96.0 * c["u"] * c["v"], flops=c["n"] * 6000.0)


# ----------------------------------------------------------------------
# the same results in 64 bits
# ----------------------------------------------------------------------
def _eye(n):
    return torch.eye(3, dtype=torch.float64, device="cuda").expand(n, 3, 3)


def _polar(F):
    R = F
    for _ in range(4):
        R = 0.5 * (R + torch.linalg.inv(R).transpose(1, 2))
    return R


class _Grid:
    """Dense grid sums in f64; offsets beyond the grid are dropped."""

    def __init__(self, c, pos, dx):
        self.res = c["res"]
        self.cell = torch.trunc(pos / dx).long()
        f = pos / dx - self.cell
        self.f = f
        self.w = [0.5 * (1 - f) ** 2, 0.75 - (f - 0.5) ** 2, 0.5 * f ** 2]
        self.dw = [f - 1.0, -2.0 * (f - 0.5), f]

    def nodes(self):
        for oz in range(3):
            for oy in range(3):
                for ox in range(3):
                    o = torch.tensor([ox - 1, oy - 1, oz - 1], device="cuda")
                    g = self.cell + o
                    ok = ((g >= 0) & (g < self.res)).all(1)
                    idx = (g[:, 2] * self.res + g[:, 1]) * self.res + g[:, 0]
                    w = [self.w[ox][:, 0], self.w[oy][:, 1], self.w[oz][:, 2]]
                    d = [self.dw[ox][:, 0], self.dw[oy][:, 1], self.dw[oz][:, 2]]
                    grad = torch.stack([d[0] * w[1] * w[2], w[0] * d[1] * w[2], w[0] * w[1] * d[2]], 1)
                    yield idx, ok, (w[0] * w[1] * w[2])[:, None], grad, o - self.f + 0.5, g


def _scatter_add(n_cells, nodes, value):
    grid = torch.zeros((n_cells, 3), dtype=torch.float64, device="cuda")
    for idx, ok, w, grad, off, g in nodes:
        grid.index_add_(0, idx[ok], value(w, grad, off, g)[ok])
    return grid


def _simulate(c, prm, rec):
    """The MPM substeps of a scene without collider contact, in f64: rec [n, 48] -> [n, 48]."""
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    n, res, dt = rec.shape[0], c["res"], f32(c["dt"])
    dx = f32(c["size"] / res)
    r = rec.double()
    pos, vel, mass = r[:, 0:3].clone(), r[:, 4:7].clone(), r[:, 7:8].clone()
    cols = lambda a: r[:, a:a + 12].view(n, 3, 4)[:, :, :3].transpose(1, 2).clone()  # noqa: E731
    Fe, Fp, dxp, D = cols(8), cols(20), r[:, 32:35].clone(), cols(36)
    gravity = torch.tensor([f32(x) for x in prm["gravity"]], device="cuda", dtype=torch.float64)
    lo, hi = f32(1.0 - prm["theta_c"]), f32(1.0 + prm["theta_s"])
    young, nu = prm["youngs_modulus"], prm["poissons_ratio"]
    mu0, la0 = young / (2 * (1 + nu)), young * nu / ((1 + nu) * (1 - 2 * nu))
    pb = c["method"] == "pbmpm"
    touch = _touch(c)
    k = torch.arange(res ** 3, device="cuda")
    cells = [k % res, (k // res) % res, k // (res * res)]

    def boundary(v):
        if prm["boundary_mode"] != 1:
            return v
        b = prm["bc_cells"]
        for a in range(3):
            v[:, a] = torch.where((cells[a] < b) & (v[:, a] < 0) | (cells[a] >= res - b) & (v[:, a] > 0), 0.0, v[:, a])
        v[cells[prm["ground_axis"]] < b] = 0.0
        return v

    def force(g):
        if touch is None:
            return gravity / prm["force_divisor"]
        d = g.double() - torch.tensor(touch["pos"], device="cuda", dtype=torch.float64)
        dist = d.norm(dim=1, keepdim=True)
        pd = torch.where(dist > 1e-3, d / dist.clamp_min(1e-30),
                         torch.tensor([0.0, 0.0, 1.0], device="cuda", dtype=torch.float64))
        push = pd * touch["strength"] * (1 - (dist / touch["radius"]) ** 2)
        return (gravity + torch.where(dist < touch["radius"], push, 0.0)) / prm["force_divisor"]

    for _ in range(c["substeps"]):
        G = _Grid(c, pos, dx)
        m = _scatter_add(res ** 3, G.nodes(), lambda w, grad, off, g: (w * mass).expand(-1, 3))
        rm = torch.where(m > 0, 1.0 / m.clamp_min(1e-300), 0.0)
        if not pb:
            e = torch.exp(f32(prm["hardening_explicit"]) * (1 - torch.linalg.det(Fp)))[:, None, None]
            J = torch.linalg.det(Fe)[:, None, None]
            P = 2 * mu0 * e * (Fe - _polar(Fe)) + la0 * e * (J - 1) * J * torch.linalg.inv(Fe).transpose(1, 2)
            M = -(mass / prm["density"])[:, :, None] * P.transpose(1, 2)
            mom = _scatter_add(res ** 3, G.nodes(), lambda w, grad, off, g:
                               w * mass * vel + (M @ (grad / dx)[:, :, None])[:, :, 0] * dt)
            v = boundary(torch.where(m > 0, mom * rm + gravity * dt, 0.0))
        else:
            Fei = torch.linalg.inv(Fe)
            relax = (1 - 0.5 * torch.exp(-f32(prm["hardening_pbmpm"]) / torch.linalg.det(Fp)))[:, None, None]
        for it in range(prm["n_iter"] if pb else 1):
            if pb:
                Ft = (_eye(n) + D) @ Fe
                R = _polar(Ft)
                vs = torch.linalg.det(Ft).abs()[:, None, None] ** prm["pbmpm_volume_exponent"]
                b = f32(prm["pbmpm_blend"])
                D = D + relax * ((b * vs + (1 - b)) * R @ Fei - _eye(n) - D)
                mom = _scatter_add(res ** 3, G.nodes(), lambda w, grad, off, g:
                                   w * mass * (dxp + (D @ off[:, :, None])[:, :, 0]) / dt + force(g) * w * mass * dt)
                v = boundary(mom * rm)
            vel = torch.zeros_like(vel)
            D = torch.zeros_like(D)
            for idx, ok, w, grad, off, g in G.nodes():
                vc = torch.where(ok[:, None], v[idx.clamp(0, res ** 3 - 1)], 0.0)
                vel += w * vc
                D += vc[:, :, None] * (w * off if pb else grad)[:, None, :]
            D *= dt * (4.0 if pb else 1.0)
            dxp = vel * dt
        pos = pos + dxp
        Fe = (_eye(n) + D) @ Fe
        R = _polar(Fe)
        sg = torch.diagonal(R.transpose(1, 2) @ Fe, dim1=1, dim2=2)
        act = ((sg < lo) | (sg > hi)).any(1)[:, None, None]
        Fn = R * sg.clamp(lo, hi)[:, None, :]
        Fp = torch.where(act, torch.linalg.inv(Fn) @ Fe @ Fp, Fp)
        Fe = torch.where(act, Fn, Fe)
        for a in range(3):
            out = (pos[:, a] < 0) | (pos[:, a] >= c["size"])
            vel[:, a] = torch.where(out, vel[:, a] * prm["restitution"], vel[:, a])
            dxp[:, a] = torch.where(out, dxp[:, a] * prm["restitution"], dxp[:, a])
        pos = pos.clamp(0.0, c["size"])
    o = torch.zeros((n, 48), dtype=torch.float64, device="cuda")
    o[:, 0:3], o[:, 3], o[:, 4:7], o[:, 7:8], o[:, 32:35] = pos, r[:, 3], vel, mass, dxp
    for a, X in ((8, Fe), (20, Fp), (36, D)):
        o[:, a:a + 12].view(n, 3, 4)[:, :, :3] = X.transpose(1, 2)
    return o


def exact(case, seed):
    c = case
    if c["kind"] in ("step", "noalloc"):
        # no closed form of the mesh contact: it follows the tree's traversal.  (The box case's walls and obstacle
        # are out of the snow's reach within a pass.)
        if c["collider"] == "terrain":
            return None
        rec = _records(c, torch.Generator(device="cuda").manual_seed(seed))
        return _simulate(c, _constants(c), rec)
    if c["kind"] == "batch":
        sims, recs = _batch_specs(c, seed)
        return torch.cat([_simulate(s, pkg.scenes.config_params(1.0 / s["res"], youngs_modulus=s["young"],
                                                                theta_c=s["theta_c"]), r) for s, r in zip(sims, recs)])
    # scatter, ray march and marching cubes branch on f32 comparisons (a candidate's ray parity, a dense sample, the
    # isovalue): the same run in 64 bits takes other branches and is another answer, not a more exact one
    return None
