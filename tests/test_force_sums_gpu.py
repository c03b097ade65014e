"""The PBMPM force sums that the first transfer forms for the iterations, against
the oracle, bit for bit: gravity along each single axis, several or none, the
interaction force in both modes, every tile edge, one to four iterations, and
scales that are and are not a power of two."""
import numpy as np
import pytest

from helpers import GpuScene, compare_states, run_oracle

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
