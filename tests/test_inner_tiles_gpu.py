"""Tiles whose halo lies inside the grid and out of the boundary's reach skip the
cells' checks: scenes in a corner of the grid, with both kinds of tiles side by
side, against the oracle, bit for bit, over boundary widths (none, one cell, wider
than the snow), ground axes, tile edges, methods and iteration counts."""
import numpy as np
import pytest

from helpers import GpuScene, compare_states, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n_iter,edge", [("explicit", 3, 0), ("explicit", 3, 8), ("explicit", 3, 16), ("pbmpm", 1, 8),
                                              ("pbmpm", 3, 0), ("pbmpm", 3, 8), ("pbmpm", 3, 12), ("pbmpm", 2, 16)])
@pytest.mark.parametrize("mode,cells,axis,corner", [(0, 3, 2, "low"), (1, 0, 1, "low"), (1, 1, 0, "high"), (1, 3, 2, "low"),
                                                    (1, 3, 1, "high"), (1, 20, 2, "low")])
def test_corner_scene(gpu, oracle_mod, kind, n_iter, edge, mode, cells, axis, corner):
    spec = gpu.scenes.parity_scene(kind=kind, n_side=24, seed=61, n_iter=n_iter, res=64)
    p = spec.particles["pos"]
    p -= p.min(axis=0) - np.float32(0.4 / 64)        # the snow starts in the grid's first cells
    if corner == "high":
        spec.particles["pos"] = np.float32(1.0) - p
    spec.params.update(boundary_mode=mode, bc_cells=cells, ground_axis=axis)
    g = GpuScene(gpu, spec, tile_edge=edge)
    assert g.step(2) == 0
    got = g.particles()
    g.close()
    o, want = run_oracle(oracle_mod, spec, n_steps=2)
    o.close()
    compare_states(got, want)
