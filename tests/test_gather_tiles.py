"""The grid gathers of the force scatter and G2P from their shared-memory tiles: one step
against the FP64 oracle at particle counts around a thread block (64 or 128 particles), at
the switch between the two block forms of G2P, with stencils inside and outside the tile
(1.5 particles per cell: a block's particles lie in many node blocks), with nodes
whose velocity before friction differs, and at the grid's border."""
from __future__ import annotations

import numpy as np
import pytest

from anisotropicelastoplasticity_gb300 import capi, scenes
from anisotropicelastoplasticity_gb300.solver import LevelSet

from .parity_util import make_pair, max_rel, perturbed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,where", [(n, w) for n in (1, 63, 64, 65, 127, 129, 700) for w in ("box", "border")] +
                         [(38912, "border"), (38913, "border")])
def test_step_around_block_sizes(n, where):
    sc = scenes.sand_column(n=n, res=32, seed=n)
    rng = np.random.default_rng(n)
    x = sc.particles.positions
    if where == "border":  # at the low-x wall and on the ground: cut stencils, sticking nodes
        x[:, 0] = 0.003 + 0.06 * rng.random(n)
        x[:, 2] = 0.004 + 0.1 * rng.random(n)
        sc.levelset = LevelSet.ground(0.04) | LevelSet.sphere([0.3, 0.5, 0.0], 0.12)
    else:  # 1.5 particles per cell, half of the box below the ground's surface
        side = (n / 1.5) ** (1.0 / 3.0) / 32
        x[:] = 0.5 + side * (rng.random((n, 3)) - 0.5)
        sc.levelset = LevelSet.ground(0.5)
    sc.particles.material[::3] = capi.AEP_SNOW
    sc = perturbed(sc, seed=n + 1)
    gpu, orc = make_pair(sc)
    gpu.step(sc.dt)
    orc.init(volumes=False)
    orc.step(sc.dt)
    g, o = gpu.get_particles(), orc.get_particles()
    # FP32 against FP64, the bounds of the one-step parity suite at this resolution
    assert np.abs(g["positions"] - o["positions"]).max() < 5e-7
    assert max_rel(g["velocities"], o["velocities"]) < 1e-4
    assert np.abs(g["elastic_deformation_gradients"] - o["elastic_deformation_gradients"]).max() < 2e-6
    scale = max(np.abs(o["affine_momenta"]).max(), np.abs(o["velocities"]).max() * float(sc.grid.h.min()))
    assert np.abs(g["affine_momenta"] - o["affine_momenta"]).max() / scale < 1e-3
    assert np.abs(g["plastic"] - o["plastic"]).max() < 2e-6
    gpu.close()
