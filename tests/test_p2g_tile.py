"""P2G's grid tile at the ends of the grid's rows: particles at the low-x and the high-x wall,
so that the order goes from the last node block of a row to the first of the next one, and
base nodes at every place of a node block."""
from __future__ import annotations

import numpy as np
import pytest

from anisotropicelastoplasticity_gb300 import capi, scenes

from .parity_util import make_pair, mass_weighted_rel, max_rel, perturbed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,res", [(64, 32), (600, 29), (600, 30), (5000, 31), (30000, 32)])
def test_p2g_at_both_walls(n, res):
    sc = scenes.sand_column(n=n, res=res, seed=n)
    rng = np.random.default_rng(n + res)
    x = sc.particles.positions
    x[:] = 0.1 + 0.8 * rng.random((n, 3))
    x[:, 0] = np.where(rng.random(n) < 0.5, 0.004 + 0.1 * rng.random(n), 0.996 - 0.1 * rng.random(n))
    sc = perturbed(sc, seed=n + 1)
    gpu, orc = make_pair(sc)
    gpu.step_stage(sc.dt, capi.AEP_STAGE_P2G)
    orc.init(volumes=False)
    g, o = gpu.get_grid(), orc.get_grid()
    # the bounds of the P2G parity test (FP32 against FP64)
    assert max_rel(g["masses"], o["masses"]) < 2e-6
    assert mass_weighted_rel(g["velocities"], o["velocities"], o["masses"]) < 2e-5
    gpu.close()
