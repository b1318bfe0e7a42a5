"""P2G and the force scatter of small systems, where two or four warps share a batch of 32
particles: the grid against the FP64 oracle at particle counts around a batch, a thread
block and the switches of each kernel (152 SMs: P2G at 24,320 and 48,640 particles, the
force scatter at 29,184 and 58,368)."""
from __future__ import annotations

import numpy as np
import pytest

from anisotropicelastoplasticity_gb300 import capi, scenes

from .parity_util import make_pair, mass_weighted_rel, max_rel, perturbed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 33, 159, 161, 24320, 24321, 29184, 29185, 48640, 48641, 58368, 58369])
def test_shared_batches(n):
    sc = perturbed(scenes.sand_column(n=n, res=32, seed=n), seed=n + 1)
    gpu, orc = make_pair(sc)
    orc.init(volumes=False)
    gpu.step_stage(sc.dt, capi.AEP_STAGE_P2G)
    g, o = gpu.get_grid(), orc.get_grid()
    # the bounds of the P2G and force parity tests (FP32 against FP64)
    assert max_rel(g["masses"], o["masses"]) < 2e-6
    assert abs(g["masses"].sum() - o["masses"].sum()) / o["masses"].sum() < 1e-6
    assert mass_weighted_rel(g["velocities"], o["velocities"], o["masses"]) < 2e-5
    gpu.close()
    gpu, orc = make_pair(sc)
    orc.init(volumes=False)
    gpu.step_stage(sc.dt, capi.AEP_STAGE_FORCES)
    orc.step(sc.dt, stage=capi.AEP_STAGE_FORCES)
    g, o = gpu.get_grid(), orc.get_grid()
    f = o["forces"] - o["masses"][:, None] * np.array(list(sc.params.gravity))
    assert max_rel(g["forces"], f) < 2e-4
    gpu.close()
