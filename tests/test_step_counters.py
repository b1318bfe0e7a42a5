"""The counters of consecutive steps, kept in two buffers in turn: after every whole or
partial step they are that step's alone."""
from __future__ import annotations

import pytest

from anisotropicelastoplasticity_gb300 import HybridSolver, capi

from .parity_util import small_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interval", [1, 4])
def test_counters_are_of_the_last_step(interval):
    sc = small_scene("sand")
    sc.params.reorder_interval = interval
    s = HybridSolver(sc.particles, sc.grid, sc.params)
    s.set_level_set(sc.levelset)
    s.init_volumes()
    P, F, G = capi.AEP_STAGE_P2G, capi.AEP_STAGE_FORCES, capi.AEP_STAGE_GRID
    mass, orderings = None, s.stats()["orderings"]
    for stage in (None, None, P, None, P, P, F, None, G, None, None, None, None, None, None):
        if stage is None:
            s.step(sc.dt)
        else:
            s.step_stage(sc.dt, stage)
        st = s.stats()
        mass = st["total_mass"] if mass is None else mass
        assert st["total_mass"] == mass  # one step's sums, exact
        assert st["active_nodes"] == int((s.get_grid()["masses"] > 0).sum())
        assert st["overflow"] == 0 and st["out_of_domain"] == 0
        # movers are counted in the steps that order the particles, and only there
        assert st["orderings"] > orderings or st["sort_movers"] == 0
        orderings = st["orderings"]
    s.close()
