"""aep_solve at a step that overflows the fixed-point accumulators: whether the steps are
waited for one by one (with a callback) or launched ahead, that step is the last one."""
from __future__ import annotations

import numpy as np
import pytest

from anisotropicelastoplasticity_gb300 import AepError, HybridSolver, capi

from .parity_util import small_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfl,gravity", [(0.05, 1e6), (0.05, 2e5), (1.0, 1e6)])
def test_no_step_follows_an_overflow(cfl, gravity):
    """A snow block falling under a large acceleration: with 50 momentum bits its nodes
    (about twelve particles each) overflow 2^61 near 170 m/s, in the first or a later step."""
    res = []
    for callback in (lambda d: False, None):
        sc = small_scene("snow")
        sc.params.momentum_bits = 50
        sc.params.gravity[2] = -gravity
        s = HybridSolver(sc.particles, sc.grid, sc.params)
        s.set_level_set(sc.levelset)
        with pytest.raises(AepError) as e:
            s.solve(cfl, 1.0, callback=callback, max_steps=400)
        assert e.value.status == capi.AEP_OVERFLOW
        st, grid = s.stats(), s.get_grid()
        assert st["overflow"] and st["steps"] == s.solve_state()["steps"] + 1
        assert st["active_nodes"] == int((grid["masses"] > 0).sum())
        res.append((s.solve_state(), st, s.get_particles(), grid))
        s.close()
    a, b = res
    assert a[0] == b[0] and a[1] == b[1]
    for k in (2, 3):
        for name in a[k]:
            np.testing.assert_array_equal(a[k][name], b[k][name])
