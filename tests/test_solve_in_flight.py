"""aep_solve launches a step before the one ahead of it has been read back, where no callback
is set: the same steps, clock, statistics and state as with a callback, which waits for every
step, at ends by time, by the step limit, and around the ends of frames."""
from __future__ import annotations

import numpy as np
import pytest

from anisotropicelastoplasticity_gb300 import AepError, HybridSolver, capi

from .parity_util import small_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfl,maxt,max_steps", [(0.05, -1.0, 0), (0.05, 0.0, 1), (0.05, 0.0, 2), (0.05, 0.0, 0), (0.7, 0.0, 0),
                                                (0.7, 0.04, 0), (0.7, 0.04, 11), (6.0, 0.06, 0)])
def test_without_a_callback_as_with_one(cfl, maxt, max_steps):
    res = []
    for callback in (None, lambda d: False):
        sc = small_scene("mixed")
        s = HybridSolver(sc.particles, sc.grid, sc.params)
        s.set_level_set(sc.levelset)
        try:
            s.solve(cfl, maxt, callback=callback, max_steps=max_steps)
            first = s.solve_state()
            s.solve(cfl, maxt, callback=callback, max_steps=3)  # and again from there
            res.append((first, s.solve_state(), s.stats(), s.get_particles()))
        except AepError as e:  # the steps of the last one are too large: both overflow alike
            assert e.status == capi.AEP_OVERFLOW and cfl > 1
            res.append((s.solve_state(), s.stats()["overflow"]))
        s.close()
    a, b = res
    assert a[:3] == b[:3]
    for k in a[3] if len(a) > 3 else ():
        np.testing.assert_array_equal(a[3][k], b[3][k])
