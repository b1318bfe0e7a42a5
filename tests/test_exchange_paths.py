"""Readbacks and uploads of any selection of fields, by records or in the caller's order: around
the limits between the two, and at sizes whose columns do not begin on whole lines or whose
last blocks are short.  Both convert the same values, so device, page-locked and pageable
arrays agree bit for bit with the values given."""
from __future__ import annotations

import numpy as np
import pytest

from anisotropicelastoplasticity_gb300 import HybridSolver, capi, scenes

from .test_device_exchange import _ptr, _set, _state

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "B", "Fe", "Fp", "vol", "plastic")
VALUES = (3, 3, 9, 9, 9, 1, 1)


def _make(kind, k):
    import torch

    t = torch.full((k,), -7.0, dtype=torch.float64, device="cuda" if kind == "device" else "cpu")
    return t.pin_memory() if kind == "page-locked" else t


@pytest.mark.parametrize("n", [1, 15, 17, 127, 129, 1009, 1025, 32767, 32768, 39999, 40000, 99999, 100001, 263169])
def test_particles_by_any_fields(n):
    import torch

    sc = scenes.snow_block(n=8, res=32)
    sc.params.track_plastic_F = 1
    s = HybridSolver(None, sc.grid, sc.params)
    s.set_level_set(sc.levelset)
    _set(s, n, _state(n, True, 1))
    s.step(1e-5)  # the device's order is no longer the caller's
    for kind in ("device", "page-locked", "pageable"):
        new = _state(n, True, 3 + len(kind))
        given = [torch.from_numpy(a) for a in new]
        if kind == "device":
            given = [a.cuda() for a in given]
        elif kind == "page-locked":
            given = [a.pin_memory() for a in given]
        torch.cuda.synchronize()
        _set(s, n, given)
        want = [new[i].astype(np.float32).astype(np.float64).reshape(-1) for i in (0, 1, 2, 3, 4, 6, 7)]
        for out in ("device", "page-locked", "pageable"):
            for pick in ((0, 1, 2, 3, 4, 5, 6), (0, 1, 2, 3, 5, 6), (2, 3), (0, 2), (0, 3), (0, 1), (4,), (3, 4), (5, 6)):
                got = [_make(out, VALUES[f] * n) if f in pick else None for f in range(7)]
                torch.cuda.synchronize()
                assert s._lib.aep_get_particles(s._h, n, *[_ptr(a) for a in got]) == capi.AEP_OK
                for f in pick:
                    np.testing.assert_array_equal(got[f].cpu().numpy(), want[f], err_msg=f"{kind} {out} {FIELDS[f]}")
    s.close()


@pytest.mark.parametrize("nside", [3, 33, 223, 225])  # 148,297 and 150,977 items around the limit
def test_mesh_state_by_any_fields(nside):
    import torch

    sc = scenes.cloth_drape(nside=nside, res=32)
    s = HybridSolver(None, sc.grid, sc.params)
    s.set_level_set(sc.levelset)
    s.set_lagrangian_mesh(sc.mesh)
    s.step(1e-6)
    nv, nf = len(sc.mesh.vertex_positions), len(sc.mesh.faces)
    size = [k * (nv if f < 3 else nf) for f, k in enumerate((3, 3, 9, 3, 3, 9, 9))]
    r = np.random.default_rng(nside)
    state = [None] * 7
    for kind in ("device", "page-locked", "pageable"):
        for pick in (range(7), (0, 1, 2), (0, 2), (3, 4, 5, 6), (0, 2, 3, 5, 6), (0, 1, 2, 3, 4, 5), (6,), (1, 4)):
            new = {f: r.random(size[f]) for f in pick}
            given = [torch.from_numpy(new[f]) if f in pick else None for f in range(7)]
            if kind != "pageable":
                given = [a if a is None else a.cuda() if kind == "device" else a.pin_memory() for a in given]
            torch.cuda.synchronize()
            assert s._lib.aep_set_mesh_state(s._h, nv, nf, *[_ptr(a) for a in given]) == capi.AEP_OK
            state = [new.get(f, state[f]) for f in range(7)]  # the first selection is all seven
            for out in ("device", "page-locked", "pageable"):
                for want in (range(7), pick):
                    got = [_make(out, size[f]) if f in want else None for f in range(7)]
                    torch.cuda.synchronize()
                    assert s._lib.aep_get_mesh(s._h, *[_ptr(a) for a in got]) == capi.AEP_OK
                    for f in want:
                        np.testing.assert_array_equal(got[f].cpu().numpy(),
                                                      state[f].astype(np.float32).astype(np.float64))
    s.close()
