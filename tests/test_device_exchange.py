"""State exchange with arrays in device memory against host arrays (the
caller's order): both convert the same FP64 values, so they agree bit for bit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from anisotropicelastoplasticity_gb300 import HybridSolver, capi, scenes

pytestmark = pytest.mark.gpu


def _state(n, fp, seed):
    """The C-ABI's particle arrays as host arrays: x, v, B, Fe, Fp, m, vol, plastic, material."""
    r = np.random.default_rng(seed)
    f = lambda *s: r.standard_normal(s)  # noqa: E731
    eye = np.eye(3).reshape(9)
    return [0.3 + 0.4 * r.random((3, n)), f(3, n), 1e-3 * f(9, n), eye + 0.01 * f(n, 9),
            eye + 0.01 * f(n, 9) if fp else None, 1e-3 * (1 + r.random(n)), 1e-6 * (1 + r.random(n)), 0.1 * r.random(n),
            (r.random(n) < 0.5).astype(np.uint8)]


def _ptr(a, kind=C.c_double):
    if a is None:
        return None
    addr = a.ctypes.data if isinstance(a, np.ndarray) else a.data_ptr()
    return C.cast(C.c_void_p(addr), C.POINTER(kind))


def _set(s, n, arrs):
    st = s._lib.aep_set_particles(s._h, n, *[_ptr(a) for a in arrs[:8]], _ptr(arrs[8], C.c_uint8))
    assert st == capi.AEP_OK


def _get(s, n, fp, make):
    out = [make(k * n) if k else None for k in (3, 3, 9, 9, 9 if fp else 0, 1, 1)]
    assert s._lib.aep_get_particles(s._h, n, *[_ptr(a) for a in out]) == capi.AEP_OK
    return out


@pytest.mark.parametrize("n,fp,mesh", [(1, False, False), (255, True, False), (257, False, True), (1000, True, True),
                                       (70001, True, False), (2200001, False, False), (4300000, False, False)])
def test_device_arrays_match_host_arrays(n, fp, mesh):
    import torch

    sc = scenes.cloth_drape(nside=9, res=32) if mesh else scenes.snow_block(n=8, res=32)
    sc.params.track_plastic_F = int(fp)
    s = HybridSolver(None, sc.grid, sc.params)
    s.set_level_set(sc.levelset)
    _set(s, n, _state(n, fp, 1))
    if mesh:
        s.set_lagrangian_mesh(sc.mesh)
    s.step(1e-5)  # the device's order is no longer the caller's
    new = _state(n, fp, 2)
    dev = [None if a is None else torch.from_numpy(a).cuda() for a in new]
    torch.cuda.synchronize()
    _set(s, n, dev)  # slot order
    want = [None if a is None else a.astype(np.float32).astype(np.float64).reshape(-1) for a in new]
    snow = new[8] == capi.AEP_SNOW
    plastic = want[7].copy()
    if fp:
        plastic = None  # J_P of snow follows F_P at the next step
    else:
        plastic[snow] = want[7][snow]
    expect = [want[0], want[1], want[2], want[3], want[4], want[6], plastic]
    host = _get(s, n, fp, np.empty)
    on_dev = _get(s, n, fp, lambda k: torch.empty(k, dtype=torch.float64, device="cuda"))
    pinned = _get(s, n, fp, lambda k: torch.empty(k, dtype=torch.float64).pin_memory())
    for w, a, b, c in zip(expect, host, on_dev, pinned):
        if a is None:
            continue
        np.testing.assert_array_equal(a, b.cpu().numpy())
        np.testing.assert_array_equal(a, c.numpy())
        if w is not None:
            np.testing.assert_array_equal(a, w)
    # the same values from host memory (the caller's order) leave the same state
    _set(s, n, new)
    for a, b in zip(host, _get(s, n, fp, np.empty)):
        if a is not None:
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n", [31, 129, 4097])
@pytest.mark.parametrize("want", ["x", "xv", "B", "xF", "vB", "Fq", "FP", "xvBFPVq"])
def test_device_readback_of_some_fields(n, want):
    """Any subset of the fields, by way of records (12 values per item and more) or each on
    its own, gives the values that the host readback gives."""
    import torch

    sc = scenes.snow_block(n=8, res=32)
    sc.params.track_plastic_F = 1
    s = HybridSolver(None, sc.grid, sc.params)
    s.set_level_set(sc.levelset)
    _set(s, n, _state(n, True, 3))
    s.step(1e-5)
    host = _get(s, n, True, np.empty)
    out = [torch.full((k * n,), 7.0, dtype=torch.float64, device="cuda") for k in (3, 3, 9, 9, 9, 1, 1)]
    asked = [o if c in want else None for o, c in zip(out, "xvBFPVq")]
    torch.cuda.synchronize()
    assert s._lib.aep_get_particles(s._h, n, *[_ptr(a) for a in asked]) == capi.AEP_OK
    for a, b, c in zip(host, out, "xvBFPVq"):
        np.testing.assert_array_equal(b.cpu().numpy(), a if c in want else np.full(len(a), 7.0))


def test_device_arrays_bad_mass_is_refused():
    import torch

    sc = scenes.snow_block(n=8, res=32)
    s = HybridSolver(None, sc.grid, sc.params)
    good = _state(300, False, 1)
    _set(s, 300, good)
    bad = [None if a is None else torch.from_numpy(a.copy()).cuda() for a in good]
    bad[5][137] = float("nan")
    torch.cuda.synchronize()
    st = s._lib.aep_set_particles(s._h, 300, *[_ptr(a) for a in bad[:8]], _ptr(bad[8], C.c_uint8))
    assert st == capi.AEP_INVALID_ARG


@pytest.mark.parametrize("nside", [2, 9, 40])
@pytest.mark.parametrize("want", [(0, 1, 2, 3, 4, 5, 6), (0, 3), (2, 6), (3, 4, 5), (6,), (0, 1, 2)])
def test_mesh_state_on_the_device(nside, want):
    """The mesh state from and into device arrays, whole records or single fields, is what the
    host arrays give; fields that are not given keep their values."""
    import torch

    sc = scenes.cloth_drape(nside=nside, res=32)
    s = HybridSolver(None, sc.grid, sc.params)
    s.set_level_set(sc.levelset)
    n = 33
    _set(s, n, _state(n, False, 1))
    s.set_lagrangian_mesh(sc.mesh)
    s.step(1e-5)
    nv, nf = len(sc.mesh.vertex_positions), len(sc.mesh.faces)
    sizes = [3 * nv, 3 * nv, 9 * nv, 3 * nf, 3 * nf, 9 * nf, 9 * nf]

    def get(make, which=range(7)):
        out = [make(k) if f in which else None for f, k in enumerate(sizes)]
        assert s._lib.aep_get_mesh(s._h, *[_ptr(a) for a in out]) == capi.AEP_OK
        return out

    before = get(np.empty)
    on_dev = get(lambda k: torch.empty(k, dtype=torch.float64, device="cuda"), want)
    for f in want:
        np.testing.assert_array_equal(on_dev[f].cpu().numpy(), before[f])
    rng = np.random.default_rng(5)
    new = [(0.3 + 0.4 * rng.random(k)).astype(np.float32).astype(np.float64) for k in sizes]
    dev = [torch.from_numpy(a).cuda() if f in want else None for f, a in enumerate(new)]
    torch.cuda.synchronize()
    assert s._lib.aep_set_mesh_state(s._h, nv, nf, *[_ptr(a) for a in dev]) == capi.AEP_OK
    after = get(np.empty)
    for f in range(7):
        np.testing.assert_array_equal(after[f], new[f] if f in want else before[f])
