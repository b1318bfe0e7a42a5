"""The ordering at the sizes where its kernels change: the radix sort around a short tile
(1,024 pairs) and the switch to long tiles (2^22 pairs), and the incremental ordering of
small systems and of mover counts around a staged tile (1,024) and the brute-force limit
(8,192), against the full sort."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from anisotropicelastoplasticity_gb300 import HybridSolver, capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bits", [(1023, 9), (1024, 17), (1025, 24), (2047, 31), ((1 << 22) - 1, 24), (1 << 22, 27),
                                    ((1 << 22) + 1, 28)])
def test_sort_pairs_around_tiles(n, bits):
    import torch

    lib = capi.load()
    g = torch.Generator().manual_seed(n)
    keys = torch.randint(0, 1 << min(bits, 30), (n,), generator=g, dtype=torch.int64)
    keys[::3] = keys[0]  # long runs of equal keys
    k = keys.to(torch.int32).cuda()
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    ko, vo = torch.empty_like(k), torch.empty_like(v)
    size = lib.aep_sort_pairs_temp_bytes(n, bits)
    temp = torch.empty(size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    st = lib.aep_sort_pairs(C.c_void_p(k.data_ptr()), C.c_void_p(ko.data_ptr()), C.c_void_p(v.data_ptr()),
                            C.c_void_p(vo.data_ptr()), n, bits, C.c_void_p(temp.data_ptr()), size, None)
    assert st == capi.AEP_OK
    torch.cuda.synchronize()
    order = np.argsort(keys.numpy(), kind="stable")
    assert np.array_equal(vo.cpu().numpy(), order)
    assert np.array_equal(ko.cpu().numpy(), keys.numpy()[order])


@pytest.mark.parametrize("n,moved", [(1, 0.0), (31, 0.1), (700, 0.05), (4095, 0.2), (4096, 0.3), (40000, 0.025), (40000, 0.026),
                                     (60000, 0.13), (60000, 0.14)])
def test_incremental_ordering_of_any_size(n, moved):
    """Between two steps a share of the particles is put elsewhere: the ordering (movers
    merged, or a full sort) against full_sort = 1, the same grid mass bit for bit and the
    particles up to the FP32 rounding of the per-run sums."""
    res = {}
    for full in (0, 1):
        sc = scenes.snow_block(n=n, res=32, seed=5)
        sc.params.full_sort = full
        sc.params.reorder_interval = 1
        s = HybridSolver(sc.particles, sc.grid, sc.params)
        s.set_level_set(sc.levelset)
        s.init_volumes()
        s.step(sc.dt)
        st = s.get_particles()
        rng = np.random.default_rng(7)
        pick = rng.choice(n, size=int(moved * n), replace=False)
        ps = sc.particles
        ps.positions = st["positions"].copy()
        ps.positions[pick, 0] += 3.0 / 32
        ps.velocities, ps.affine_momenta = st["velocities"], st["affine_momenta"]
        ps.elastic_deformation_gradients, ps.volumes = st["elastic_deformation_gradients"], st["volumes"]
        s.set_particle_system(ps)
        s.step(sc.dt)
        info = s.stats()
        if not full:
            want = len(pick)  # and the few particles that crossed a cell in the first step
            if want > min(8192, n // 4):
                assert info["sort_movers"] == -1
            else:
                assert want <= info["sort_movers"] <= want + 0.02 * n + 8
        res[full] = (s.get_particles(), info["total_mass"])
        s.close()
    a, b = res[0][0], res[1][0]
    assert res[0][1] == res[1][1]
    assert np.abs(a["positions"] - b["positions"]).max() < 1e-6
    assert np.abs(a["velocities"] - b["velocities"]).max() <= 1e-4 * max(np.abs(b["velocities"]).max(), 1e-9)
