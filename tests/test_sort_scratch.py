"""The radix sort's scratch is sized once for the largest number of pairs and then serves
every smaller one, across the switch from long tiles (from 2^22 pairs) to short ones."""
from __future__ import annotations

import numpy as np
import pytest

from anisotropicelastoplasticity_gb300 import HybridSolver, capi, scenes


@pytest.mark.parametrize("bits", [1, 8, 27, 32])
def test_scratch_size_never_falls_as_n_grows(bits):
    lib = capi.load()
    rng = np.random.default_rng(bits)
    big = 1 << 22
    n = np.concatenate([np.arange(0, 5000), big + np.arange(-3000, 3000), np.arange(big // 2, 2 * big, 9973),
                        np.unique(np.exp(rng.uniform(0, np.log(2 ** 30 - 1), 2000)).astype(np.int64))])
    size = [lib.aep_sort_pairs_temp_bytes(int(k), bits) for k in np.sort(n)]
    assert min(size) > 0 and np.all(np.diff(size) >= 0)


@pytest.mark.gpu
@pytest.mark.parametrize("largest,n", [(1 << 22, (1 << 22) - 1), (4300000, 4190000), (4300000, 1000)])
def test_sort_in_scratch_of_a_larger_size(largest, n):
    import torch

    lib = capi.load()
    keys = torch.randint(0, 1 << 27, (n,), generator=torch.Generator().manual_seed(n), dtype=torch.int32)
    k, v = keys.cuda(), torch.arange(n, dtype=torch.int32, device="cuda")
    ko, vo = torch.empty_like(k), torch.empty_like(v)
    size = lib.aep_sort_pairs_temp_bytes(largest, 27)
    temp = torch.empty(size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert lib.aep_sort_pairs(k.data_ptr(), ko.data_ptr(), v.data_ptr(), vo.data_ptr(), n, 27, temp.data_ptr(), size,
                              None) == capi.AEP_OK
    torch.cuda.synchronize()
    order = np.argsort(keys.numpy(), kind="stable")
    np.testing.assert_array_equal(vo.cpu().numpy(), order)
    np.testing.assert_array_equal(ko.cpu().numpy(), keys.numpy()[order])


@pytest.mark.gpu
@pytest.mark.parametrize("full", [0, 1])
def test_fewer_particles_on_the_same_handle(full):
    """A handle that held 4,300,000 particles takes 4,190,000 and steps as a fresh one."""
    res = {}
    for sizes in ((4300000, 4190000), (4190000,)):
        s = None
        for n in sizes:
            sc = scenes.snow_block(n=n, res=64, seed=3)
            if s is None:
                sc.params.full_sort = full
                sc.params.reorder_interval = 1
                s = HybridSolver(sc.particles, sc.grid, sc.params)
                s.set_level_set(sc.levelset)
            else:
                s.set_particle_system(sc.particles)
            for _ in range(2):
                s.step(sc.dt)
        st = s.stats()
        res[len(sizes)] = (s.get_particles(), st["total_mass"], st["sort_movers"])
        s.close()
    a, b = res[2], res[1]
    assert a[1:] == b[1:]
    for k in a[0]:
        np.testing.assert_array_equal(a[0][k], b[0][k])
