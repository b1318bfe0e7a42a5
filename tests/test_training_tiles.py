"""Training at the row counts where its blocks (64 rows) and passes (16,384 rows) begin and
end: the gradient against the oracle, and the Adam update that the last reduction makes
against FP64 Adam on that gradient."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp_oracle as mo

from .test_learned import NP, random_params, random_records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 128, 16384, 16385, 40000])
def test_gradient_and_update_around_blocks(n):
    import torch

    from anisotropicelastoplasticity_gb300.learned import ReturnMapMLP

    rec = random_records(n, seed=n)
    d = torch.from_numpy(rec).cuda()
    torch.cuda.synchronize()
    p = random_params(n + 1)
    m = ReturnMapMLP(seed=0)
    m.set_params(p)
    g, loss = m.gradient(d.data_ptr(), n)
    loss_o, g_o = mo.loss_and_grad(p.astype(np.float64), rec, bf=True)
    assert abs(loss - loss_o) / loss_o < 1e-4 + 2.0 ** -8 / np.sqrt(n)
    go, gg = mo.unpack(g_o), mo.unpack(g.astype(np.float64))
    for name, _ in mo.LAYOUT:
        ref, got = go[name], gg[name]
        if name == "w1t":
            ref, got = ref[:, :7], got[:, :7]
        elif name in ("w4t", "b4"):
            ref, got = ref[:3], got[:3]
        # the gradient test's bound, and one activation of a row (of 64) on the other side
        # of its bfloat16 rounding: 2^-8 / 8 of that row's share
        assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 5e-5 + 2.0 ** -11 / np.sqrt(n), name
    p = m.get_params().astype(np.float64)
    lr = 2e-3
    m.train(d.data_ptr(), n, steps=1, batch=n, lr=lr, lr_final=lr)
    want, _, _ = mo.adam_step(p, g, np.zeros(NP), np.zeros(NP), 1, lr)
    # FP32 update arithmetic: a few units of spacing of the parameter, or 1e-5 of the step
    bound = 4 * np.spacing(np.abs(want).astype(np.float32)).astype(np.float64) + 1e-5 * lr
    assert np.all(np.abs(m.get_params() - want) <= bound)
