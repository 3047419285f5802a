"""Learned-term systems made one after the other in a context take the
workspaces that the last one released, and give what the first gave."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import RunConfig, System, crystal


# 20 steps from the same state: FP64 sums whose order varies (atomics) move
# forces by some 1e-15, the FP32 network's output by its BF16 roundings: 1e-6
# of the largest force.
@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(2, 2, 2), (1, 2, 1)])
def test_workspaces_of_a_released_system(ctx, sizes):
    import torch
    from fuller_md_en_b200.surrogate import Surrogate
    from oracle import sg_oracle
    P = sg_oracle.init_params(3)
    P["b0"], P["bs"] = 0.95, 0.02
    model = Surrogate(ctx, P)
    first, free = {}, []
    for nc in sizes + sizes:
        s = crystal.atomistic(nc, jitter=0.01, seed=nc, T=300.0)
        na = s["pos"].size // 3
        cfg = RunConfig(dt=0.5, T=300.0, Pe=0.0, nsteps=100, nlup=20, nc=nc, nmol=s["nmol"])
        y = System.airebo(ctx, cfg, s["pos"], s["vel"], s["mass"], s["mol_id"], s["h"],
                          crystal.npt_atom(300.0, 0.0, na))
        y.init()
        y.use_surrogate(model, judge_every=10, rmse_max=1e9)
        y.run(1, 20)
        F = y.forces()[0].copy()
        y.close()
        free.append(torch.cuda.mem_get_info()[0])
        assert np.abs(F - first.setdefault(nc, F)).max() <= 1e-6 * np.abs(F).max()
    assert free[len(sizes):] == [free[-1]] * len(sizes)          # nothing more is taken the second time round
    model.close()
