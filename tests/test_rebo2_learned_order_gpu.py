"""fmd_system_set_rebo2 and fmd_system_use_surrogate before init, in either
order: the step's energy and virial sum every record the learned term writes."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import Rebo2Knots, RunConfig, System, crystal
from fuller_md_en_b200._lib import FMD_REBO2_LJ_SWITCH

pytestmark = pytest.mark.gpu


# The same sums in both orders, and of one state: FP64 sums of some 10^4 terms
# in an order that atomics vary, 1e-12 of the energy and of the largest virial.
# The learned term's records reach beyond one per molecule, or beyond 592: the
# crystals are large, or each atom has some nine bonds.
@pytest.mark.parametrize("nc,size", [(7, 1.0), (4, 0.8)])
@pytest.mark.parametrize("flags", [0, FMD_REBO2_LJ_SWITCH])
def test_record_count_in_either_order(ctx, nc, size, flags):
    from fuller_md_en_b200.surrogate import Surrogate
    from oracle import sg_oracle
    P = sg_oracle.init_params(3)
    P["b0"], P["bs"] = 0.95, 0.02
    model = Surrogate(ctx, P)
    got = []
    for rebo2_last in (False, True):
        s = crystal.atomistic(nc, coords=size * crystal.c60_ih(), jitter=0.01, seed=nc, T=300.0)
        na = s["pos"].size // 3
        cfg = RunConfig(dt=0.5, T=300.0, Pe=0.0, nsteps=100, nlup=20, nc=nc, nmol=s["nmol"])
        y = System.airebo(ctx, cfg, s["pos"], s["vel"], s["mass"], s["mol_id"], s["h"],
                          crystal.npt_atom(300.0, 0.0, na))
        for call in ((1, 0) if rebo2_last else (0, 1)):
            if call == 0:
                y.set_rebo2(Rebo2Knots(), flags)
            else:
                y.use_surrogate(model, judge_every=1000, rmse_max=1e9)
        y.init()
        F, _, E = y.forces()
        W, _ = y.virial()
        out = y.download()
        _, _, cb, lb = y.lists(400, 12)
        E_sg, _, _ = model.rebo_forces(out["pos"], out["h"], ctx.mat_inv9(out["h"]), cb, lb)
        got.append((np.array(E), np.array(W), F.copy(), E_sg))
        y.close()
    model.close()
    for E, W, F, E_sg in got:
        assert abs(E[1] - E_sg) <= 1e-9 * abs(E_sg), (E[1], E_sg)
        assert np.abs(E - got[0][0]).max() <= 1e-12 * np.abs(got[0][0]).max()
        assert np.abs(W - got[0][1]).max() <= 1e-12 * np.abs(got[0][1]).max()
        assert np.abs(F - got[0][2]).max() <= 1e-9 * np.abs(got[0][2]).max()
