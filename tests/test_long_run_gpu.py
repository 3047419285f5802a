"""A long run of the reference's own AIREBO forces, which heat the crystal until
it comes apart: crowded molecules, rows cut at 12 bonds, then a gas, over every
kind of row the LJ gather walks.  Forces, energies and virial of the states on
the way against the oracle over the system's own lists."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import RunConfig, System, crystal
from fuller_md_en_b200._lib import FMD_PREC_FP32_PAIR, FMD_PREC_FP64

pytestmark = pytest.mark.gpu


# As in test_rebo_mol_gpu.py and test_lj_clus_gpu.py: sums of up to some hundred
# terms, 1e-12 of the largest force; FP32 pair terms 2e-6.
@pytest.mark.parametrize("nc,st,prec,tol", [(2, "FCC", FMD_PREC_FP64, 1e-12), (3, "FCC", FMD_PREC_FP64, 1e-12),
                                            (2, "BCC", FMD_PREC_FP64, 1e-12), (2, "FCC", FMD_PREC_FP32_PAIR, 2e-6)])
def test_states_on_the_way_match_oracle(ctx, oracle, nc, st, prec, tol):
    s = crystal.atomistic(nc, T=300.0, jitter=0.01, seed=42, st=st)
    na = s["pos"].size // 3
    cfg = RunConfig(dt=0.5, T=300.0, Pe=0.0, nsteps=10 ** 6, nlup=20, nc=nc, nmol=s["nmol"], precision=prec)
    y = System.airebo(ctx, cfg, s["pos"], s["vel"], s["mass"], s["mol_id"], s["h"], crystal.npt_atom(300.0, 0.0, na))
    y.init()
    done, cut, walked = 0, 0, set()
    for g in (70, 110, 150, 190, 225, 260, 333, 400):
        before = y.lj_gathers()
        y.run(done + 1, g)
        done = g
        walked |= {k for k, v in y.lj_gathers().items() if v > before[k]}
        F, _, E = y.forces()
        W, _ = y.virial()
        d = y.download()
        ca, la, cb, lb = y.lists(400, 12)
        cut = max(cut, int((cb >= 12).sum()))
        Er, Fr, Wr = oracle.airebo_forces(d["pos"], d["h"], crystal.inv9(d["h"]), cb, lb, ca, la, na)
        big = np.abs(Fr).max()
        assert np.abs(F - np.ravel(Fr)).max() <= tol * big, (g, np.abs(F - np.ravel(Fr)).max(), big)
        assert np.abs(E[1] - Er[1]) <= tol * big * na and np.abs(E[2] - Er[2]) <= tol * big * na, (g, E, Er)
        assert np.abs(W - Wr).max() <= tol * big * na, g
    assert cut > na // 20 and {"clusters_built", "clusters_walked"} <= walked, (cut, walked)
    assert st == "BCC" or "full" in walked, walked               # this crystal holds together longer
    y.close()
