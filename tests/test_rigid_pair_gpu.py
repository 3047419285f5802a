"""The rigid model's pair kernel (rigidpair.cu) against the oracle over the
system's own lists: sites per molecule at the lanes' edges, rows cut at the
list width (entries without their reverse), a few and many warps per molecule,
molecules in contact with themselves' images, FP64 and FP32 pairs."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import RunConfig, System, crystal
from fuller_md_en_b200._lib import FMD_PREC_FP32_PAIR, FMD_PREC_FP64

pytestmark = pytest.mark.gpu


# FP64: ~20,000 pair terms a molecule, each a few ulp, the partner's torque
# over a lever arm of at most three radii: 1e-11 of the largest.  FP32: a pair
# whose FP32 distance falls on the other side of the cutoff moves 8.4e-6 eV/A
# (3e-5 over a molecule, against a few tenths), pair terms to 1e-6.
@pytest.mark.parametrize("nc,natom,cap,prec", [
    (1, 33, 80, FMD_PREC_FP64), (2, 1, 80, FMD_PREC_FP64), (2, 60, 80, FMD_PREC_FP64), (3, 60, 20, FMD_PREC_FP64),
    (2, 64, 7, FMD_PREC_FP64), (4, 32, 128, FMD_PREC_FP64), (2, 60, 80, FMD_PREC_FP32_PAIR),
    (3, 64, 20, FMD_PREC_FP32_PAIR), (6, 60, 80, FMD_PREC_FP32_PAIR), (1, 60, 80, FMD_PREC_FP32_PAIR),
])
def test_pair_kernel_matches_oracle(ctx, oracle, nc, natom, cap, prec):
    inner = 0.9 * np.array([[1, 1, 1], [-1, -1, 1], [1, -1, -1], [-1, 1, -1]], float)
    coords = np.concatenate([crystal.c60_ih(), inner])[:natom]
    s = crystal.rigid(nc, coords=coords, seed=natom + nc, a0=14.02)
    n = s["n"]
    I0 = max(s["I0"], 1.0)
    rmcut = 3.0 * 3.431 + 2 * s["Rmol"] + 1.0
    cfg = RunConfig(dt=1.0, T=300.0, Pe=0.5, nsteps=100, nlup=4, nc=nc, nmol=n, precision=prec)
    omg = s["omg"] if natom > 1 else np.zeros(3 * n)
    y = System.rigid(ctx, cfg, natom, s["body"], I0, s["Mmol"], rmcut, s["pos"], s["vel"], s["qv"], omg, s["h"],
                     crystal.npt_rigid(300.0, 0.5, n), max_neigh=cap)
    y.init()
    f64 = prec == FMD_PREC_FP64
    for first, last in ((0, 0), (1, 2), (3, 5)):      # set-up, the step's own sums, after a list build
        if last:
            y.run(first, last)
        F, T, E = y.forces()
        W, _ = y.virial()
        d = y.download()
        c, l, _, _ = y.lists(cap)
        e, oF, oT, oW = oracle.rigid_forces(d["pos"], d["qv"], s["body"], d["h"], crystal.inv9(d["h"]), c, l, n, natom,
                                            rmcut * rmcut, cap=cap)
        assert abs(E[0] - e) <= (1e-11 if f64 else 1e-6) * max(abs(e), 1e-3)
        assert np.abs(F - oF).max() <= (1e-11 if f64 else 2e-4) * max(np.abs(oF).max(), 1e-6)
        assert np.abs(T - oT).max() <= (1e-11 if f64 else 5e-4) * max(np.abs(oT).max(), 1e-6)
        assert np.abs(W - oW).max() <= (1e-11 if f64 else 2e-6) * max(np.linalg.norm(oW), 1e-3)
    y.close()
