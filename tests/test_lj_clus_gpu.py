"""The cluster gather (ljclus.cu) against the oracle's LJ over the system's own
lists: molecule sizes whose last cluster is partial or full, cells so narrow
that a partner needs an entry per image, molecules across the cell's faces,
single and double precision pairs, and a cell that shrinks until no cluster
rows can be built."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import RunConfig, System, crystal
from fuller_md_en_b200._lib import FMD_PREC_FP32_PAIR, FMD_PREC_FP64

pytestmark = pytest.mark.gpu


def _molecule(S):
    """S atoms beyond the REBO cutoff of 2 A from one another: a C60 of 1.7 times the size and atoms inside it."""
    inner = 1.7 * np.array([[1, 1, 1], [-1, -1, 1], [1, -1, -1], [-1, 1, -1]], float)
    return np.concatenate([1.7 * crystal.c60_ih(), inner])[:S]


def _system(ctx, nc, S, a0, prec, shift=0.0, P=0.0, nlup=5, delta=0.5):
    s = crystal.atomistic(nc, coords=_molecule(S), jitter=0.05, seed=S + nc, T=100.0)
    na = s["pos"].size // 3
    f = a0 / s["a0"]
    h = s["h"] * f
    centres = np.repeat(s["pos"].reshape(-1, S, 3).mean(axis=1), S, axis=0)
    pos = (s["pos"].reshape(-1, 3) + (f - 1.0) * centres + shift).reshape(-1)
    cfg = RunConfig(dt=0.5, T=100.0, Pe=P, nsteps=1000, nlup=nlup, nc=nc, nmol=s["nmol"], precision=prec)
    y = System.airebo(ctx, cfg, pos, s["vel"], s["mass"], s["mol_id"], h, crystal.npt_atom(100.0, P, na))
    y.set_lj_prune(delta)
    y.init()
    return y, na


# FP64: sums of a few hundred pair terms, each a few ulp from the reference's,
# over forces of mixed sign: 1e-12 of the largest force.  FP32 pairs: each term
# to a few 2^-24, likewise summed: 2e-6.
@pytest.mark.parametrize("nc,S,a0,shift,prec,tol", [
    (1, 32, 21.9, 7.3, FMD_PREC_FP64, 1e-12),      # clusters of 4; the narrowest cell
    (1, 45, 22.5, 0.0, FMD_PREC_FP64, 1e-12),      # a partial last cluster
    (2, 60, 21.0, 11.1, FMD_PREC_FP64, 1e-12),
    (1, 64, 24.0, 5.0, FMD_PREC_FP32_PAIR, 2e-6),
    (3, 60, 26.0, 3.0, FMD_PREC_FP32_PAIR, 2e-6),
])
def test_cluster_rows_match_oracle(ctx, oracle, nc, S, a0, shift, prec, tol):
    y, na = _system(ctx, nc, S, a0, prec, shift)
    for first, last in ((0, 0), (1, 3), (4, 7)):     # built rows, walked rows, after a list build
        if last:
            y.run(first, last)
        F, _, E = y.forces()
        W, _ = y.virial()
        d = y.download()
        cl, ll, _, _ = y.lists(400, 12)
        e, oF, oW = oracle.lj(d["pos"], d["h"], crystal.inv9(d["h"]), cl, ll, na)
        assert abs(E[1]) == 0.0 and abs(E[2] - e) <= tol * np.abs(oF).max() * na
        assert np.abs(F - oF).max() <= tol * np.abs(oF).max(), (last, np.abs(F - oF).max(), np.abs(oF).max())
        assert np.abs(W - oW).max() <= 30 * tol * np.abs(oW).max()
    st = y.lj_prune()
    assert 2 <= st["prunes"] < st["evaluations"] == 8, st     # rows were walked, not only built
    y.close()


def test_shrinking_cell_leaves_cluster_rows(ctx):
    """A cell pressed from above the width that cluster rows need to below it:
    the run goes on over the full rows as one without pruning."""
    ys = [_system(ctx, 1, 60, 21.96, FMD_PREC_FP64, P=400.0, nlup=20, delta=d)[0] for d in (0.5, 0.0)]
    for g in range(1, 241):
        a, b = ys[0].run(g, g), ys[1].run(g, g)
        assert abs(a.E[2] - b.E[2]) <= 1e-8 * abs(b.E[2]), g
    edge = ys[0].download()["h"][0]
    st = ys[0].lj_prune()
    assert edge < 21.5 and 0 < st["prunes"] < st["evaluations"], (edge, st)
    for y in ys:
        y.close()
