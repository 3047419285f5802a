"""Which rows the LJ gather of a system of equal molecules walks: clusters
while they pay, atoms where the cell or the atoms' motion says so, and the
same pairs either way."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import Batch, RunConfig, System, crystal
from fuller_md_en_b200._lib import FMD_PREC_FP32_PAIR, FMD_PREC_FP64
from fuller_md_en_b200.api import Topology

pytestmark = pytest.mark.gpu


def _airebo(ctx, nc, delta, T, f=1.0, P=0.0, nlup=10):
    s = crystal.atomistic(nc, jitter=0.02, seed=8, T=T)
    na = s["pos"].size // 3
    centres = np.repeat(s["pos"].reshape(-1, 60, 3).mean(axis=1), 60, axis=0)
    pos = (s["pos"].reshape(-1, 3) + (f - 1.0) * centres).reshape(-1)
    cfg = RunConfig(dt=0.5, T=T, Pe=P, nsteps=10 ** 6, nlup=nlup, nc=nc, nmol=s["nmol"])
    y = System.airebo(ctx, cfg, pos, s["vel"], s["mass"], s["mol_id"], f * s["h"], crystal.npt_atom(T, P, na))
    y.set_lj_prune(delta)
    y.init()
    return y


def _same(a, b, what, tol=1e-9):
    """The same pairs, other orders of the sums."""
    for k in range(8):
        assert abs(a.E[k] - b.E[k]) <= tol * max(1e-3, abs(b.E[k])), (what, k, a.E[k], b.E[k])


def _gas(ctx, nc, T, prec=FMD_PREC_FP64, seed=4):
    """Molecules of 60 atoms without bonded terms: forces are the LJ term's."""
    z = lambda *k: np.zeros(k)
    topo = Topology(z(0, 2), z(0), z(0), z(0, 3), z(0), z(0), z(0, 4), z(0), z(0), z(0), z(0, 4), z(0), z(0))
    s = crystal.atomistic(nc, jitter=0.02, seed=seed, T=T, mol_base=0)
    na = s["pos"].size // 3
    cfg = RunConfig(dt=0.5, T=T, Pe=0.0, nsteps=1000, nlup=10, nc=nc, nmol=s["nmol"], precision=prec)
    return System.mm(ctx, cfg, s["pos"], s["vel"], s["mol_id"], topo, s["h"], crystal.npt_atom(T, 0.0, na))


# As in test_lj_clus_gpu.py: FP64 sums of a few hundred pair terms, each a few
# ulp from the reference's, 1e-12 of the largest force; FP32 pair terms 2e-6.
def _matches_oracle(oracle, y, prec, what):
    tol = 1e-12 if prec == FMD_PREC_FP64 else 2e-6
    F, _, E = y.forces()
    W, _ = y.virial()
    d = y.download()
    cl, ll = y.lists(400)[:2]
    e, oF, oW = oracle.lj(d["pos"], d["h"], crystal.inv9(d["h"]), cl, ll, F.size // 3, mm=True)
    top, w = np.abs(oF).max(), [0, 4, 8]
    assert np.abs(F - oF).max() <= tol * top, (what, np.abs(F - oF).max(), top)
    assert abs(E[4] - e) <= tol * top * (F.size // 3), (what, E[4], e)
    assert np.abs(W[w] - oW[w]).max() <= 30 * tol * np.abs(oW[w]).max(), (what, W[w], oW[w])


# The fastest atom moves some 0.13 A a step at 6e4 K, 0.45 A at 6e5 K: it uses up
# the buffer of 0.5 A in two steps or in one.
@pytest.mark.parametrize("T,prec", [(6e4, FMD_PREC_FP64), (6e4, FMD_PREC_FP32_PAIR), (6e5, FMD_PREC_FP64),
                                    (6e5, FMD_PREC_FP32_PAIR)])
def test_fast_atoms_get_rows_of_atoms(ctx, oracle, T, prec):
    y = _gas(ctx, 2, T, prec)
    y.init()
    for g in range(1, 26):
        y.run(g, g)
        _matches_oracle(oracle, y, prec, g)
    n = y.lj_gathers()
    assert n["clusters_built"] >= 3 and n["clusters_built"] + n["clusters_walked"] == 10, n   # until the first build
    if T < 1e5:
        assert n["atoms_built"] >= 5 and n["atoms_walked"] >= 3 and n["full"] == 0, n
    else:                                            # every evaluation pruned: not any more
        assert n["full"] == 16 and n["atoms_built"] + n["atoms_walked"] == 0, n
    assert sum(n.values()) == 26 and n["atoms_built"] + n["clusters_built"] == y.lj_prune()["prunes"]
    y.close()


def test_prunes_are_counted_again(ctx, oracle):
    """Eight builds of full rows, then one of pruned rows, and so on."""
    y = _gas(ctx, 2, 6e5, seed=6)
    y.init()
    seen = []
    for g in range(1, 221):
        y.run(g, g)
        if g % 10 == 5:
            before = y.lj_gathers()
            y.run(g + 1000000, g + 1000000)          # a step more, no build
            after = y.lj_gathers()
            seen.append([k for k in after if after[k] > before[k]][0])
            _matches_oracle(oracle, y, FMD_PREC_FP64, g)
    y.close()
    assert seen[1:9] == ["full"] * 8 and seen[9] == "atoms_built" and seen[10:18] == ["full"] * 8, seen


def test_slow_atoms_keep_clusters(ctx):
    y = _airebo(ctx, 2, 0.5, 100.0)
    y.run(1, 40)
    n = y.lj_gathers()
    assert n["atoms_built"] + n["atoms_walked"] == 0 and n["clusters_walked"] > 2 * n["clusters_built"] >= 10, n
    y.close()


def test_batch_chooses_by_replica(ctx, oracle):
    reps = [_gas(ctx, 2, 50.0), _gas(ctx, 2, 6e5, seed=5)]
    b = Batch(ctx, reps)
    for g in range(1, 26):
        b.run(g, g)
        for r, y in enumerate(reps):
            _matches_oracle(oracle, y, FMD_PREC_FP64, (g, r))
    b.close()
    cold, hot = (y.lj_gathers() for y in reps)
    assert cold["atoms_built"] + cold["atoms_walked"] == 0 and cold["clusters_walked"] > 15, cold
    assert hot["full"] == 16, hot
    for y in reps:
        y.close()


def test_shrinking_cell_without_rebuilds(ctx):
    """Steps 1-10 over and over, none of them a rebuild, from an edge that
    leaves the full rows out to one below the width of cluster rows (21.5 A)."""
    ys = [_airebo(ctx, 1, d, 300.0, f=21.9 / 14.016, P=400.0, nlup=20) for d in (0.5, 0.0)]
    r = 0
    while ys[0].download()["h"][0] > 21.45 and r < 60:
        _same(ys[0].run(1, 10), ys[1].run(1, 10), r, 1e-8)
        r += 1
    _same(ys[0].run(1, 10), ys[1].run(1, 10), r, 1e-8)
    n = ys[0].lj_gathers()
    assert ys[0].download()["h"][0] < 21.5 and n["clusters_walked"] > 20 and n["atoms_built"] > 0, n
    for y in ys:
        y.close()
