"""The cases of test_lj_clus_gpu.py and more, with the rows the gather walked:
molecules whose last cluster is partial, cells so narrow that a partner needs an
entry per image, a cell that shrinks below the width of cluster rows, and a
replica batch of such systems."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import Batch, RunConfig, System, crystal
from fuller_md_en_b200._lib import FMD_PREC_FP32_PAIR, FMD_PREC_FP64
from fuller_md_en_b200.api import Topology
from test_lj_clus_gpu import _molecule, _system

pytestmark = pytest.mark.gpu


# Tolerances as in test_lj_clus_gpu.py.
@pytest.mark.parametrize("nc,S,a0,shift,prec,tol", [
    (1, 32, 21.9, 7.3, FMD_PREC_FP64, 1e-12),      # the narrowest cell: two images of a partner
    (1, 45, 22.5, 0.0, FMD_PREC_FP64, 1e-12),      # and a partial last cluster
    (1, 33, 24.0, 2.0, FMD_PREC_FP64, 1e-12),      # a last cluster of one
    (1, 62, 21.9, 5.0, FMD_PREC_FP32_PAIR, 2e-6),
    (2, 60, 21.0, 11.1, FMD_PREC_FP64, 1e-12),
    (1, 64, 24.0, 5.0, FMD_PREC_FP32_PAIR, 2e-6),
    (3, 60, 26.0, 3.0, FMD_PREC_FP32_PAIR, 2e-6),
])
def test_cluster_rows_are_walked(ctx, oracle, nc, S, a0, shift, prec, tol):
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
    n = y.lj_gathers()
    assert n["clusters_built"] >= 2 and n["clusters_walked"] >= 1 and sum(n.values()) == 8, n
    assert n["clusters_built"] + n["clusters_walked"] == 8, n
    y.close()


def test_shrinking_cell_goes_over_to_atoms(ctx):
    """A cell pressed from above the width that cluster rows need (21.5 A) to
    below it: cluster rows, then rows of atoms, as one without pruning."""
    ys = [_system(ctx, 1, 60, 21.96, FMD_PREC_FP64, P=400.0, nlup=20, delta=d)[0] for d in (0.5, 0.0)]
    was = {}
    for g in range(1, 241):
        a, b = ys[0].run(g, g), ys[1].run(g, g)
        assert abs(a.E[2] - b.E[2]) <= 1e-8 * abs(b.E[2]), g
        if g % 20 == 0:
            n, edge = ys[0].lj_gathers(), ys[0].download()["h"][0]
            new = {k for k in n if n[k] > was.get(k, 0)}
            if edge > 21.5:
                assert new <= {"clusters_built", "clusters_walked"}, (g, edge, n)
            was = n
    assert ys[0].download()["h"][0] < 21.5 and was["clusters_walked"] > 0 and was["atoms_walked"] > 0, was
    for y in ys:
        y.close()


def test_batch_walks_clusters(ctx, oracle):
    z = lambda *k: np.zeros(k)
    topo = Topology(z(0, 2), z(0), z(0), z(0, 3), z(0), z(0), z(0, 4), z(0), z(0), z(0), z(0, 4), z(0), z(0))
    reps = []
    for S, a0 in ((45, 22.5), (33, 24.0), (64, 22.3)):
        s = crystal.atomistic(1, coords=_molecule(S), jitter=0.05, seed=S, T=100.0, mol_base=0)
        na = s["pos"].size // 3
        f = a0 / s["a0"]
        centres = np.repeat(s["pos"].reshape(-1, S, 3).mean(axis=1), S, axis=0)
        pos = (s["pos"].reshape(-1, 3) + (f - 1.0) * centres).reshape(-1)
        cfg = RunConfig(dt=0.5, T=100.0, Pe=0.0, nsteps=1000, nlup=5, nc=1, nmol=s["nmol"])
        reps.append(System.mm(ctx, cfg, pos, s["vel"], s["mol_id"], topo, s["h"] * f, crystal.npt_atom(100.0, 0.0, na)))
    b = Batch(ctx, reps)
    for g in (3, 7):
        b.run(1 if g == 3 else 4, g)
        for y in reps:
            F, _, E = y.forces()
            W, _ = y.virial()
            d = y.download()
            cl, ll = y.lists(400)[:2]
            e, oF, oW = oracle.lj(d["pos"], d["h"], crystal.inv9(d["h"]), cl, ll, F.size // 3, mm=True)
            top = np.abs(oF).max()
            assert np.abs(F - oF).max() <= 1e-12 * top and abs(E[4] - e) <= 1e-12 * top * (F.size // 3)
            assert np.abs((W - oW)[[0, 4, 8]]).max() <= 30e-12 * np.abs(oW[[0, 4, 8]]).max()
    b.close()
    for y in reps:
        n = y.lj_gathers()
        assert n["clusters_walked"] >= 1 and n["atoms_built"] + n["atoms_walked"] + n["full"] == 0, n
        y.close()
