"""The REBO term by molecules (rebomol.cu): against the oracle over the
system's own lists for molecules of one and of two warps' worth of lanes, atoms
with one to four bonds, more than four (the bond-wise code) and rows truncated
at the list's width; and its gradient form against the slot kernels, which the
same atoms in an interleaved order take."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import RunConfig, System, crystal
from fuller_md_en_b200._lib import FMD_PHYS_REBO

pytestmark = pytest.mark.gpu


def _molecule(kind, S):
    if kind == "c60":
        return crystal.c60_ih()[:S]
    if kind == "chain":                                   # one and two bonds
        return np.array([[1.3 * k, 0.3 * (k % 2), 0.1 * (k % 3)] for k in range(S)]) - [0.65 * S, 0, 0]
    n = int(np.ceil(S ** (1 / 3)))
    grid = np.array([[x, y, z] for x in range(n) for y in range(n) for z in range(n)], float)
    if kind == "diamond":                                 # up to four bonds
        d = np.array([[0, 0, 0], [0, 2, 2], [2, 0, 2], [2, 2, 0], [1, 1, 1], [1, 3, 3], [3, 1, 3], [3, 3, 1]], float)
        pts = (d[None] + 4.0 * grid[:, None]).reshape(-1, 3) * (1.54 / np.sqrt(3.0))
        return pts[np.argsort(((pts - pts.mean(0)) ** 2).sum(1), kind="stable")[:S]]
    return grid[:S] * (1.6 if kind == "cubic" else 1.25)  # six bonds; eighteen, more than a row holds


def _system(ctx, kind, S, nc, phys, order=None):
    s = crystal.atomistic(nc, coords=_molecule(kind, S), jitter=0.02, seed=S, T=20.0)
    na = s["pos"].size // 3
    a0 = 24.0 if kind != "chain" else 30.0
    h = s["h"] * (a0 / s["a0"])
    centres = np.repeat(s["pos"].reshape(-1, S, 3).mean(axis=1), S, axis=0)
    pos = s["pos"].reshape(-1, 3) + (a0 / s["a0"] - 1.0) * centres
    order = np.arange(na) if order is None else order
    cfg = RunConfig(dt=1e-3, T=20.0, Pe=0.0, nsteps=100, nlup=50, nc=nc, nmol=s["nmol"])
    y = System.airebo(ctx, cfg, pos[order].reshape(-1), s["vel"].reshape(-1, 3)[order].reshape(-1), s["mass"][order],
                      s["mol_id"][order], h, crystal.npt_atom(20.0, 0.0, na))
    if phys:
        y.set_physics(FMD_PHYS_REBO)
    y.init()
    return y, na


# Each force is a sum of some tens of terms, each a few ulp from the
# reference's and some a hundred times the sum: 1e-12 of the largest force.
@pytest.mark.parametrize("kind,S,nc", [("c60", 60, 2), ("c60", 33, 1), ("chain", 5, 2), ("chain", 16, 1),
                                       ("diamond", 64, 1), ("diamond", 90, 1), ("diamond", 128, 2),
                                       ("cubic", 27, 1), ("dense", 64, 1)])
def test_molecules_match_oracle(ctx, oracle, kind, S, nc):
    y, na = _system(ctx, kind, S, nc, False)
    y.run(1, 1)
    F, _, E = y.forces()
    W, _ = y.virial()
    st = y.download()
    ca, la, cb, lb = y.lists(400, 12)
    y.close()
    Er, Fr, Wr = oracle.airebo_forces(st["pos"], st["h"], crystal.inv9(st["h"]), cb, lb, ca, la, na)
    big = np.abs(Fr).max()
    assert abs(E[1] - Er[1]) <= 1e-12 * np.abs(Er[1]) and np.abs(F - np.ravel(Fr)).max() <= 1e-12 * big
    assert np.abs(W - Wr).max() <= 1e-12 * big * na


@pytest.mark.parametrize("kind,S,nc", [("c60", 60, 1), ("diamond", 64, 1), ("chain", 16, 1), ("cubic", 27, 1)])
def test_gradient_matches_slot_kernels(ctx, kind, S, nc):
    got = []
    na = 4 * nc ** 3 * S
    order = np.arange(na).reshape(-1, S).T.reshape(-1)    # atom 0 of every molecule, atom 1, ...
    for o in (np.arange(na), order):
        y, _ = _system(ctx, kind, S, nc, True, o)
        F, _, E = y.forces()
        W, _ = y.virial()
        y.close()
        G = np.empty((na, 3))
        G[o] = F.reshape(-1, 3)
        got.append((G, E, W))
    (F, E, W), (Fr, Er, Wr) = got
    assert np.abs(F - Fr).max() <= 1e-12 * np.abs(Fr).max() and abs(E[1] - Er[1]) <= 1e-12 * abs(Er[1])
    assert np.abs(W - Wr).max() <= 1e-12 * np.abs(Fr).max() * na
