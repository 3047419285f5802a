"""The bonded terms by molecules (mmmol.cu) against the term-wise kernel
(mm.cu): the same terms, once in the copies' order, which the first takes, and
once with each kind reversed, which it does not."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import RunConfig, System, crystal
from fuller_md_en_b200._lib import FMD_PHYS_MM_BONDED
from fuller_md_en_b200.api import Topology

pytestmark = pytest.mark.gpu


def _terms(S, copies_of_torsions, rng):
    """One molecule's terms over a chain of its S atoms: {kind: (indices, parameters)}."""
    chain = lambda k: np.stack([np.arange(S - k + 1) + q for q in range(k)], axis=1).reshape(-1, k)
    b, a, d = chain(2), chain(3), np.concatenate([chain(4)] * copies_of_torsions)
    im = chain(4)[:, [1, 0, 2, 3]]
    u = lambda n, lo, hi: rng.uniform(lo, hi, n)
    mult = rng.choice([0, 1, 2, 2, 3, -2, 8, 9, -13], len(d)).astype(np.int32)
    return {"b": (b, u(len(b), 5, 20), u(len(b), 1.2, 3.0)), "a": (a, u(len(a), 1, 3), u(len(a), 1.5, 2.5)),
            "d": (d, u(len(d), 0.2, 0.7), mult, u(len(d), -3, 3)), "i": (im, u(len(im), 0.2, 0.7), u(len(im), -3, 3))}


def _topology(t, S, nmol, reverse):
    def rep(v):
        idx = (v[0][None] + (np.arange(nmol) * S)[:, None, None]).reshape(-1, v[0].shape[1])
        out = [idx] + [np.tile(p, nmol) for p in v[1:]]
        return [x[::-1].copy() for x in out] if reverse else out
    return Topology(*rep(t["b"]), *rep(t["a"]), *rep(t["d"]), *rep(t["i"]))


# Each of an atom's (at most 60) term forces is off by a few ulp times the
# condition of its angle (chains of a C60's atoms: sines above 0.1) and, for a
# multiple angle of 13, 13 ulp; sums of mixed sign: 1e-11 of the largest force.
@pytest.mark.parametrize("S,nc,a0,reps,physical", [
    (4, 3, 12.0, 1, False),            # one torsion a molecule
    (33, 2, 14.2, 2, True),
    (60, 1, 14.2, 5, False),           # atoms beyond a quarter of the cell: images per vector
    (60, 2, 14.2, 5, True),
    (60, 2, 14.2, 20, False),          # more force slots than a block holds: term-wise either way
])
def test_molecules_match_terms(ctx, S, nc, a0, reps, physical):
    rng = np.random.default_rng(S + nc)
    s = crystal.atomistic(nc, coords=crystal.c60_ih()[:S], jitter=0.03, seed=S, T=50.0, mol_base=0)
    na = s["pos"].size // 3
    h = s["h"] * (a0 / s["a0"])
    centres = np.repeat(s["pos"].reshape(-1, S, 3).mean(axis=1), S, axis=0)
    pos = (s["pos"].reshape(-1, 3) + (a0 / s["a0"] - 1.0) * centres + 5.3).reshape(-1)
    t = _terms(S, reps, rng)
    got = []
    for reverse in (False, True):
        cfg = RunConfig(dt=0.02, T=50.0, Pe=0.0, nsteps=100, nlup=5, nc=nc, nmol=s["nmol"])
        y = System.mm(ctx, cfg, pos, s["vel"], s["mol_id"], _topology(t, S, s["nmol"], reverse), h,
                      crystal.npt_atom(50.0, 0.0, na))
        if physical:
            y.set_physics(FMD_PHYS_MM_BONDED)
        y.init()
        y.run(1, 2)
        F, _, E = y.forces()
        got.append((F, E, y.virial()[0]))
        y.close()
    (F, E, W), (Fr, Er, Wr) = got
    assert np.isfinite(F).all() and np.abs(Fr).max() > 0.1
    assert np.abs(F - Fr).max() <= 1e-11 * np.abs(Fr).max()
    assert np.abs(E - Er).max() <= 1e-12 * np.abs(Er).max()
    assert np.abs(W - Wr).max() <= 1e-11 * np.abs(Fr).max() * np.sqrt(na)


def test_replicated_molecule_is_the_same_system(ctx):
    """One molecule's topology replicated on the device and the full flat one: bit for bit."""
    S = 60
    s = crystal.atomistic(2, jitter=0.02, seed=3, T=300.0, mol_base=0)
    c = crystal.c60_ih()
    bonds = crystal.bonds_from_geometry(c)
    got = []
    for full in (False, True):
        t = crystal.mm_topology(c, bonds, s["nmol"] if full else 1)
        topo = Topology(t["bonds"], t["kb"], t["r0"], t["angles"], t["kth"], t["th0"], t["dihedrals"], t["vn"],
                        t["mult"], t["gamma"], t["impropers"], t["ki"], t["igamma"])
        cfg = RunConfig(dt=0.1, T=300.0, Pe=0.0, nsteps=100, nlup=20, nc=2, nmol=s["nmol"])
        n = crystal.npt_atom(300.0, 0.0, S * s["nmol"])
        y = (System.mm(ctx, cfg, s["pos"], s["vel"], s["mol_id"], topo, s["h"], n) if full else
             System.mm_replicated(ctx, cfg, s["nmol"], S, s["pos"], s["vel"], topo, s["h"], n))
        y.init()
        y.run(1, 5)
        got.append((y.forces()[0], y.virial()[0], y.download()["pos"]))
        y.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
