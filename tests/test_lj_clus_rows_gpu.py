"""A cell that leaves the form cluster rows need between two list builds, which
left the full rows unbuilt (it shears).  The gather then builds the rows
itself, and the run goes on as one over full rows."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import Batch, RunConfig, System, crystal
from fuller_md_en_b200.api import _c60_molecule_topology

pytestmark = pytest.mark.gpu


def _airebo(ctx, nc, delta, shear=0.0):
    s = crystal.atomistic(nc, jitter=0.02, seed=8)
    na = s["pos"].size // 3
    npt = crystal.npt_atom(300.0, 0.0, na)
    npt[3] = shear                                   # Vg[0][1]
    cfg = RunConfig(dt=0.5, T=300.0, Pe=0.0, nsteps=10 ** 6, nlup=20, nc=nc, nmol=s["nmol"])
    y = System.airebo(ctx, cfg, s["pos"], s["vel"], s["mass"], s["mol_id"], s["h"], npt)
    y.set_lj_prune(delta)
    y.init()
    return y


def _same(a, b, what):
    """The same pairs, other orders of the sums: 1e-9 of each energy."""
    for k in range(8):
        assert abs(a.E[k] - b.E[k]) <= 1e-9 * max(1e-3, abs(b.E[k])), (what, k, a.E[k], b.E[k])


def test_sheared_cell(ctx):
    p, f = (_airebo(ctx, 2, d, shear=1e-3) for d in (0.5, 0.0))
    full = f.lj_rows()[0]
    for g in range(1, 31):                           # the shear starts with step 1, lists are built at 20
        _same(p.run(g, g), f.run(g, g), g)
        if g < 20:
            assert np.array_equal(p.lj_rows()[0], full), g
    assert p.download()["h"][1] > 0.01
    for y in (p, f):
        y.close()


def test_sheared_batch(ctx):
    coords, topo = _c60_molecule_topology()

    def make(delta, shear):
        s = crystal.atomistic(2, coords=coords, jitter=0.01, seed=4, mol_base=0)
        na = s["pos"].size // 3
        npt = crystal.npt_atom(300.0, 0.0, na)
        npt[3] = shear
        cfg = RunConfig(dt=0.1, T=300.0, Pe=0.0, nsteps=10 ** 6, nlup=20, nc=2, nmol=s["nmol"])
        y = System.mm_replicated(ctx, cfg, s["nmol"], 60, s["pos"], s["vel"], topo, s["h"], npt)
        y.set_lj_prune(delta)
        y.init()
        return y
    ps = [make(0.5, v) for v in (0.0, 1e-3)]
    fs = [make(0.0, v) for v in (0.0, 1e-3)]
    b = Batch(ctx, ps)
    for g in range(1, 26):
        for o, f in zip(b.run(g, g), fs):
            _same(o, f.run(g, g), g)
    b.close()
    for y in ps + fs:
        y.close()
