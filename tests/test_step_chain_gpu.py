"""Plain steps replayed several to a graph against the same steps one by one:
cold start, rebuilds, averages and a run that ends inside a chain."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import RunConfig, System, crystal
from fuller_md_en_b200.api import mm_replica

pytestmark = pytest.mark.gpu


def _system(ctx, kind, nlup):
    if kind == "mm":
        return mm_replica(ctx, 1, 300.0, 0.0, nlup=nlup, jitter=0.01)
    s = crystal.atomistic(1, jitter=0.01, seed=3, T=300.0)
    na = s["pos"].size // 3
    cfg = RunConfig(dt=0.5, T=300.0, Pe=0.0, coldstart=9, warmup=4, nsteps=200, nlup=nlup, gavg_from=20, gavg_to=150,
                    nc=1, nmol=s["nmol"])
    return System.airebo(ctx, cfg, s["pos"], s["vel"], s["mass"], s["mol_id"], s["h"],
                         crystal.npt_atom(300.0, 0.0, na))


# The same kernels on the same data, none of which adds by atomics in an order
# of its own: 1e-12 of the largest value leaves room for nothing but that.
@pytest.mark.parametrize("kind,nlup,last", [("airebo", 20, 133), ("airebo", 7, 100), ("airebo", 3, 80), ("mm", 25, 90)])
def test_chained_steps_are_the_same_steps(ctx, kind, nlup, last):
    got = []
    for chained in (True, False):
        y = _system(ctx, kind, nlup)
        y.init()
        if chained:
            o = y.run(1, last)
        else:
            for g in range(1, last + 1):
                o = y.run(g, g)
        d = y.download()
        got.append((o.step, np.array([o.T, o.P, o.a, o.KE, *o.E]), d["pos"].copy(), d["vel"].copy(), d["h"].copy()))
        y.close()
    assert got[0][0] == got[1][0] == last
    for a, b in zip(got[0][1:], got[1][1:]):
        assert np.abs(a - b).max() <= 1e-12 * max(1.0, np.abs(b).max())
