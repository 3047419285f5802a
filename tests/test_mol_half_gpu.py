"""Half rows and full-row tables from candidate bitmaps (molnlist.cu) against
the oracle's lists: one and four atoms a warp, molecules whose last group of
four is partial, cells where one image serves a partner molecule and cells
where each pair takes its own, rows that are truncated."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rows, same_rows
from fuller_md_en_b200 import RunConfig, System, crystal
from fuller_md_en_b200.api import Topology

pytestmark = pytest.mark.gpu


def _no_terms():
    z = lambda *k: np.zeros(k)
    return Topology(z(0, 2), z(0), z(0), z(0, 3), z(0), z(0), z(0, 4), z(0), z(0), z(0), z(0, 4), z(0), z(0))


@pytest.mark.parametrize("nc,S,a0,size", [
    (2, 32, 13.0, 1.0),                # one atom a warp
    (3, 45, 12.0, 1.7),
    (5, 45, 12.5, 1.0),                # four, the last group of one; one image a partner
    (4, 60, 13.0, 2.0),                # four, an image a pair
    (6, 33, 11.0, 1.0),
    (4, 64, 12.5, 1.7),
])
def test_rows_match_oracle(ctx, oracle, nc, S, a0, size):
    inner = np.array([[1, 1, 1], [-1, -1, 1], [1, -1, -1], [-1, 1, -1]], float)
    mol = size * np.concatenate([crystal.c60_ih(), inner])[:S]
    s = crystal.atomistic(nc, coords=mol, jitter=0.1, seed=nc + S, T=50.0, mol_base=0)
    na = s["pos"].size // 3
    f = a0 / s["a0"]
    h = s["h"] * f
    centres = np.repeat(s["pos"].reshape(-1, S, 3).mean(axis=1), S, axis=0)
    pos = (s["pos"].reshape(-1, 3) + (f - 1.0) * centres + 4.7).reshape(-1)
    cfg = RunConfig(dt=0.01, T=50.0, Pe=0.0, nsteps=100, nlup=1, nc=nc, nmol=s["nmol"])
    y = System.mm(ctx, cfg, pos, s["vel"], s["mol_id"], _no_terms(), h, crystal.npt_atom(50.0, 0.0, na))
    y.init()
    p, hh = pos, h
    for step in (0, 1):                # unwrapped positions, then the wrapped ones of a step's start
        if step:
            p, hh = (y.download()[k] for k in ("pos", "h"))
            y.run(1, 1)
        c, l = y.lists(400)[:2]
        oc, ol, _ = oracle.nlist_half_threaded(p, hh, crystal.inv9(hh), na, s["mol_id"], 3.0 * 3.431 + 2.0)
        assert np.array_equal(c, oc) and same_rows(rows(c, l, 400), rows(oc, ol, 400)), step
    y.close()
