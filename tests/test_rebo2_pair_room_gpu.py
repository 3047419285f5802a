"""The list of close pairs of the switched LJ term takes 64 pairs an atom, all
within 2^(1/6) sigma: a system with exactly as many and one pair barely beyond
is accepted."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import Rebo2Knots, RunConfig, System, crystal
from fuller_md_en_b200._lib import FMD_REBO2_LJ_SWITCH

pytestmark = pytest.mark.gpu


def test_full_room_and_a_pair_beyond_the_radius(ctx):
    rng = np.random.default_rng(2)
    rmax = 2.0 ** (1.0 / 6.0) * 3.40
    ball = lambda c: np.array(c) + (v := rng.normal(size=(128, 3))) / np.linalg.norm(v, axis=1)[:, None] * 0.5
    c = np.array([-3.0, 0.0, 0.0])
    pos = np.concatenate([ball([0, 0, 0]), ball([1.5, 0, 0]), [c], [c - [np.sqrt(rmax ** 2 + 0.004), 0, 0]]]) + 20.0
    mol = np.repeat([1, 2, 3, 4], [128, 128, 1, 1]).astype(np.int32)
    na = len(pos)
    d2 = ((pos[:, None] - pos[None]) ** 2).sum(-1)
    pairs = (mol[:, None] < mol[None]) & (d2 < rmax ** 2)
    assert pairs.sum() == 64 * na                                   # the room
    assert ((mol[:, None] < mol[None]) & (d2 < rmax ** 2 + 0.01)).sum() == 64 * na + 1
    cfg = RunConfig(dt=1e-4, T=1.0, Pe=0.0, nsteps=10, nlup=5, nc=1, nmol=4)
    h = np.diag([40.0] * 3).reshape(-1)
    y = System.airebo(ctx, cfg, pos.reshape(-1), np.zeros(3 * na), np.full(na, crystal.MC), mol, h,
                      crystal.npt_atom(1.0, 0.0, na))
    y.set_rebo2(Rebo2Knots(), FMD_REBO2_LJ_SWITCH)
    y.init()                                                        # a capacity error before
    assert np.isfinite(y.forces()[0]).all()
    y.close()
