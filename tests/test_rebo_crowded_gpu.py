"""REBO of molecules with more than four bonds an atom, with rows cut at the
list's width so that i lists j while j's row lacks i: forces, energy and virial
against the oracle, the gradient form against the slot kernels (which the same
atoms in an interleaved order take), and the same bits on every run."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rows
from fuller_md_en_b200 import crystal
from test_rebo_mol_gpu import _system

pytestmark = pytest.mark.gpu


def _missing(cnt, lst):
    r = rows(cnt, lst, 12)
    sets = [set(x) for x in r]
    return sum(i not in sets[j] for i in range(len(r)) for j in r[i])


# As in test_rebo_mol_gpu.py: each force a sum of some tens of terms, some a
# hundred times the sum: 1e-12 of the largest force.
@pytest.mark.parametrize("S,nc", [(40, 1), (64, 2), (96, 1), (128, 1)])
def test_cut_rows_match_oracle(ctx, oracle, S, nc):
    y, na = _system(ctx, "dense", S, nc, False)
    y.run(1, 1)
    F, _, E = y.forces()
    W, _ = y.virial()
    st = y.download()
    ca, la, cb, lb = y.lists(400, 12)
    y.close()
    assert _missing(cb, lb) > S // 4                       # bonds whose far end does not list them
    Er, Fr, Wr = oracle.airebo_forces(st["pos"], st["h"], crystal.inv9(st["h"]), cb, lb, ca, la, na)
    big = np.abs(Fr).max()
    assert abs(E[1] - Er[1]) <= 1e-12 * np.abs(Er[1]) and np.abs(F - np.ravel(Fr)).max() <= 1e-12 * big
    assert np.abs(W - Wr).max() <= 1e-12 * big * na


@pytest.mark.parametrize("S", [40, 64, 128])
def test_gradient_of_cut_rows_matches_slot_kernels(ctx, S):
    got = []
    na = 4 * S
    order = np.arange(na).reshape(-1, S).T.reshape(-1)     # atom 0 of every molecule, atom 1, ...
    for o in (np.arange(na), order):
        y, _ = _system(ctx, "dense", S, 1, True, o)
        F, _, E = y.forces()
        W, _ = y.virial()
        cb, lb = y.lists(400, 12)[2:]
        y.close()
        assert _missing(cb, lb) > S // 4
        G = np.empty((na, 3))
        G[o] = F.reshape(-1, 3)
        got.append((G, E, W))
    (F, E, W), (Fr, Er, Wr) = got
    assert np.abs(F - Fr).max() <= 1e-12 * np.abs(Fr).max() and abs(E[1] - Er[1]) <= 1e-12 * abs(Er[1])
    assert np.abs(W - Wr).max() <= 1e-12 * np.abs(Fr).max() * na


@pytest.mark.parametrize("kind,S,phys", [("cubic", 27, False), ("cubic", 64, True), ("dense", 64, False),
                                         ("dense", 64, True)])
def test_same_bits_on_every_run(ctx, kind, S, phys):
    first = None
    for _ in range(4):
        y, _ = _system(ctx, kind, S, 2, phys)
        y.run(1, 8)
        out = [y.forces()[0], y.forces()[2], y.virial()[0], y.download()["pos"], y.download()["vel"]]
        y.close()
        first = first or out
        for a, b in zip(out, first):
            assert np.array_equal(a, b)
