"""The training kernels (k_sg_chain, k_sg_wgrad) where a thread block has one
and several tiles of 128 rows, and the last tile is partial: the loss gradient
against the FP64 restatement with the same BF16 rounding points."""
from __future__ import annotations

import numpy as np
import pytest

from fuller_md_en_b200 import crystal
from oracle import sg_oracle as sg


# Rounding to BF16 (2^-9) flips where FP32 and FP64 sums differ, and averages
# over rows: the bounds of the same comparison at 720 rows (3e-2, 0.999).
@pytest.mark.gpu
@pytest.mark.parametrize("nc", [1, 3, 4])   # 6, 152 and 360 tiles; the first two end in a partial one
def test_gradient_over_tiles(ctx, oracle, nc):
    from fuller_md_en_b200.surrogate import Surrogate
    s = crystal.atomistic(nc, T=300.0, seed=40 + nc, jitter=0.05)
    na = s["pos"].size // 3
    pos = s["pos"].copy()
    oracle.apply_pbc(pos, s["h"], s["hi"])
    cnt, lst, _ = oracle.nlist_intra(pos, s["h"], s["hi"], na, s["mol_id"])
    g = sg.rows(pos, s["h"], s["hi"], cnt, lst)
    X, _ = sg.descriptors(g)
    P = sg.init_params(5)
    P["m"], P["s"] = X.mean(0), X.std(0) + 1e-3
    bex = sg.exact_bond_order(g)
    P["b0"], P["bs"] = float(bex.mean()), float(bex.std())
    Er, Fr, Wr = oracle.rebo(pos, s["h"], s["hi"], cnt, lst, na)
    w = dict(wE=0.3, wF=1.0, wW=0.2)
    L, grads, _, _, _ = sg.loss_and_grad(P, g, Er, Fr, Wr, rnd=True, **w)
    S = Surrogate(ctx, P)
    Lg, gg = S.loss_grad(pos, s["h"], s["hi"], cnt, lst, Fr, Er, Wr, **w)
    S.close()
    assert abs(Lg - L) <= 2e-3 * L
    for k in ("W1", "W2", "W3", "w4"):
        a, b = gg[k].ravel(), grads[k].ravel()
        rel = np.linalg.norm(a - b) / np.linalg.norm(b)
        cos = a @ b / (np.linalg.norm(a) * np.linalg.norm(b))
        assert rel < 3e-2 and cos > 0.999, (k, rel, cos)
