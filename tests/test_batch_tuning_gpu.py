"""The batch tuner's cached shapes belong to the kernels they were timed on: a
batch over rows of atoms does not take those of a batch of the same size over
cluster rows, nor the other way round."""
from __future__ import annotations

import pytest

from fuller_md_en_b200 import Batch, mm_replica
from fuller_md_en_b200._lib import FMD_PREC_FP32_PAIR, FMD_PREC_FP64

pytestmark = pytest.mark.gpu


def test_shapes_by_kernel(ctx):
    def tuning(delta, prec):
        reps = [mm_replica(ctx, 2, 200.0, 0.0, seed=k, precision=prec) for k in (61, 62, 63)]
        for y in reps:
            y.set_lj_prune(delta)
        b = Batch(ctx, reps)
        t = b.tuning()
        b.run(1, 2)
        b.close()
        for y in reps:
            y.close()
        return t
    clus, atoms, again, single = (tuning(d, p) for d, p in ((0.5, FMD_PREC_FP64), (0.0, FMD_PREC_FP64),
                                                            (0.5, FMD_PREC_FP64), (0.5, FMD_PREC_FP32_PAIR)))
    assert clus["lj_atoms_per_block"] == again["lj_atoms_per_block"] == single["lj_atoms_per_block"] == 144
    assert clus["lj_threads"] == again["lj_threads"] == 384 and single["lj_threads"] == 256
    assert atoms["lj_atoms_per_block"] in (8, 16, 32, 64) and atoms["lj_threads"] in (128, 256)
    assert again["lj_ms"] == clus["lj_ms"] > 0                  # cached
