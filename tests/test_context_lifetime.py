"""Handles are destroyed once and before their context, in whatever order their
objects are closed or collected (a stand-in for the library notes the calls)."""
from __future__ import annotations

import gc

import pytest

from fuller_md_en_b200 import Batch, Context, System


class _Lib:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda h: self.calls.append((name, h))


def _context(lib):
    c = Context.__new__(Context)
    c.lib, c.h, c._owned = lib, "ctx", {}
    return c


def _system(ctx, h):
    return System(ctx, h, 1, 0)


def _batch(ctx, h, systems):
    b = Batch.__new__(Batch)
    b.ctx, b.systems, b.h = ctx, systems, h
    ctx.adopt(b)
    return b


def _make(lib):
    ctx = _context(lib)
    a, b = _system(ctx, "a"), _system(ctx, "b")
    return ctx, a, b, _batch(ctx, "ab", [a, b])


ALL = [("fmd_batch_destroy", "ab"), ("fmd_ctx_destroy", "ctx"), ("fmd_system_destroy", "a"),
       ("fmd_system_destroy", "b")]


@pytest.mark.parametrize("order", ["ctx first", "ctx last", "cycle"])
def test_each_handle_once_and_before_the_context(order):
    lib = _Lib()
    ctx, a, b, ab = _make(lib)
    if order == "ctx first":
        ctx.close()
        for o in (a, b, ab, ctx):
            assert not o.h
            o.close()
    elif order == "ctx last":
        for o in (b, ab, a, ctx):
            o.close()
    else:                                # one garbage cycle: finalised in the collector's order
        ring = {"all": (ctx, a, b, ab)}
        for o in ring["all"]:
            o.ring = ring
        del ring, o
    del ctx, a, b, ab
    gc.collect()
    assert sorted(lib.calls) == ALL and lib.calls[-1] == ("fmd_ctx_destroy", "ctx"), lib.calls
