"""Chebyshev.c_op gives every caller a C operator of its own (no GPU: matrices are
stand-ins that carry a handle)."""
from __future__ import annotations

from types import SimpleNamespace

from rsatb_b200.calc import Chebyshev


def _cheby(handle=7):
    return Chebyshev(SimpleNamespace(shape=(4, 4), handle=handle), -1.0, 3.0)


def test_a_callers_change_stays_in_its_own_operator():
    c = _cheby()
    mine = c.c_op()
    mine.center, mine.half_width, mine.H = 100.0, 1.0, 9
    op = c.c_op()
    assert (op.center, op.half_width, op.H) == (1.0, 2.0, 7)
    op = c._op()
    assert (op.center, op.half_width, op.H) == (1.0, 2.0, 7)


def test_the_kept_operator_follows_the_object():
    c = _cheby()
    assert c._op() is c._op()
    c.set_window(-2.0, 2.0)
    assert (c._op().center, c._op().half_width) == (0.0, 2.0)
    c.H = SimpleNamespace(shape=(4, 4), handle=11)
    assert c._op().H == 11
