"""Probe rows: row n holds the fields at the probe cells after step n.  A call
that steps records the row of the last step before it again, from the fields as
they are then (the caller may have restored or set them), and a call of no steps
does just that.  Exact: probes and fields are read from the same arrays."""
import numpy as np
import pytest

from gsvit_copy_b200 import abi, plan
from gsvit_copy_b200.solver import Solver
from tests._util import random_fields

pytestmark = pytest.mark.gpu


def _scene(tsf):
    s = plan.small_scene("lintab", nsteps=24)
    if not tsf:
        s.tsf = None
    return s


def _at_probes(g, s):
    f = g.fields()
    return np.array([[a[tuple(p)] for a in f] for p in s.probes])


STEPS = {"eager": lambda g, n: g.step(n), "graph": lambda g, n: g.step_graph(n, 4),
         "static": lambda g, n: abi.check(g.lib.fdtd_step_static_scratch(g.h, n)),
         "timed": lambda g, n: g.step_timed(n), "profile": lambda g, n: g.step_profile(n)}


@pytest.mark.parametrize("tsf", [True, False], ids=["tsf", "dark"])
@pytest.mark.parametrize("how", STEPS)
def test_rows_across_calls(how, tsf):
    s = _scene(tsf)
    shape = (s.xres, s.yres, s.zres)
    g = Solver(s)
    g.set_fields(random_fields(shape, 2))
    g.step(6)
    row = _at_probes(g, s)
    snap = bytes(g.snapshot())
    STEPS[how](g, 5)                       # rows 6 .. 10
    assert np.array_equal(g.probes()[:, 5], row)
    whole, last = g.probes(), _at_probes(g, s)
    assert np.array_equal(whole[:, 10], last)
    h = Solver(s)                          # the restored plan has no rows yet
    h.restore(bytearray(snap))
    STEPS[how](h, 5)
    got = h.probes()
    assert not got[:, :5].any()
    assert np.array_equal(got[:, 5:], whole[:, 5:])
    g.set_fields(random_fields(shape, 3))  # row 10 follows the fields the next call starts from
    new = _at_probes(g, s)
    STEPS[how](g, 1)
    got = g.probes()
    assert np.array_equal(got[:, 10], new)
    assert np.array_equal(got[:, :10], whole[:, :10])
    g.close()
    h.close()


def test_no_steps_record_the_current_row():
    s = _scene(True)
    shape = (s.xres, s.yres, s.zres)
    g = Solver(s)
    g.step(4)
    for q, how in enumerate(("eager", "graph", "static")):
        g.set_fields(random_fields(shape, 5 + q))
        STEPS[how](g, 0)
        assert np.array_equal(g.probes()[:, 3], _at_probes(g, s))
        assert not g.probes()[:, 4:].any()
    g.close()
