"""Through a fake of a runtime call, in a child process.

A launch that fails in the middle of a stepping call (nothing is launched in its
place): the plan stays at the last step queued whole, its field set, step count,
device counter (probe rows), far-field sums and replay graphs agreeing, and steps
on from there to the bits of a run without the failure.  The scene has no TSF
box: the 1D grid alone runs ahead of the steps."""
import pytest

from tests._fakecuda import run_child

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes, os, sys
import numpy as np
from gsvit_copy_b200 import abi, plan
from gsvit_copy_b200.solver import Solver
from tests._util import random_fields
fake = ctypes.CDLL(os.environ["LD_PRELOAD"])
s = plan.small_scene("full", nsteps=24)
s.tsf = None
init = random_fields((s.xres, s.yres, s.zres), 6)

def out(g):
    return g.fields(dtype=np.float32) + [g.probes(), g.nfff_spectrum()]

with Solver(s) as w:
    w.set_fields(init)
    w.step(12)
    want = out(w)
static = lambda g, n: abi.check(g.lib.fdtd_step_static_scratch(g.h, n))
for how, step, done in (("eager", lambda g, n: g.step(n), 3), ("static", static, 3),
                        ("graph", lambda g, n: g.step_graph(n, 8), 0)):
    with Solver(s) as g:
        g.set_fields(init)
        fake.fake_arm(4)
        try:
            step(g, 9)
            sys.exit("the launch did not fail")
        except abi.FdtdError as e:
            assert "launch" in str(e), e
        assert g.step_count == done, g.step_count
        step(g, 12 - done)
        assert g.step_count == 12
        same = [np.array_equal(a, b) for a, b in zip(out(g), want)]
        assert all(same), (how, same)
print("agree")
"""


def test_plan_after_a_failed_launch(tmp_path):
    run_child(CHILD, tmp_path)


PROFILE = r"""
import ctypes, os
from gsvit_copy_b200 import plan
from gsvit_copy_b200.solver import Solver
fake = ctypes.CDLL(os.environ["LD_PRELOAD"])
s = plan.small_scene("full", shape=(40, 52, 72))
with Solver(s) as g:
    made = fake.fake_mallocs()
    g.step(2)
    assert fake.fake_mallocs() == made
    first = g.step_profile(1)
    assert fake.fake_mallocs() == made + 2      # the block lists of the interior and of the rest
    again = g.step_profile(1)
    assert fake.fake_mallocs() == made + 2
    assert first["bulk_bytes"] == again["bulk_bytes"] > 0 and first["slab_bytes"] == again["slab_bytes"] > 0
print("agree")
"""


def test_profile_makes_its_own_lists(tmp_path):
    """What fdtd_step_profile alone needs is made by its first call, not with the plan."""
    run_child(PROFILE, tmp_path)
