"""A launch that fails in the middle of a stepping call, from a fake of the failing
runtime call in a child process (nothing is launched in its place): the plan
stays at the last step queued whole, its field set, step count, device counter
(probe rows), far-field sums and replay graphs agreeing, and steps on from there
to the bits of a run without the failure.  The scene has no TSF box: the 1D grid
alone runs ahead of the steps."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
static int left, pending;
void fake_arm(int k) { left = k; }            /* the k-th launch of the flat E kernel from now fails */
static void *real(const char *n) { return dlsym(dlopen("libcudart.so.12", RTLD_NOW | RTLD_NOLOAD), n); }
int cudaLaunchKernelExC(const void *c, const void *f, void **a)
{
    if (left > 0 && --left == 0) return pending = 701;   /* cudaErrorLaunchOutOfResources */
    return ((int (*)(const void *, const void *, void **))real("cudaLaunchKernelExC"))(c, f, a);
}
int cudaGetLastError(void)
{
    int e = pending;
    pending = 0;
    return e ? e : ((int (*)(void))real("cudaGetLastError"))();
}
"""

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
    src, so = tmp_path / "fake.c", tmp_path / "fake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "agree" in r.stdout, r.stdout + r.stderr
