"""Plans of their own in several host threads: stepping, capturing and replaying in
one while another creates and destroys plans.  Bit for bit the plan stepped alone."""
import threading

import numpy as np
import pytest

from gsvit_copy_b200 import plan
from gsvit_copy_b200.solver import Batch, Solver
from tests._util import random_fields

pytestmark = pytest.mark.gpu


def test_plans_are_made_while_another_thread_captures():
    s = plan.small_scene("full", nsteps=200)
    init = random_fields((s.xres, s.yres, s.zres), 14)

    def run(g, n):   # another chunk each call: a new graph each call
        for q in range(n):
            g.step_graph(8, (2, 4)[q & 1])
        return g.fields(dtype=np.float32) + [g.probes(), g.nfff_spectrum()]

    with Solver(s) as g:
        g.set_fields(init)
        want = run(g, 24)
    errors, got, stop = [], {}, threading.Event()

    def guard(f, *a):
        try:
            f(*a)
        except Exception as e:
            errors.append(e)
            stop.set()

    def capture(k):
        with Solver(s) as g:
            g.set_fields(init)
            got[k] = run(g, 24)

    def create():
        while not stop.is_set():
            with Solver(s) as g:
                g.step_profile(1)
            Batch([s, s]).close()

    maker = threading.Thread(target=guard, args=(create,))
    takers = [threading.Thread(target=guard, args=(capture, k)) for k in range(2)]
    for t in [maker, *takers]:
        t.start()
    for t in takers:
        t.join()
    stop.set()
    maker.join()
    assert not errors, errors
    for k in got:
        assert all(np.array_equal(a, b) for a, b in zip(got[k], want)), k
    assert len(got) == 2
