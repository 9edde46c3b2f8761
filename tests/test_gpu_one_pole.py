"""The E kernel of media with one pole and no Drude term (fdtd_flat_*.cu)
against the kernel that steps every term, bitwise: an unused material with a
Drude term sends the same grid to the latter.  Also after a restored state that
holds what the former takes for zero, alone and in a batch, step by step and
replayed."""
import numpy as np
import pytest

from gsvit_copy_b200 import abi, plan
from gsvit_copy_b200.solver import Batch, Solver
from oracle.pyoracle import CpuSolver
from tests._util import rel_l2, random_fields

pytestmark = pytest.mark.gpu

CASES = [((24, 20, 28), 5), ((23, 22, 29), 6), ((22, 26, 30), 7)]


def _scene(shape, depth, storage=abi.STORE_F32, general=False):
    s = plan.small_scene("ade", shape=shape, nsteps=24)
    one = plan.ade_material(2.0, 0.0, 0.0, 0.0, [plan.lorentz_as_cp(5.0, 2.0, 4e15, 1e14), (0, 0, 0, 0)], s.dt)
    drude = s.mats[-1]
    s.mats[-1] = one
    if general:
        s.mats.append(drude)
    s.cpml = plan.cpml_all(depth, 3, -1, 2.0, 0.02, s.dx)
    s.tsf["box"] = ((4, 4, 5), (shape[0] - 5, shape[1] - 4, shape[2] - 6))
    s.nfff = None
    s.storage = storage
    return s


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a.fields(), b.fields()))


@pytest.mark.parametrize("storage,tol", [(abi.STORE_F32, 1e-5), (abi.STORE_F64, 1e-10), (abi.STORE_F16, None)],
                         ids=["f32", "f64", "f16"])
@pytest.mark.parametrize("shape,depth", CASES)
def test_against_the_general_kernel(shape, depth, storage, tol):
    init = random_fields(shape, 17)
    runs = [Solver(_scene(shape, depth, storage, general)) for general in (False, True)]
    for v in runs:
        v.set_fields(init)
        v.step(24)
    assert _same(*runs)
    if tol:
        o = CpuSolver(_scene(shape, depth, storage))
        o.set_fields(init)
        o.step(24)
        assert max(rel_l2(x, y) for x, y in zip(runs[0].fields(), o.fields())) < tol
        o.close()
    for v in runs:
        v.close()


def _with_state(buf, shape, seed):
    """The snapshot with random Q, p and q of every term (FP32 plan: the 12
    field arrays, then Q, p0, q0, p1, q1 of each component)."""
    n = int(np.prod(shape))
    a = np.frombuffer(buf, dtype=np.float32, offset=8)
    a = a.copy()
    a[12 * n:27 * n] = 1e-14 * np.random.default_rng(seed).standard_normal(15 * n)
    return bytearray(bytes(buf[:8]) + a.tobytes())


@pytest.mark.parametrize("graph", [False, True])
def test_restored_state_takes_the_general_kernel(graph):
    shape, depth = CASES[0]
    one, ref = Solver(_scene(shape, depth)), Solver(_scene(shape, depth, general=True))
    empty = one.snapshot()
    go = (lambda v: v.step_graph(8, 4)) if graph else (lambda v: v.step(8))
    go(one)
    state = _with_state(empty, shape, 3)
    for v in (one, ref):
        v.restore(state)
        go(v)
    assert _same(one, ref)
    assert np.abs(one.fields()[0]).max() > 0
    for v in (one, ref):      # and back
        v.restore(empty)
        v.set_fields(random_fields(shape, 4))
        go(v)
    assert _same(one, ref)
    one.close()
    ref.close()


def test_batch():
    scenes = [_scene(sh, d) for sh, d in CASES]
    b, alone = Batch(scenes), [Solver(s) for s in scenes]
    for turn in range(2):
        for q, s in enumerate(scenes):
            state = alone[q].snapshot()
            if turn:
                state = _with_state(state, CASES[q][0], q)
            for v in (b[q], alone[q]):
                v.restore(state)
                v.set_fields(random_fields(CASES[q][0], 60 + q))
            alone[q].step(8)
        b.step_graph(8, 4)
        b.sync()
        for q in range(len(scenes)):
            assert _same(b[q], alone[q])
    b.close()
    for v in alone:
        v.close()
