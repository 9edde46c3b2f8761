"""GPU parity of the flat step kernels (fdtd_flat_*.cu) at the sizes where their
work lists can go wrong, through the C ABI against the FP64 CPU oracle: k rows
of every remainder of the vector width, slabs that end inside a group, slabs of
both sides in one group or one box, faces without CPML, and boxes of less than
a block.  Random initial fields, so that every cell is active.

Tolerance: relative L2 1e-5 for FP32, 1e-10 for FP64 fields (the tolerances of
the other parity tests)."""
import numpy as np
import pytest

from gsvit_copy_b200 import abi, plan
from gsvit_copy_b200.solver import Batch, Solver
from oracle.pyoracle import CpuSolver
from tests._util import rel_l2, random_fields

pytestmark = pytest.mark.gpu

# shape, CPML depth, faces with CPML (x0 xn y0 yn z0 zn)
ALL = (0, 1, 2, 3, 4, 5)
CASES = [((24, 20, 28), 5, ALL), ((23, 22, 29), 6, ALL), ((25, 21, 30), 7, ALL), ((22, 26, 27), 8, ALL),
         ((20, 21, 20), 9, ALL),          # z slabs less than a group apart
         ((16, 16, 32), 8, ALL),          # x and y slabs that meet
         ((24, 28, 32), 6, (0, 3, 4)), ((24, 28, 32), 6, (1, 2, 5)), ((21, 23, 25), 4, (4, 5)), ((40, 36, 64), 10, ALL)]


def _scene(kind, shape, depth, faces, storage):
    s = plan.small_scene(kind, shape=shape, nsteps=24)
    s.cpml = {f: c for f, c in plan.cpml_all(depth, 3, -1, 2.0, 0.02, s.dx).items() if f in faces}
    s.tsf["box"] = ((4, 4, 5), (shape[0] - 5, shape[1] - 4, shape[2] - 6))
    s.nfff = None
    s.probes = np.asarray([(1, 2, 3), (shape[0] - 2, shape[1] - 2, shape[2] - 2)], dtype=np.int32)
    s.storage = storage
    return s


@pytest.mark.parametrize("storage,tol", [(abi.STORE_F32, 1e-5), (abi.STORE_F64, 1e-10)], ids=["f32", "f64"])
@pytest.mark.parametrize("kind", ["lintab", "full"])
@pytest.mark.parametrize("shape,depth,faces", CASES)
def test_flat_random_state_parity(shape, depth, faces, kind, storage, tol):
    s = _scene(kind, shape, depth, faces, storage)
    g, o = Solver(s), CpuSolver(s)
    init = random_fields(shape, 31)
    g.set_fields(init)
    o.set_fields(init)
    g.step(24)
    o.step(24)
    errs = [rel_l2(a, b) for a, b in zip(g.fields(), o.fields())]
    assert max(errs) < tol, errs
    assert rel_l2(g.probes(), o.probes()) < tol
    g.close()
    o.close()


def test_flat_batch_of_mixed_widths_bitwise():
    """Instances of vector and of single-cell rows in one batch, against each alone."""
    scenes = [_scene("full", sh, d, f, abi.STORE_F32) for sh, d, f in CASES[:6]]
    batch = Batch(scenes)
    for q, (v, sc) in enumerate(zip(batch.views, scenes)):
        v.set_fields(random_fields((sc.xres, sc.yres, sc.zres), 60 + q))
    batch.step(11)
    batch.sync()
    for q, sc in enumerate(scenes):
        alone = Solver(sc)
        alone.set_fields(random_fields((sc.xres, sc.yres, sc.zres), 60 + q))
        alone.step(11)
        for x, y in zip(batch[q].fields(dtype=np.float32), alone.fields(dtype=np.float32)):
            assert np.array_equal(x, y)
        alone.close()
    batch.close()
