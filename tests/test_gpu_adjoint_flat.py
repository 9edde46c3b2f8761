"""The transposed step's group kernels at the sizes where they can go wrong --
k rows of every remainder of the vector width, CPML depths that end inside a
group, slabs that meet, faces without CPML -- against the FP64 transpose
(oracle/adjoint.py); relative L2 1e-5, as the other transpose tests."""
import numpy as np
import pytest

from gsvit_copy_b200 import plan
from gsvit_copy_b200.solver import Solver
from oracle.adjoint import LinearStep
from oracle.pyoracle import CpuSolver
from tests._util import rel_l2, random_fields

pytestmark = pytest.mark.gpu

ALL = (0, 1, 2, 3, 4, 5)


@pytest.mark.parametrize("shape,depth,faces", [((18, 16, 20), 5, ALL), ((17, 18, 21), 6, ALL), ((16, 17, 22), 4, ALL),
                                               ((18, 18, 16), 8, ALL), ((20, 18, 24), 4, (0, 3, 4)), ((18, 20, 23), 5, (1, 2, 5))])
def test_transposed_step(shape, depth, faces):
    s = plan.small_scene("lintab", shape=shape, nsteps=8)
    s.mat[:] = 0
    s.mat[6:10, 5:9, 7:11] = 1
    s.cpml = {f: c for f, c in plan.cpml_all(depth, 3, -1, 2.0, 0.02, s.dx).items() if f in faces}
    s.tsf = None
    s.nfff = None
    s.probes = np.asarray([(3, 3, 3)], dtype=np.int32)
    g, o = Solver(s), CpuSolver(s)
    step = LinearStep(o)
    init = random_fields(shape, 12)
    st = step.zero_state()
    for c in range(3):
        st["E"][c][:], st["H"][c][:] = init[c], init[3 + c]
    for _ in range(4):
        step.adjoint(st)
    out = g.adjoint_transpose(init, 4)
    for c in range(3):
        assert rel_l2(out[c], st["E"][c]) < 1e-5
        assert rel_l2(out[3 + c], st["H"][c]) < 1e-5
    g.close()
