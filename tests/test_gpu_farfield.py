"""The far-field kernels at the sizes where they can go wrong, against the FP64
oracle: one frequency, a full group of them and one more; points whose
retarded time falls on an integer (diagonals of the grid, where the Courant
ratio is rational), points in a surface cell itself, points of a block's second
half alone (129), one more than a block takes (257), a second block in part.  Relative L2 1e-5, as the other far-field tests (FP32 fields)."""
import numpy as np
import pytest

from gsvit_copy_b200 import plan
from gsvit_copy_b200.solver import Solver
from oracle.pyoracle import CpuSolver, series_spectrum
from tests._util import rel_l2

pytestmark = pytest.mark.gpu

NSTEPS = 120


def _scene(points, nfreq, shape=(28, 26, 30), series=False):
    s = plan.small_scene("lintab", shape=shape, nsteps=NSTEPS)
    pts = np.asarray(points, dtype=np.int32)
    s.nfff = dict(box=((6, 6, 6), tuple(n - 6 for n in shape)), points=pts,
                  istart=plan.nfff_istart(pts, s.dt, s.dx, shared=False),
                  omega=np.array([2 * np.pi * plan.C0 / w for w in np.linspace(400e-9, 900e-9, nfreq)]), series=series)
    return s


def _sphere(n, radius, centre=(14, 13, 15)):
    rng = np.random.default_rng(5)
    v = rng.standard_normal((n, 3))
    return np.rint(np.asarray(centre) + radius * v / np.linalg.norm(v, axis=1, keepdims=True)).astype(int)


DIAGONAL = [(6 + 40 * q, 6 + 40 * q, 6 + 40 * q) for q in range(1, 9)]


@pytest.mark.parametrize("nfreq", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("points", [DIAGONAL, _sphere(129, 90), _sphere(5, 3000), _sphere(257, 90), _sphere(400, 400)],
                         ids=["diagonal", "near", "far", "two_blocks", "two_blocks_far"])
def test_spectrum(points, nfreq):
    s = _scene(points, nfreq)
    g, o = Solver(s), CpuSolver(s)
    g.step(NSTEPS)
    o.step(NSTEPS)
    ref = series_spectrum(o.nfff_series(), s.nfff["omega"], s.dt)
    spec = g.nfff_spectrum()
    assert rel_l2(spec, ref) < 1e-5, rel_l2(spec, ref)
    g.close()
    o.close()


def test_point_in_a_surface_cell():
    """Its own value has r = 0 in it; the other points are as without it."""
    points = [tuple(p) for p in _sphere(6, 90)]
    a, b = Solver(_scene(points, 3)), Solver(_scene(points + [(6, 12, 12)], 3))
    for v in (a, b):
        v.step(NSTEPS)
    sa, sb = a.nfff_spectrum(), b.nfff_spectrum()
    assert rel_l2(sb[:6], sa) < 1e-12 and not np.isfinite(sb[6]).all()
    a.close()
    b.close()


@pytest.mark.parametrize("shape,points", [((20, 18, 400), [(10, 9, 900), (10, 9, -700)]),     # cells of a CTA that arrive far apart
                                          ((28, 26, 30), _sphere(3, 60)), ((28, 26, 30), _sphere(70, 400))],
                         ids=["long", "near", "many"])
def test_series(shape, points):
    s = _scene(points, 2, shape=shape, series=True)
    g, o = Solver(s), CpuSolver(s)
    g.step(NSTEPS)
    o.step(NSTEPS)
    ser, ref = g.nfff_series(), o.nfff_series()
    assert ser.shape == ref.shape
    assert rel_l2(ser, ref) < 1e-5, rel_l2(ser, ref)
    g.close()
    o.close()
