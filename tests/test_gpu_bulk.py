"""The TMA bulk kernel over the interior beside the flat H kernel, then the flat E
kernel: the path of FP32 grids of 25 M cells and more and of 16-bit grids of any
size, here on small uneven grids (GSVIT_B200_BULK=1), whose interior boxes end
off the tiles' edges.  Poles, PEC, lossy and design cells in the box and on its
rim; eager, replayed and batched, with TSF, probes and NFFF on their side streams.

Tolerance: relative L2 against the FP64 oracle 1e-5 (FP32), 5e-3 (FP16: 40 steps
of white noise, as in test_gpu_storage.py); bit for bit between the ways to step."""
import numpy as np
import pytest

from gsvit_copy_b200 import abi, plan
from gsvit_copy_b200.solver import Batch, Solver
from oracle.pyoracle import CpuSolver, series_spectrum
from tests._util import rel_l2, random_fields

pytestmark = pytest.mark.gpu
TOL = {abi.STORE_F32: 1e-5, abi.STORE_F16: 5e-3}
STORES = [pytest.param(abi.STORE_F32, id="f32"), pytest.param(abi.STORE_F16, id="f16")]
CASES = [("full", (40, 52, 72), 5), ("full", (33, 47, 64), 7), ("ade", (25, 21, 40), 6), ("lintab", (18, 70, 24), 4)]


@pytest.fixture(autouse=True)
def _bulk_on(monkeypatch):
    monkeypatch.setenv("GSVIT_B200_BULK", "1")


def _scene(kind, shape, depth, storage=abi.STORE_F32, nsteps=40):
    s = plan.small_scene(kind, shape=shape, nsteps=nsteps)
    s.cpml = plan.cpml_all(depth, 3, -1, 2.0, 0.02, s.dx)
    m = depth + 3
    s.tsf["box"] = ((m, m, m), tuple(n - m for n in shape))
    s.nfff["box"] = ((m - 1,) * 3, tuple(n - m + 1 for n in shape))
    s.storage = storage
    return s


def _bulk_steps(g):
    """1D grid, TSF faces, flat H, bulk, flat E, NFFF samples and fold."""
    return int(g.step_profile(1)["launches_per_step"]) == 7


@pytest.mark.parametrize("storage", STORES)
@pytest.mark.parametrize("kind,shape,depth", CASES)
def test_random_state_parity(kind, shape, depth, storage):
    s = _scene(kind, shape, depth, storage)
    g, o = Solver(s), CpuSolver(s)
    init = random_fields(shape, 12)
    g.set_fields(init)
    o.set_fields(init)
    g.step(17)
    g.step_graph(23, 6)
    o.step(40)
    errs = [rel_l2(a, b) for a, b in zip(g.fields(), o.fields())]
    assert max(errs) < TOL[storage], errs
    assert rel_l2(g.probes(), o.probes()) < TOL[storage]
    ref = series_spectrum(o.nfff_series(), s.nfff["omega"], s.dt)
    assert rel_l2(g.nfff_spectrum(), ref) < TOL[storage]
    assert _bulk_steps(g)
    g.close()
    o.close()


def test_design_cells_vs_oracle():
    s = plan.adjoint_scene(shape=(32, 32, 32), cpml_depth=6, design_shape=(4, 4, 2), glass_cells=3, nsteps=250,
                           pulse_delay=2e-15, pulse_width=0.7e-15, seed=3)
    obj = plan.cone_objective(s, nth=5, nph=7)
    g, o = Solver(s), CpuSolver(s.expanded())
    assert obj and _bulk_steps(Solver(s))
    g.step(250)
    o.step(250)
    fg, fo = g.fields(), o.fields()
    for sl in (slice(0, 3), slice(3, 6)):   # E and H as vector fields
        assert rel_l2(np.stack(fg[sl]), np.stack(fo[sl])) < 1e-5
    assert rel_l2(g.nfff_spectrum(), series_spectrum(o.nfff_series(), s.nfff["omega"], s.dt)) < 1e-5


@pytest.mark.parametrize("storage", STORES)
def test_replay_and_batch_give_the_bits_of_single_steps(storage):
    """fdtd_step one by one, fdtd_step in one call, fdtd_step_graph, and a batch."""
    scenes = [_scene(k, sh, d, storage) for k, sh, d in CASES]

    def out(g):
        return g.fields(dtype=np.float32) + [g.probes(), g.nfff_spectrum()]

    ways = {"singly": lambda g: [g.step(1) for _ in range(26)], "call": lambda g: g.step(26), "graph": lambda g: g.step_graph(26, 8)}
    want = []
    for q, s in enumerate(scenes):
        init = random_fields((s.xres, s.yres, s.zres), 70 + q)
        for way, steps in ways.items():
            with Solver(s) as g:
                g.set_fields(init)
                steps(g)
                if way == "singly":
                    want.append(out(g))
                else:
                    assert all(np.array_equal(a, b) for a, b in zip(out(g), want[q])), (way, q)
    b = Batch(scenes)
    for q, s in enumerate(scenes):
        b[q].set_fields(random_fields((s.xres, s.yres, s.zres), 70 + q))
    assert b.config()["items"] > 0
    b.step(14)
    b.step_graph(12, chunk=4)
    for q in range(len(scenes)):
        assert all(np.array_equal(x, y) for x, y in zip(out(b[q]), want[q])), q
    b.close()
