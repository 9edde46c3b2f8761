"""Host copies that change the element type (fdtd_set_fields / fdtd_get_fields
and their FP32 forms) convert on the device, in chunks of the staging buffer
(2^22 doubles, 2^23 floats).  Against numpy / torch conversions, bit for bit, on
a grid of more than one chunk and on one smaller than a block: double to float,
then to the storage type to nearest (H times 2^9 at 16 bits); FP64 storage keeps
doubles."""
import ctypes as C

import numpy as np
import pytest
import torch

from gsvit_copy_b200 import abi, plan
from gsvit_copy_b200.solver import Solver
from tests._util import random_fields

pytestmark = pytest.mark.gpu


def _stored(x, storage, scale):
    if storage == abi.STORE_F64:
        return x
    f = x.astype(np.float32)
    if storage == abi.STORE_F32:
        return f.astype(np.float64)
    t = torch.float16 if storage == abi.STORE_F16 else torch.bfloat16
    v = torch.from_numpy(f * np.float32(scale)).to(t).to(torch.float32).numpy() / np.float32(scale)
    return v.astype(np.float64)


@pytest.mark.parametrize("storage", [abi.STORE_F32, abi.STORE_F16, abi.STORE_BF16, abi.STORE_F64],
                         ids=["f32", "f16", "bf16", "f64"])
@pytest.mark.parametrize("shape", [(9, 7, 5), (172, 170, 291)])   # 315 and 8.5 M cells
def test_round_trip_bits(shape, storage):
    dx = 10e-9
    s = plan.Scene(name="copy", xres=shape[0], yres=shape[1], zres=shape[2], dx=dx, dt=plan.plan_dt(dx, dx, dx, 0.5), nsteps=1)
    s.mats = [plan.vacuum_material()]
    s.mat = np.zeros(shape, dtype=np.int32)
    s.storage = storage
    g = Solver(s)
    init = random_fields(shape, 8)
    g.set_fields(init)
    want = [_stored(np.asarray(c, dtype=np.float64), storage, 1.0 if q < 3 else 512.0) for q, c in enumerate(init)]
    for a, b in zip(g.fields(), want):
        assert np.array_equal(a, b)
    for a, b in zip(g.fields(dtype=np.float32), want):
        assert np.array_equal(a, b.astype(np.float32))
    g.close()


def test_staging_is_made_by_the_first_copy_that_converts():
    """An FP32 plan read and set as FP32 holds no staging buffer (8 bytes a cell, at
    most 32 MB; device memory comes in pieces of 2 MB)."""
    n = 128
    s = plan.small_scene("lintab", shape=(n, n, n), nsteps=1)
    f = [np.zeros((n, n, n), dtype=np.float32) for _ in range(6)]
    free = lambda: torch.cuda.mem_get_info()[0]
    with Solver(plan.small_scene("lintab", nsteps=1)) as g:   # loads the conversion kernels
        g.set_fields(g.fields())
    with Solver(s) as g:
        a = free()
        abi.check(g.lib.fdtd_set_fields_f32(g.h, abi.EH, abi.field_ptrs(f, C.c_float)))
        g.fields(dtype=np.float32)
        b = free()
        g.fields()
        c = free()
        g.set_fields(f)
        g.fields()
        d = free()
    assert b >= a - (2 << 20)
    assert 8 * n ** 3 - (2 << 20) <= b - c <= 8 * n ** 3 + (2 << 20)
    assert d >= c - (2 << 20)


def test_error_returns_after_the_copies_queued_before_it():
    """Page-locked arrays, so that the copies are the device's alone (16 M cells: ms)."""
    shape = (256, 256, 256)
    s = plan.Scene(name="copy", xres=256, yres=256, zres=256, dx=10e-9, dt=plan.plan_dt(10e-9, 10e-9, 10e-9, 0.5), nsteps=1)
    s.mats = [plan.vacuum_material()]
    s.mat = np.zeros(shape, dtype=np.int32)
    st = torch.cuda.Stream()
    with Solver(s) as g:
        g.set_stream(st.cuda_stream)
        for dt, ct in ((torch.float64, C.c_double), (torch.float32, C.c_float)):
            host = torch.zeros(shape, dtype=dt).pin_memory().numpy()
            p = abi.field_ptrs([host, None, None, None, None, None], ct)
            f32 = "_f32" if dt == torch.float32 else ""
            for fn in ("fdtd_set_fields" + f32, "fdtd_get_fields" + f32):
                with pytest.raises(abi.FdtdError, match="NULL"):
                    abi.check(getattr(g.lib, fn)(g.h, 3, p), fn)
                assert st.query(), fn
        g.set_stream(None)
