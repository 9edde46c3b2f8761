"""The bench's per-kernel block names the kernels that ran, which the launches of a
profiled step tell, and gives a kernel's profiled DRAM bytes to that kernel alone."""
import pytest

import bench


@pytest.mark.parametrize("launches,inner,rest", [(8, "tile_kernel, bulk", "tile_kernel, CPML"),
                                                 (7, "tile_kernel, bulk", "flat_h_kernel"),
                                                 (6, "flat_h_kernel", "flat_h_kernel")])
def test_kernels_by_launches(launches, inner, rest, monkeypatch):
    monkeypatch.setattr(bench, "ncu_traffic", lambda res, kernel="bulk_kernel": 5.0e9)
    prof = dict(bulk_ms=3.0, bulk_bytes=6e9, slab_ms=1.0, slab_bytes=2e9, aux_ms=0.1, nfff_ms=0.2, total_ms=4.3,
                launches_per_step=float(launches))
    roof, ks, step = bench.kernel_rooflines(prof, 2, 8e9, 2.0, 6500.0, "measured", 512)
    assert ks["bulk"]["kernel"].startswith(inner) and ks["cpml"]["kernel"].startswith(rest)
    assert roof["kernel"] == ks["bulk"]["kernel"]
    assert roof["traffic"] == (None if launches == 6 else 5.0e9)
    assert roof["frac"] == pytest.approx(6e9 / 1.5e-3 / 6500e9) and step["achieved"] == pytest.approx(4000.0)
