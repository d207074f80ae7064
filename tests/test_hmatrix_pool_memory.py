"""Device memory of the H-matrix construction: when a factor or near-field pool cannot grow, the
workspace that is kept between batches of blocks is given back and the growth is tried again (the
failure is injected on the host, no allocation runs out)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# batches of at most 16 MiB and blocks of at most 8 MiB: the allocations of 24 MiB and more are
# those of the pools, which double from 8 MiB
@pytest.mark.parametrize("size", [24 << 20, 48 << 20, 100 << 20])
def test_pool_growth_gives_the_workspace_back(size, monkeypatch):
    import torch
    import spinfemx_b200 as spx
    from spinfemx_b200 import _lib, hmatrix
    monkeypatch.setattr(hmatrix, "MIN_WORKSPACE", 1 << 60)  # no second build with half the workspace
    geom = spx.BoundaryGeometry(*spx.kuhn_box(70, 70, 2, 2.5))
    cfg = spx.HMatrixBuildConfig(epsilon=1e-6, leaf_size=64, batch_bytes=16 << 20,
                                 max_temporary_block_bytes=8 << 20)
    a = spx.HMatrixGPUPackedFused(geom, cfg, precision="f64")
    x = torch.as_tensor(np.random.default_rng(3).standard_normal(geom.Nb), device="cuda")
    y = a.matvec(x)
    try:
        _lib.call("spx_debug_fail_alloc", size, 1)
        b = spx.HMatrixGPUPackedFused(geom, cfg, precision="f64")
    finally:
        _lib.call("spx_debug_fail_alloc", 0, 0)
    assert torch.equal(b.matvec(x), y)
