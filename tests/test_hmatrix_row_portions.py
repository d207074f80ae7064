"""The single-vector H-matrix apply where a CTA passes many row segments: more than its two buffers of
partial sums and more than its warps, which take turns at finishing a segment, with segments of
one to four rows whose chunks are fewer than the warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# unit roundoff of the stored entries plus the ACA tolerance (BF16 factors as the packing states)
@pytest.mark.parametrize("precision,tol", [("f64", 2e-6), ("f32", 2e-6), ("bf16", 1e-4)])
@pytest.mark.parametrize("dims,leaf", [((12, 10, 1), 4), ((30, 21, 1), 2), ((40, 33, 1), 3)])
def test_many_small_segments(dims, leaf, precision, tol):
    import torch
    import spinfemx_b200 as spx
    g = spx.BoundaryGeometry(*spx.kuhn_box(*dims, 2.5))
    H = spx.HMatrixGPUPackedFused(g, spx.HMatrixBuildConfig(epsilon=1e-6, leaf_size=leaf), precision=precision)
    x = torch.as_tensor(np.random.default_rng(leaf).standard_normal(g.Nb), device="cuda")
    ref = g.dense_B() @ x
    y = H.matvec(x)
    assert float((y - ref).norm() / ref.norm()) < tol
    for _ in range(20):
        assert torch.equal(H.matvec(x), y)
