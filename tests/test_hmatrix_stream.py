"""The single-vector H-matrix apply against the dense operator where its plan can go wrong: fewer
tiles than warps, segments cut between CTAs, ragged leaves, ranks past one vector per lane, every
packing, strided and offset inputs, and the partial-sum counters after repeated applies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _geom(nx, ny, nz):
    import spinfemx_b200 as spx
    return spx.BoundaryGeometry(*spx.kuhn_box(nx, ny, nz, 2.5))


# unit roundoff of the stored factors, plus the ACA tolerance; BF16 factors: 2^-9 relative to the
# largest block, as the packing states (1e-4 of the result at these sizes)
@pytest.mark.parametrize("dims,leaf", [((2, 2, 1), 64), ((5, 3, 2), 8), ((24, 24, 2), 64), ((31, 17, 3), 33),
                                       ((61, 40, 1), 17), ((48, 48, 2), 100)])
@pytest.mark.parametrize("precision,tol", [("f64", 2e-6), ("f32", 2e-6), ("mixed", 1e-4), ("f32_f16", 5e-6)])
def test_apply_matches_dense(dims, leaf, precision, tol):
    import torch
    import spinfemx_b200 as spx
    g = _geom(*dims)
    H = spx.HMatrixGPUPackedFused(g, spx.HMatrixBuildConfig(epsilon=1e-6, leaf_size=leaf), precision=precision)
    B = g.dense_B()
    rng = np.random.default_rng(dims[0])
    for _ in range(3):
        x = torch.as_tensor(rng.standard_normal(g.Nb + 1), device="cuda")[1:]  # 8-byte aligned only
        y, ref = H.matvec(x), B @ x
        assert float(torch.linalg.norm(y - ref) / torch.linalg.norm(ref)) < tol
    x = torch.as_tensor(rng.standard_normal((g.Nb, 2)), device="cuda")[:, 1]   # strided
    ref = B @ x
    assert float(torch.linalg.norm(H.matvec(x) - ref) / torch.linalg.norm(ref)) < tol
    assert torch.equal(H.matvec(x), H.matvec(x))  # fixed order of every sum
    assert H.tensor_core_status() == 0


def test_ranks_past_one_vector_per_lane():
    """Blocks of rank above 128 (FP64: more than 64 vectors of a V^T row) at a tight tolerance."""
    import torch
    import spinfemx_b200 as spx
    g = _geom(40, 40, 2)
    H = spx.HMatrixGPUPackedFused(g, spx.HMatrixBuildConfig(epsilon=1e-11, eta=10.0, leaf_size=128), precision="f64")
    assert H.max_rank > 128
    x = torch.as_tensor(np.random.default_rng(1).standard_normal(g.Nb), device="cuda")
    ref = g.dense_B() @ x
    assert float(torch.linalg.norm(H.matvec(x) - ref) / torch.linalg.norm(ref)) < 1e-9
