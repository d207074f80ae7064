"""Several right-hand sides at once where a block's V^T row has more 16-byte vectors than a warp has
lanes (FP64 ranks above 64, FP32 ranks above 128), beside blocks of one strip (BF16: all of
them): every state against the single-vector product with the same factors, in every chunk of
states and with blocks that one warp and several warps share."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def geom():
    import spinfemx_b200 as spx
    return spx.BoundaryGeometry(*spx.kuhn_box(40, 40, 2, 2.5))


# both sides add FP64 products of the same factors in other orders
@pytest.mark.parametrize("precision", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("leaf", [128, 400])
def test_matmat_equals_matvecs(geom, precision, leaf):
    import torch
    import spinfemx_b200 as spx
    H = spx.HMatrixGPUPackedFused(geom, spx.HMatrixBuildConfig(epsilon=1e-11, eta=10.0, leaf_size=leaf),
                                  precision=precision)
    assert H.max_rank > 128
    X = torch.as_tensor(np.random.default_rng(2).standard_normal((11, geom.Nb)), device="cuda")
    y = torch.stack([H.matvec(x) for x in X])
    for R in (1, 2, 3, 4, 7, 8, 11):
        Y = H.matmat(X[:R])
        assert float(((Y - y[:R]).norm(dim=1) / y[:R].norm(dim=1)).max()) < 1e-13, R
        assert torch.equal(Y, H.matmat(X[:R]))
