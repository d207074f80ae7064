"""Dense boundary blocks of an ensemble where the row tiles and vector batches end raggedly: fewer
rows than a tile's warps take together, tiles of one row pair, rows shorter than a batch, row
lengths that are no multiple of a 16-byte vector.  Each sample against the sample on its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOXES = [(2, 2, 2), (3, 2, 2), (5, 4, 3), (6, 5, 2), (11, 3, 2), (15, 14, 2), (23, 17, 2)]


# both sides solve to 1e-12 of their right-hand sides; "mixed" adds FP32 operator entries (6e-8
# each) on the two sides
@pytest.mark.parametrize("precision,tol", [("f64", 1e-9), ("mixed", 2e-6)])
def test_dense_blocks_equal_single_samples(precision, tol):
    import torch
    import spinfemx_b200 as spx
    ms = [spx.kuhn_box(*b, 2.0) for b in BOXES]
    X, T, off = spx.ensemble_mesh(ms)
    kw = dict(precision=precision, ksp_rtol_u1=1e-12, ksp_rtol_u2=1e-12, ksp_atol=0.0)
    d = spx.DemagFieldLindholmGPU(X, T, 8e5, boundary_backend="ensemble", sample_offsets=off, dense_max_nb=4096, **kw)
    rng = np.random.default_rng(5)
    m = rng.normal(size=(X.shape[0], 3))
    m = torch.as_tensor((m / np.linalg.norm(m, axis=1)[:, None]).ravel(), device="cuda")
    H = torch.empty_like(m)
    d.compute_vec(m, H)
    for k, (Xs, Ts) in enumerate(ms):
        s = slice(3 * int(off[k]), 3 * int(off[k + 1]))
        ref = torch.empty_like(m[s])
        spx.DemagFieldLindholmGPU(Xs, Ts, 8e5, boundary_backend="dense", **kw).compute_vec(m[s].clone(), ref)
        assert float(torch.linalg.norm(H[s] - ref) / torch.linalg.norm(ref)) < tol, BOXES[k]
