"""A call whose device allocation fails raises MemoryError and leaves the object usable: the next call
allocates again (a buffer that kept its size without its memory would be handed to the kernels).
The failure is injected on the host, before any allocation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _twice(call, *args):
    """call() with its first allocation failing, then again"""
    from spinfemx_b200 import _lib
    try:
        _lib.call("spx_debug_fail_alloc", 1, 1)
        with pytest.raises(MemoryError):
            call(*args)
    finally:
        _lib.call("spx_debug_fail_alloc", 0, 0)
    return call(*args)


def test_products_after_a_failed_allocation():
    import torch
    import spinfemx_b200 as spx
    g = spx.BoundaryGeometry(*spx.kuhn_box(20, 14, 3, 2.0))
    cfg = spx.HMatrixBuildConfig(epsilon=1e-5, leaf_size=16)
    a, b = (spx.HMatrixGPUPackedFused(g, cfg, precision="f64") for _ in range(2))
    X = torch.as_tensor(np.random.default_rng(1).standard_normal((8, g.Nb)), device="cuda")
    assert torch.equal(_twice(b.matvec, X[0]), a.matvec(X[0]))
    assert torch.equal(_twice(b.matmat, X), a.matmat(X))


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_field_after_a_failed_allocation(precision):
    import torch
    import spinfemx_b200 as spx
    X, T = spx.kuhn_box(9, 8, 4, 2.0)
    m = np.random.default_rng(2).normal(size=(X.shape[0], 3))
    m = torch.as_tensor((m / np.linalg.norm(m, axis=1)[:, None]).ravel(), device="cuda")
    kw = dict(boundary_backend="hmatrix", precision=precision, hmatrix_leaf_size=16)
    a, b = (spx.DemagFieldLindholmGPU(X, T, 8e5, **kw) for _ in range(2))

    def run(d):
        return d.compute_vec(m, torch.empty_like(m))

    def back(d):
        return d.compute_vec_transpose(m, torch.empty_like(m))

    assert torch.equal(_twice(run, b), run(a))
    assert torch.equal(_twice(back, b), back(a))
