"""The persistent Krylov kernels with their matrices in shared memory, against each other: the
AMG-PCG and the Jacobi CG (other arithmetic, the same FP64 residual rule) on meshes where a CTA's
block of slices is empty, partial, wholly resident, or larger than its shared memory, and where
the Jacobi CG runs on one CTA, on a cluster or on the grid; with the stiffness matrix's exact
zeros (lattice meshes, dropped) and without (moved vertices)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(nx, ny, nz, jitter):
    import spinfemx_b200 as spx
    X, T = spx.kuhn_box(nx, ny, nz, 2.0)
    if jitter:
        d = np.random.default_rng(5).uniform(-0.2, 0.2, X.shape)
        for c, n in enumerate((nx, ny, nz)):
            d[(X[:, c] < 1.0) | (X[:, c] > 2.0 * n - 1.0), c] = 0.0
        X = X + d
    return X, T


# nodes: 80 (3 slices: one CTA; most CTAs of the PCG without rows), 1,008 (32 slices: two CTAs),
# 4,736 (148 slices: one a CTA of the PCG, a cluster of eight), 4,800 (two more slices), 29,791
# (grid), and 638,976 off the lattice, more matrix than the CTAs' shared memory
@pytest.mark.parametrize("dims,jitter,precision", [
    ((4, 3, 3), False, "mixed"), ((4, 3, 3), True, "f64"), ((20, 11, 3), True, "f64"), ((36, 15, 7), False, "mixed"),
    ((39, 11, 9), True, "f64"), ((30, 30, 30), True, "mixed"), ((30, 30, 30), False, "f64"),
    ((95, 103, 63), True, "mixed")])
def test_amg_pcg_matches_jacobi(dims, jitter, precision):
    import torch
    import spinfemx_b200 as spx
    X, T = _mesh(*dims, jitter)
    N = X.shape[0]
    rng = np.random.default_rng(N)
    m = rng.normal(size=(N, 3))
    m = torch.as_tensor((m / np.linalg.norm(m, axis=1)[:, None]).ravel(), device="cuda")
    rtol, u = 1e-10, []
    for pc in ("amg", "jacobi"):
        d = spx.DemagFieldLindholmGPU(X, T, 8e5, boundary_backend="auto", dense_gpu_max_bytes=64 << 20,
                                      precision=precision, ksp_rtol_u1=rtol, ksp_rtol_u2=rtol, ksp_atol=0.0,
                                      ksp_maxit_u1=20000, ksp_maxit_u2=20000, u1_preconditioner=pc)
        d.compute_vec(m, torch.empty_like(m))
        assert d.last_res_u1 <= rtol and d.last_res_u2 <= rtol
        u.append(d.potentials()[0])
        del d
    # each solution is off by at most cond(A) rtol, cond(A) below (largest dimension)^2 for the
    # Neumann problem's nonzero modes
    tol = 2 * rtol * max(dims) ** 2
    assert float(torch.linalg.norm(u[0] - u[1]) / torch.linalg.norm(u[1])) < tol
