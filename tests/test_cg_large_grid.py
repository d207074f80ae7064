"""The Jacobi CG on systems past one cluster, in its two forms on the grid: matrix and records in
shared memory (up to 27,000 entries and 80 slices a CTA in FP32, 8,000 entries in FP64) and plain vectors
in global memory.
The residuals of the returned potentials, from the host's matrices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(dims, jitter):
    import spinfemx_b200 as spx
    X, T = spx.kuhn_box(*dims, 2.0)
    if jitter:
        d = np.random.default_rng(5).uniform(-0.2, 0.2, X.shape)
        for c, n in enumerate(dims):
            d[(X[:, c] < 1.0) | (X[:, c] > 2.0 * n - 1.0), c] = 0.0
        X = X + d
    return X, T


# entries a CTA of the u1 / u2 systems: 7,680 / 7,680 (below both lines), 9,600 / 8,160 (past the line of
# FP64), 29,280 / 26,880 (u1 past that of FP32 too, u2 just below it), 54,240 / 49,920 (several rounds of the
# warps); on the lattice (7 entries a row) 25,312 / 23,520
@pytest.mark.parametrize("dims,jitter", [((40, 41, 39), True), ((44, 43, 45), True), ((65, 64, 66), True),
                                         ((81, 80, 79), True), ((80, 79, 81), False)])
@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_residuals_of_the_potentials(dims, jitter, precision):
    import scipy.sparse as sp
    import torch
    import spinfemx_b200 as spx
    X, T = _mesh(dims, jitter)
    N, Ms, rtol = X.shape[0], 8e5, 1e-9
    f = spx.geometry.fem_assemble(X, T)
    m = np.random.default_rng(1).normal(size=(N, 3)) + np.array([1.0, 0.3, 0.2])
    m /= np.linalg.norm(m, axis=1)[:, None]
    A = sp.csr_matrix((f["A"], f["col"], f["rowptr"]), shape=(N, N))
    b = Ms * sum(sp.csr_matrix((f["Div"][:, c], f["col"], f["rowptr"]), shape=(N, N)) @ m[:, c] for c in range(3))
    inner = np.setdiff1d(np.arange(N), spx.geometry.boundary_data(X, T)["bverts"])
    d = spx.DemagFieldLindholmGPU(X, T, Ms, boundary_backend="hmatrix", precision=precision, ksp_rtol_u1=rtol,
                                  ksp_rtol_u2=rtol, ksp_atol=0.0, ksp_maxit_u1=20000, ksp_maxit_u2=20000,
                                  u1_preconditioner="jacobi")
    mt = torch.as_tensor(m.ravel(), device="cuda")
    d.compute_vec(mt, torch.empty_like(mt))
    u1, u2 = (u.cpu().numpy() for u in d.potentials())
    r1 = b - b.mean() - A @ u1
    # the right-hand side's FP32 operator ("mixed"): unit roundoff of each term, a few of them alike
    assert np.linalg.norm(r1) <= (1.01 * rtol + (1e-6 if precision == "mixed" else 0.0)) * np.linalg.norm(b)
    g = np.zeros(N)
    outer = np.setdiff1d(np.arange(N), inner)
    g[outer] = u2[outer]
    # u2 is a difference of potentials: their rounding times the rows' sums, far below rtol
    assert np.linalg.norm((A @ u2)[inner]) <= 1.1 * rtol * np.linalg.norm((A @ g)[inner])
