"""The demag solves over the scale of their right-hand sides.  The field, its transpose and the
reverse step are linear, so an input scaled by a power of two scales the result; cotangents of a
mean over the nodes or of late trajectory steps are many orders below one, and the solves must
not lose them to the range of FP32.  Meshes whose u2 system runs on one CTA, on a cluster and on
the grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# cubes of the box; interior unknowns 512 (16 slices: one CTA), 1,444 (a cluster), 30,752 (the grid)
MESHES = [(9, 9, 9), (20, 20, 5), (33, 32, 32)]


def _mesh(dims):
    import spinfemx_b200 as spx
    X, T = spx.kuhn_box(*dims, 2.0)
    d = np.random.default_rng(5).uniform(-0.2, 0.2, X.shape)
    for c, n in enumerate(dims):
        d[(X[:, c] < 1.0) | (X[:, c] > 2.0 * n - 1.0), c] = 0.0
    return X + d, T


def _unit(N, seed):
    import torch
    m = np.random.default_rng(seed).normal(size=(N, 3)) + np.array([1.0, 0.3, 0.2])
    return torch.as_tensor((m / np.linalg.norm(m, axis=1)[:, None]).ravel(), device="cuda")


def _tol(rtol, precision, dims):
    """Two solves to rtol of their right-hand sides, and with FP32 vectors two roundings of every
    nodal value on each side; the condition number is below (largest dimension)^2."""
    return (2 * rtol + (4 * 2.0 ** -24 if precision == "f32" else 0.0)) * max(dims) ** 2


def _rel(a, b):
    return float((a - b).norm() / b.norm())


def _field(X, T, precision, warm, rtol=1e-10):
    import spinfemx_b200 as spx
    return spx.EffectiveField(X, T, 8e5, Aex=1.3e-11, alpha=0.1, use_demag=True, precision=precision, demag_kwargs=dict(
        boundary_backend="dense", precision=precision, ksp_rtol_u1=rtol, ksp_rtol_u2=rtol, ksp_atol=0.0,
        ksp_maxit_u1=100000, ksp_maxit_u2=100000, warm_start=warm))


def _step_vjp(hef, m, w):
    import torch
    out = torch.empty_like(m)
    return hef.step_vjp(m, 2.5e-14, w, out, torch.zeros(hef.N, dtype=torch.float64, device="cuda"),
                        torch.zeros(3, dtype=torch.float64, device="cuda"))


@pytest.mark.parametrize("dims", MESHES)
@pytest.mark.parametrize("precision", ["mixed", "f32"])
def test_reverse_products_are_linear_in_the_cotangent(dims, precision):
    import torch
    X, T = _mesh(dims)
    hef = _field(X, T, precision, False)
    m = _unit(hef.N, 1)
    lam = torch.as_tensor(np.random.default_rng(2).normal(size=3 * hef.N), device="cuda")

    def step(w):
        return _step_vjp(hef, m, w)

    def rhs(w):
        return hef.rhs_vjp(m, w, torch.empty_like(m))

    def field(w):
        return hef.demag_field.compute_vec_transpose(w, torch.empty_like(m))

    for rtol in (1e-8, 1e-10, 1e-12):
        hef.demag_field.set_tolerances(ksp_rtol_u1=rtol, ksp_rtol_u2=rtol)
        tol = _tol(rtol, precision, dims)
        for f in (step, rhs, field):
            ref = f(lam)
            assert torch.isfinite(ref).all()
            for e in (10, 20, 30, 40, 50, 60):
                got = f(lam * 2.0 ** -e) * 2.0 ** e
                assert _rel(got, ref) < tol, (rtol, f.__name__, e)
            assert _rel(f(lam), ref) < tol, (rtol, f.__name__, "after the small ones")


# starts extrapolated from the solutions of much smaller right-hand sides
@pytest.mark.parametrize("dims", MESHES)
def test_extrapolated_starts_after_small_cotangents(dims):
    import torch
    X, T = _mesh(dims)
    m = _unit(X.shape[0], 1)
    lam = torch.as_tensor(np.random.default_rng(2).normal(size=m.numel()), device="cuda")
    ref = _step_vjp(_field(X, T, "mixed", False), m, lam)
    hef = _field(X, T, "mixed", "extrapolate_corrected")
    for e in (60, 60, 40, 20, 0, 0, 0):
        assert _rel(_step_vjp(hef, m, lam * 2.0 ** -e) * 2.0 ** e, ref) < _tol(1e-10, "mixed", dims), e


# 2^-66 and 2^40 are about 1e-20 and 1e12
@pytest.mark.parametrize("dims", MESHES)
@pytest.mark.parametrize("precision,pc", [("mixed", "amg"), ("mixed", "jacobi"), ("f64", "jacobi")])
def test_field_is_linear_in_the_magnetisation(dims, precision, pc):
    import torch
    import spinfemx_b200 as spx
    X, T = _mesh(dims)
    rtol = 1e-10
    tol = _tol(rtol, precision, dims)
    m = _unit(X.shape[0], 3)

    def demag(warm):
        return spx.DemagFieldLindholmGPU(X, T, 8e5, boundary_backend="dense", precision=precision, ksp_rtol_u1=rtol,
                                         ksp_rtol_u2=rtol, ksp_atol=0.0, ksp_maxit_u1=20000, ksp_maxit_u2=20000,
                                         u1_preconditioner=pc, warm_start=warm)

    def field(d, v):
        out = torch.empty_like(v)
        d.compute_vec(v, out)
        assert d.last_res_u1 <= rtol and d.last_res_u2 <= rtol
        return out

    d = demag(False)
    ref = field(d, m)
    for e in (-66, -40, 40):
        assert _rel(field(d, m * 2.0 ** e) * 2.0 ** -e, ref) < tol, e
    d = demag(True)  # each solve starts from the one before: small ones first, a zero one in between
    for e in (-66, -40, 0, None, 0, 0):
        if e is None:
            assert float(field(d, torch.zeros_like(m)).abs().max()) == 0.0
        else:
            assert _rel(field(d, m * 2.0 ** e) * 2.0 ** -e, ref) < tol, e


# The u2 solve of the last stage (the first in reverse) starts 3e62 times too large, and a refinement
# gains 7 digits in FP64: the last of the ten refinements reaches the tolerance (3e62 1e-70 = 3e-8), the
# ninth does not (3e62 1e-63 = 0.3, less at most CG's last step per refinement).  The residual that is
# reported has to be that of the solution that is returned.
@pytest.mark.parametrize("dims", MESHES)
def test_reported_residual_is_that_of_the_solution(dims):
    import torch
    X, T = _mesh(dims)
    rtol = 1e-6
    hef = _field(X, T, "f64", "extrapolate", rtol)
    m = _unit(X.shape[0], 4)
    lam = torch.as_tensor(np.random.default_rng(2).normal(size=m.numel()), device="cuda")

    def reported():
        return hef.demag_field.solver_counters()["u2"]["final_rel_residual_sum"]

    _step_vjp(hef, m, lam * 3e62)
    before = reported()
    _step_vjp(hef, m, lam)
    assert reported() - before <= 4 * rtol  # four stages
