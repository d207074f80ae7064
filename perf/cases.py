"""The work that a program using this library has it do, as cases that can be timed.

Every case runs one public call (or the few calls of one Newton step, one field evaluation, one
short run of time steps) on a box mesh.  The sizes are those of the repository's own workloads:
the 20x20x5 box (dense boundary operator, FP64), the 400x400x2 film of the headline benchmark
(H-matrix, mixed precision), the ensemble of 64 uneven boxes, the 100x100x2 film of the gradient
workload, and the films of the tests in between; one mesh has its vertices moved off the lattice,
as a mesh generator's would be, and odd numbers of cubes.

What a program sets up once per mesh (geometry, H-matrix, solver hierarchy, field object) is
built once per process and shared by the states of a case (`_plan`); `prepare` makes the
vectors.  Krylov tolerances are 1e-10 and tighter, as in the gradient workload and the tests,
so that the results are those of the operators and not of the solver's path.
"""
import itertools
import json
import math
import os
import sys
from collections import OrderedDict

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "fenicsx-micromagnetics_b200"))
import spinfemx_b200 as spx  # noqa: E402
from spinfemx_b200.ensemble import LLGEnsemble  # noqa: E402

MU0 = 4.0e-7 * math.pi
MS, AEX = 8.0e5, 1.3e-11
GAMMA = 2.211e5
NORMAL = (0.0, 0.0, 1.0)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one right-hand side of a small element without demag (exchange, anisotropy, DMI,
        # applied field): the smallest call, launch latency
        dict(name="rhs_local_8x8x3", kind="rhs", nx=8, ny=8, nz=3, h=2.0, jitter=0.0, precision="f64"),
        # one Newton / GMRES iteration of the implicit driver: linearise, build the block
        # preconditioner, one Jacobian product, one preconditioner application
        dict(name="newton_200x200x2", kind="newton", nx=200, ny=200, nz=2, h=2.0, jitter=0.0, precision="f64"),
        # one demag field of the 20x20x5 box with the dense operator in FP64, zero start (the
        # drop-in call at its defaults but for the tolerance)
        dict(name="field_dense_20x20x5", kind="field", nx=20, ny=20, nz=5, h=2.0, jitter=0.0, precision="f64"),
        # ten RK4 steps of the same box (10 fs), extrapolated Krylov starts
        dict(name="steps_dense_20x20x5", kind="steps", nx=20, ny=20, nz=5, h=2.0, jitter=0.0, precision="f64",
             dt=1e-14, nsteps=10, alpha=0.5),
        # boundary operator applied to one vector: the film of the gradient workload (FP32
        # factors), a mesh off the lattice with odd sizes (FP64 factors), the headline film
        dict(name="matvec_100x100x2_f32", kind="matvec", nx=100, ny=100, nz=2, h=2.0, jitter=0.0, precision="mixed"),
        dict(name="matvec_97x61x3_f64", kind="matvec", nx=97, ny=61, nz=3, h=2.5, jitter=0.12, precision="f64"),
        dict(name="matvec_400x400x2_f32", kind="matvec", nx=400, ny=400, nz=2, h=2.5, jitter=0.0, precision="mixed"),
        # eight states of one film at once, far field on the tensor cores (batched films)
        dict(name="matmat8_150x150x2", kind="matmat", nx=150, ny=150, nz=2, h=2.5, jitter=0.0, precision="f32"),
        # ten RK4 steps (50 fs) of the headline film: demag, exchange and applied field
        dict(name="steps_400x400x2", kind="steps", nx=400, ny=400, nz=2, h=2.5, jitter=0.0, precision="mixed",
             dt=5e-14, nsteps=10, alpha=0.02),
        # ten RK4 steps (20 fs) of 64 boxes of uneven size integrated together
        dict(name="ensemble_64_boxes", kind="ensemble", samples=64, draw=7000, dt=2e-14, nsteps=10),
        # backward pass of one RK4 step of the gradient workload's film
        dict(name="step_vjp_100x100x2", kind="vjp", nx=100, ny=100, nz=2, h=2.0, jitter=0.0, precision="mixed",
             dt=2.5e-14),
        # a new mesh: H-matrix construction (fill, ACA, packing) and its first product
        dict(name="build_48x48x2", kind="build", nx=48, ny=48, nz=2, h=2.5, jitter=0.0, precision="f32"),
    ]


def draw(rng):
    """One more case of the same kinds: sizes log-uniform between a few cubes and the largest
    mesh whose operators a process sets up within seconds."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["rhs", "newton", "field", "steps", "steps_film", "matvec", "matvec", "matmat", "ensemble", "vjp",
                       "build"])
    jitter = rng.choice([0.0, round(rng.uniform(0.05, 0.15), 3)])
    h = rng.choice([2.0, 2.5])
    if kind in ("rhs", "newton"):
        return dict(kind=kind, nx=size(5, 200), ny=size(5, 200), nz=rng.randint(1, 5), h=h, jitter=jitter,
                    precision=rng.choice(["f64", "mixed"]))
    if kind == "field":
        return dict(kind=kind, nx=size(6, 30), ny=size(6, 30), nz=rng.randint(2, 6), h=h, jitter=jitter, precision="f64")
    if kind == "steps":
        return dict(kind=kind, nx=size(6, 30), ny=size(6, 30), nz=rng.randint(2, 6), h=h, jitter=jitter,
                    precision="f64", dt=1e-14, nsteps=rng.randint(6, 12), alpha=0.5)
    if kind == "steps_film":
        return dict(kind="steps", nx=size(30, 180), ny=size(30, 180), nz=rng.randint(1, 3), h=h, jitter=jitter,
                    precision="mixed", dt=5e-14, nsteps=rng.randint(6, 12), alpha=0.02)
    if kind == "matvec":
        return dict(kind=kind, nx=size(24, 200), ny=size(24, 200), nz=rng.randint(1, 4), h=h, jitter=jitter,
                    precision=rng.choice(["mixed", "mixed", "f64"]))
    if kind == "matmat":
        return dict(kind=kind, nx=size(30, 180), ny=size(30, 180), nz=rng.randint(1, 3), h=h, jitter=jitter,
                    precision="f32")
    if kind == "ensemble":
        return dict(kind=kind, samples=size(4, 64), draw=rng.randint(1, 1 << 30), dt=2e-14, nsteps=rng.randint(6, 12))
    if kind == "vjp":
        return dict(kind=kind, nx=size(24, 120), ny=size(24, 120), nz=rng.randint(1, 3), h=h, jitter=jitter,
                    precision="mixed", dt=2.5e-14)
    return dict(kind="build", nx=size(20, 80), ny=size(20, 80), nz=rng.randint(1, 3), h=h, jitter=jitter,
                precision=rng.choice(["f32", "f64"]))


# ------------------------------------------------------------------ meshes and plans
def _mesh(nx, ny, nz, h, jitter):
    """Box of nx x ny x nz cubes (six tets each); `jitter` moves every vertex by up to that
    fraction of h along the axes on whose faces it does not lie."""
    X, T = spx.kuhn_box(nx, ny, nz, h)
    if jitter:
        rng = np.random.default_rng(nx * 1000003 + ny * 1009 + nz)
        d = rng.uniform(-jitter * h, jitter * h, X.shape)
        for c, n in enumerate((nx, ny, nz)):
            d[(X[:, c] < 0.5 * h) | (X[:, c] > (n - 0.5) * h), c] = 0.0
        X = X + d
    return X, T


def _boxes(samples, draw):
    """Sides U[20, 120] nm, thickness 4, 6, 8 or 10 nm, in 2 nm cubes (the ensemble workload)."""
    rng = np.random.default_rng(draw)
    return [(int(round(rng.uniform(20, 120) / 2)), int(round(rng.uniform(20, 120) / 2)),
             int(rng.choice([4, 6, 8, 10])) // 2) for _ in range(samples)]


_PLANS = OrderedDict()


def _plan(make, *key):
    """What a program keeps per mesh, built once per process (the last 24 kept)."""
    k = json.dumps([make.__name__, *key])
    if k not in _PLANS:
        _PLANS[k] = make(*key)
        while len(_PLANS) > 24:
            _PLANS.popitem(last=False)
    _PLANS.move_to_end(k)
    return _PLANS[k]


def _local_field(nx, ny, nz, h, jitter, precision):
    X, T = _mesh(nx, ny, nz, h, jitter)
    return spx.EffectiveField(X, T, MS, Aex=AEX, Ku=5e5, n_ani_vec=NORMAL, D_int=3e-3, n0_int_vec=NORMAL, alpha=0.3,
                              H0_static=[0.0, 2e4, 5e4], precision=precision)


def _dense_field(nx, ny, nz, h, jitter, precision):
    X, T = _mesh(nx, ny, nz, h, jitter)
    return spx.DemagFieldLindholmGPU(X, T, MS, boundary_backend="dense", precision=precision, ksp_rtol_u1=1e-12,
                                     ksp_rtol_u2=1e-12, ksp_atol=0.0, ksp_maxit_u1=20000, ksp_maxit_u2=20000)


def _film_field(nx, ny, nz, h, jitter, precision, backend, alpha, ku):
    """LLG field object with demag: the headline film's options, or the gradient workload's with
    a nodal anisotropy map (`ku`)."""
    X, T = _mesh(nx, ny, nz, h, jitter)
    kw = dict(H0_static=[-0.025 / MU0 * math.cos(math.radians(10.0)), 0.025 / MU0 * math.sin(math.radians(10.0)), 0.0])
    if ku:
        s = X / X.max(axis=0)
        kw = dict(Ku_nodes=2e5 + 5e4 * np.cos(2 * math.pi * s[:, 0]) * np.sin(4 * math.pi * s[:, 1]),
                  n_ani_vec=NORMAL, H0_static=[0.0, 0.05 / MU0, 0.0])
    dk = dict(boundary_backend=backend, precision=precision, ksp_rtol_u1=1e-10, ksp_rtol_u2=1e-10, ksp_atol=0.0,
              ksp_maxit_u1=20000, ksp_maxit_u2=20000, warm_start="extrapolate_corrected")
    if backend == "hmatrix":
        dk.update(hmatrix_epsilon=1e-5, hmatrix_eta=2.0, hmatrix_leaf_size=64, hmatrix_recompress=True)
    return spx.EffectiveField(X, T, MS, Aex=AEX, alpha=alpha, use_demag=True, precision=precision, demag_kwargs=dk,
                              **kw)


def _hmatrix(nx, ny, nz, h, jitter, precision):
    X, T = _mesh(nx, ny, nz, h, jitter)
    H = spx.HMatrixGPUPackedFused(spx.BoundaryGeometry(X, T), _hconfig(), precision=precision)
    H.enable_tensor_cores(True)
    return H


def _geometry(nx, ny, nz, h, jitter):
    return spx.BoundaryGeometry(*_mesh(nx, ny, nz, h, jitter))


def _hconfig():
    return spx.HMatrixBuildConfig(epsilon=1e-5, eta=2.0, leaf_size=64)


def _ensemble(samples, draw):
    boxes = _boxes(samples, draw)
    Bz = np.random.default_rng(draw + 100).uniform(-0.5, 0.5, size=samples)
    return LLGEnsemble([spx.kuhn_box(*b, 2.0) for b in boxes], 1.1e6, Aex=1.6e-11, Ku=8e5, D_int=3e-3, alpha=0.3,
                       H0=[[0.0, 0.0, b / MU0] for b in Bz], dense_max_nb=4096, precision="mixed", graph=True,
                       demag_kwargs=dict(hmatrix_epsilon=1e-5, hmatrix_eta=2.0, hmatrix_leaf_size=64, ksp_rtol_u1=1e-10,
                                         ksp_rtol_u2=1e-10, ksp_atol=0.0, warm_start="extrapolate_corrected"))


def _dims(c):
    return c["nx"], c["ny"], c["nz"], c["h"], c["jitter"]


def _film_key(c):
    return (*_dims(c), c["precision"], "dense" if c["precision"] == "f64" and c["kind"] == "steps" else "hmatrix",
            c.get("alpha", 0.02), False)


# ------------------------------------------------------------------ states
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _unit(n, g, direction=None, sigma=1.0):
    """n unit vectors: `direction` plus Gaussian noise, or random directions."""
    m = sigma * torch.randn(n, 3, dtype=torch.float64, device="cuda", generator=g)
    if direction is not None:
        m += torch.tensor(direction, dtype=torch.float64, device="cuda")
    return torch.nn.functional.normalize(m, dim=1).reshape(-1).contiguous()


def _start(c, n, g):
    """Initial magnetisation: (1, 1, 1) with 10 % noise (box), x with 5 % noise (films)."""
    return _unit(n, g, (1.0, 1.0, 1.0), 0.1) if c["precision"] == "f64" else _unit(n, g, (1.0, 0.0, 0.0), 0.05)


def prepare(case, seed):
    c, g, kind = case, _gen(seed), case["kind"]
    if kind == "rhs":
        hef = _plan(_local_field, *_dims(c), c["precision"])
        m = _unit(hef.N, g)
        return dict(kind=kind, hef=hef, m=m, out=torch.empty_like(m))
    if kind == "newton":
        hef = _plan(_local_field, *_dims(c), c["precision"])
        m, v = _unit(hef.N, g), _unit(hef.N, g)
        return dict(kind=kind, hef=hef, jc=spx.JvContext(hef), m=m, v=v, y=torch.empty_like(m), z=torch.empty_like(m))
    if kind == "field":
        d = _plan(_dense_field, *_dims(c), c["precision"])
        m = _start(c, d.N, g)
        return dict(kind=kind, demag=d, m=m, out=torch.empty_like(m))
    if kind == "steps":
        hef = _plan(_film_field, *_film_key(c))
        m = _start(c, hef.N, g)
        return dict(kind=kind, hef=hef, m=m, out=torch.empty_like(m), dt=c["dt"], nsteps=c["nsteps"])
    if kind == "matvec":
        H = _plan(_film_field, *_film_key(c)).demag_field.B_hmatrix_gpu
        x = torch.randn(H.size, dtype=torch.float64, device="cuda", generator=g)
        return dict(kind=kind, H=H, x=x, out=torch.empty_like(x))
    if kind == "matmat":
        H = _plan(_hmatrix, *_dims(c), c["precision"])
        x = torch.randn(8, H.size, dtype=torch.float64, device="cuda", generator=g)
        return dict(kind=kind, H=H, x=x, out=torch.empty_like(x))
    if kind == "ensemble":
        e = _plan(_ensemble, c["samples"], c["draw"])
        return dict(kind=kind, ens=e, m=_unit(e.N, g), dt=c["dt"], nsteps=c["nsteps"])
    if kind == "vjp":
        hef = _plan(_film_field, *_dims(c), c["precision"], "hmatrix", 0.1, True)
        m = _start(c, hef.N, g)
        lam = 1e-2 * torch.randn(3 * hef.N, dtype=torch.float64, device="cuda", generator=g)
        return dict(kind=kind, hef=hef, m=m, lam=lam, out=torch.empty_like(m), dt=c["dt"],
                    gKu=torch.empty(hef.N, dtype=torch.float64, device="cuda"),
                    gH0=torch.empty(3, dtype=torch.float64, device="cuda"))
    geom = _plan(_geometry, *_dims(c))
    x = torch.randn(geom.Nb, dtype=torch.float64, device="cuda", generator=g)
    return dict(kind="build", geom=geom, x=x, precision=c["precision"])


SHIFT = 1.5e13  # 3 / (2 dt) of a BDF2 step of 0.1 ps


def run(s):
    kind = s["kind"]
    if kind == "rhs":
        s["hef"].llg_rhs_vec(s["m"], s["out"])
        return s["out"]
    if kind == "newton":
        s["hef"].update_jac_state(s["m"])
        s["jc"].update_pc_full_fast_gpu(SHIFT)
        s["jc"].mult(None, s["v"], s["y"])
        s["jc"].apply(None, s["y"], s["z"])
        return s["y"], s["z"]
    if kind == "field":
        return s["demag"].compute_vec(s["m"], s["out"])
    if kind == "steps":
        s["hef"].set_state(s["m"])
        s["hef"].step(s["dt"], s["nsteps"])
        return s["hef"].get_state(s["out"])
    if kind == "matvec":
        return s["H"].matvec(s["x"], out=s["out"])
    if kind == "matmat":
        return s["H"].matmat(s["x"], out=s["out"])
    if kind == "ensemble":
        s["ens"].set_state(s["m"])
        s["ens"].step(s["dt"], s["nsteps"])
        return s["ens"].get_state()
    if kind == "vjp":
        s["gKu"].zero_()
        s["gH0"].zero_()
        s["hef"].step_vjp(s["m"], s["dt"], s["lam"], s["out"], s["gKu"], s["gH0"])
        return s["out"], s["gKu"], s["gH0"]
    return spx.HMatrixGPUPackedFused(s["geom"], _hconfig(), precision=s["precision"]).matvec(s["x"])


# ------------------------------------------------------------------ what the work cannot do without
def _counts(nx, ny, nz):
    """(nodes, entries of the node-node pattern, boundary nodes) of the box."""
    n = (nx + 1) * (ny + 1) * (nz + 1)
    edges = (nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz + nx * ny * (nz + 1)
             + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz)
    return n, n + 2 * edges, n - (nx - 1) * (ny - 1) * max(nz - 1, 0)


def _h_entries(nb):
    """Stored entries of the H-matrix (1e-5, leaf 64) of a box with nb boundary nodes: about 930
    per row at 1,346 rows and 560 more for each doubling (films of 24 to 400 cubes a side)."""
    return nb * min(float(nb), max(64.0, 930.0 + 560.0 * (math.log2(nb) - 10.4)))


def _llg_eval(nx, ny, nz, operator_bytes, val):
    """One field and right-hand side with demag: divergence, gradient and exchange operators
    (7 values and one column per pattern entry), the stiffness once for each Poisson solve, the
    boundary operator, the state in and the rate out."""
    n, nnz, nb = _counts(nx, ny, nz)
    return 7 * val * nnz + 4 * nnz + 2 * (val + 4) * nnz + operator_bytes + 12 * 8 * n, 18.0 * nnz + 80.0 * n


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        b = f = 0.0
        for box in _boxes(case["samples"], case["draw"]):
            nb = _counts(*box)[2]
            e = float(nb) * nb if nb <= 4096 else _h_entries(nb)
            db, df = _llg_eval(*box, 4 * e, 4)
            b, f = b + db + 9 * 4 * _counts(*box)[1], f + df + 2 * e
        return {"bytes": 4 * case["nsteps"] * b, "flops": 4 * case["nsteps"] * f}
    d = (case["nx"], case["ny"], case["nz"])
    n, nnz, nb = _counts(*d)
    val = 8 if case["precision"] == "f64" else 4
    e = _h_entries(nb)
    if kind == "rhs":  # exchange and DMI blocks (10 values an entry), state, axis, field, rate
        return {"bytes": (10 * val + 4) * nnz + 4 * 24 * n, "flops": 24.0 * nnz + 60.0 * n}
    if kind == "newton":  # the operators twice (state and direction), 3x3 blocks written and read
        return {"bytes": 2 * (10 * val + 4) * nnz + 2 * 72 * n + 8 * 24 * n, "flops": 48.0 * nnz + 300.0 * n}
    if kind == "field":
        b, f = _llg_eval(*d, 8.0 * nb * nb, 8)
        return {"bytes": b, "flops": f + 2.0 * nb * nb}
    if kind == "steps":
        e = float(nb) * nb if case["precision"] == "f64" else e
        b, f = _llg_eval(*d, val * e, val)
        return {"bytes": 4 * case["nsteps"] * b, "flops": 4 * case["nsteps"] * (f + 2 * e)}
    if kind == "matvec":
        return {"bytes": val * e + 16 * nb, "flops": 2 * e}
    if kind == "matmat":
        return {"bytes": 4 * e + 8 * 16 * nb, "flops": 16 * e}
    if kind == "vjp":  # four stages forward and four transposed
        b, f = _llg_eval(*d, 4 * e, 4)
        return {"bytes": 8 * b, "flops": 8 * (f + 2 * e)}
    # construction: every entry of the partition is evaluated (two triangles' weights of about 250
    # operations each) and the kept ones are written and read once
    return {"bytes": 2 * val * e, "flops": 500.0 * nb * nb}


# ------------------------------------------------------------------ 64-bit values
def _solid_angle(a, b, c):
    na, nb, nc = (torch.linalg.norm(v, dim=-1) for v in (a, b, c))
    det = (a * torch.linalg.cross(b, c)).sum(-1)
    den = na * nb * nc + (a * b).sum(-1) * nc + (b * c).sum(-1) * na + (c * a).sum(-1) * nb
    return 2.0 * torch.atan2(det, den)


class _Exact:
    """P1 / BEM operators of one mesh in FP64 torch: matrix-free sums over the tets, dense inverses
    of the two Poisson matrices, and the dense collocated double layer with linear elements
    (Lindholm's closed form)."""

    def __init__(self, X, T, ms, demag=True):
        dev = dict(device="cuda")
        self.T = torch.as_tensor(np.asarray(T, np.int64), **dev)
        self.X = torch.as_tensor(X, dtype=torch.float64, **dev)
        self.ms, self.n = ms, X.shape[0]
        P = self.X[self.T]
        M = P[:, 1:] - P[:, :1]
        self.tv = torch.linalg.det(M).abs() / 6.0
        g = torch.linalg.inv(M).transpose(1, 2)
        self.g = torch.cat([-g.sum(1, keepdim=True), g], 1)
        self.vol = torch.zeros(self.n, dtype=torch.float64, **dev).index_add(
            0, self.T.reshape(-1), (self.tv / 4.0).repeat_interleave(4))
        self._facets()
        if demag:
            self._boundary()
            self._inverses()

    def _facets(self):
        F = torch.cat([self.T[:, list(k)] for k in itertools.combinations(range(4), 3)])
        opp = torch.cat([self.T[:, 6 - sum(k)] for k in itertools.combinations(range(4), 3)])
        key = torch.sort(F, 1)[0]
        key = (key[:, 0] * self.n + key[:, 1]) * self.n + key[:, 2]
        _, inv, cnt = torch.unique(key, return_inverse=True, return_counts=True)
        keep = cnt[inv] == 1
        F, opp = F[keep], opp[keep]
        p = self.X[F]
        nrm = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
        inward = ((self.X[opp] - p[:, 0]) * nrm).sum(1) > 0
        F = torch.where(inward[:, None], F[:, [0, 2, 1]], F)
        nrm = torch.where(inward[:, None], -nrm, nrm)
        self.area = torch.linalg.norm(nrm, dim=1) / 2.0
        self.F, self.nu = F, nrm / (2.0 * self.area)[:, None]

    def _boundary(self):
        bv = torch.unique(self.F)
        lid = torch.full((self.n,), -1, dtype=torch.int64, device="cuda")
        lid[bv] = torch.arange(bv.numel(), device="cuda")
        self.bv, nb = bv, bv.numel()
        ib = torch.ones(self.n, dtype=torch.bool, device="cuda")
        ib[bv] = False
        self.iv = torch.nonzero(ib).reshape(-1)
        fl, p = lid[self.F], self.X[self.F]
        e = torch.stack([p[:, 1] - p[:, 0], p[:, 2] - p[:, 1], p[:, 0] - p[:, 2]], 1)
        s = torch.linalg.norm(e, dim=2)
        xi = e / s[:, :, None]
        eta = torch.linalg.cross(self.nu[:, None].expand(-1, 3, -1), xi)
        gam = torch.stack([(xi.roll(-1 - i, 1)[:, :1] * xi).sum(2) for i in range(3)], 1)
        B = torch.zeros(nb, nb, dtype=torch.float64, device="cuda")
        per = max(1, 4_000_000 // fl.shape[0])
        for r0 in range(0, nb, per):
            rows = torch.arange(r0, min(nb, r0 + per), device="cuda")
            x = self.X[bv[rows]]
            rho = [p[None, :, k] - x[:, None] for k in range(3)]
            skip = (fl[None] == rows[:, None, None]).any(2)
            r = [torch.linalg.norm(v, dim=-1) for v in rho]
            om = _solid_angle(*rho)
            hh = (rho[0] * self.nu).sum(-1)
            Pl = [torch.log1p(2.0 * s[:, k] / (r[k] + r[(k + 1) % 3] - s[:, k])) for k in range(3)]
            for k in range(3):
                q = (k + 1) % 3
                gp = sum(gam[:, k, j] * Pl[j] for j in range(3))
                w = s[:, q] / (8.0 * math.pi * self.area) * ((eta[:, q] * rho[q]).sum(-1) * om - hh * gp)
                B[r0:r0 + rows.numel()].index_add_(1, fl[:, k], torch.where(skip, torch.zeros_like(w), w))
        ang = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        P = self.X[self.T]
        for j in range(4):
            o = [P[:, (j + q) % 4] - P[:, j] for q in (1, 2, 3)]
            ang = ang.index_add(0, self.T[:, j], _solid_angle(*o).abs())
        B.diagonal().add_(ang[bv] / (4.0 * math.pi) - 1.0)
        self.B = B

    def _inverses(self):
        K = torch.zeros(self.n * self.n, dtype=torch.float64, device="cuda")
        Ke = self.tv[:, None, None] * (self.g @ self.g.transpose(1, 2))
        K.index_add_(0, (self.T[:, :, None] * self.n + self.T[:, None, :]).reshape(-1), Ke.reshape(-1))
        K = K.view(self.n, self.n)
        self.inv2 = torch.cholesky_inverse(torch.linalg.cholesky(K[self.iv][:, self.iv])) if self.iv.numel() else None
        K += K.diagonal().mean() / self.n
        self.inv1 = torch.cholesky_inverse(torch.linalg.cholesky(K))

    def nodal(self, v):  # [E, 4, ...] summed to the nodes
        return torch.zeros((self.n, *v.shape[2:]), dtype=torch.float64, device="cuda").index_add(
            0, self.T.reshape(-1), v.reshape(-1, *v.shape[2:]))

    def stiff(self, u):  # A u for u [N] or [N, 3]
        gu = torch.einsum("eac,ea...->ec...", self.g, u[self.T])
        return self.nodal(self.tv.view(-1, *[1] * u.dim()) * torch.einsum("eac,ec...->ea...", self.g, gu))

    def poisson(self, b):
        u = _Solve.apply(b - b.mean(), self, 1)
        return u - u.mean()

    def demag(self, m):
        mb = m[self.T].sum(1)
        b = self.nodal(self.ms * (self.tv / 4.0)[:, None] * torch.einsum("eac,ec->ea", self.g, mb))
        u1 = self.poisson(b)
        gB = self.B @ u1[self.bv]
        u2 = torch.zeros_like(u1).index_add(0, self.bv, gB)
        if self.iv.numel():
            u2 = u2.index_add(0, self.iv, _Solve.apply(-self.stiff(u2)[self.iv], self, 2))
        gp = torch.einsum("eac,ea->ec", self.g, (u1 + u2)[self.T])
        H = self.nodal((-(self.tv / 4.0)[:, None] * gp)[:, None].expand(-1, 4, -1))
        return H / self.vol[:, None]

    def exchange(self, m, aex):
        return -2.0 * aex / (MU0 * self.ms) * 1e18 * self.stiff(m) / self.vol[:, None]

    def dmi(self, m, d):  # interfacial, uniform interface normal
        n = torch.tensor(NORMAL, dtype=torch.float64, device="cuda")
        mE = m[self.T]
        div = torch.einsum("eac,eac->e", self.g, mE)
        gn = torch.einsum("eac,ea->ec", self.g, mE @ n)
        h = self.nodal(((self.tv / 4.0)[:, None] * (div[:, None] * n - gn))[:, None].expand(-1, 4, -1))
        mF = m[self.F]
        mF = (mF.sum(1, keepdim=True) + mF) * (self.area / 12.0)[:, None, None]
        nuF = self.nu[:, None]
        f = 0.5 * (nuF * (mF @ n)[..., None] - n * (mF * nuF).sum(-1, keepdim=True))
        h = h.index_add(0, self.F.reshape(-1), f.reshape(-1, 3))
        return -2.0 * d / (MU0 * self.ms) * 1e9 * h / self.vol[:, None]


class _Solve(torch.autograd.Function):
    """Poisson solve with a dense inverse and one refinement (symmetric, so its own adjoint)."""

    @staticmethod
    def forward(ctx, b, ex, which):
        ctx.ex, ctx.which = ex, which

        def mul(u):
            if which == 1:
                return ex.stiff(u)
            full = torch.zeros(ex.n, dtype=torch.float64, device="cuda")
            full[ex.iv] = u
            return ex.stiff(full)[ex.iv]

        inv = ex.inv1 if which == 1 else ex.inv2
        if which == 1:
            b = b - b.mean()
        u = inv @ b
        return u + inv @ (b - mul(u))

    @staticmethod
    def backward(ctx, g):
        return _Solve.apply(g, ctx.ex, ctx.which), None, None


def _rate(m, H, ms, alpha):
    c = torch.linalg.cross(m, H)
    k = GAMMA / (1.0 + alpha * alpha)
    return -k * (c + alpha * torch.linalg.cross(m, c)) + 0.5 * ms * k * (1.0 - (m * m).sum(1, keepdim=True)) * m


def _rk4(f, m, dt):
    k1 = f(m)
    k2 = f(m + 0.5 * dt * k1)
    k3 = f(m + 0.5 * dt * k2)
    return m + dt / 6.0 * (k1 + 2.0 * (k2 + k3) + f(m + dt * k3))


def _vec(v):
    return torch.tensor(v, dtype=torch.float64, device="cuda")


def _uniaxial(m, ku, ms):
    n = _vec(NORMAL)
    return (2.0 * ku / (MU0 * ms)) * (m @ n)[:, None] * n


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "ensemble":
        return _exact_ensemble(c, seed)
    n, _, nb = _counts(c["nx"], c["ny"], c["nz"])
    if kind not in ("rhs", "newton") and (n > 36000 or nb > 26000):
        return None  # dense 64-bit operators would take too long
    X, T = _mesh(*_dims(c))
    ex = _Exact(X, T, MS, demag=kind not in ("rhs", "newton", "matvec", "matmat", "build"))
    g = _gen(seed)
    if kind in ("rhs", "newton"):
        h0 = _vec([0.0, 2e4, 5e4])

        def lin(v):
            return ex.exchange(v, AEX) + ex.dmi(v, 3e-3) + _uniaxial(v, 5e5, MS)

        m = _unit(n, g).view(-1, 3)
        if kind == "rhs":
            return _rate(m, lin(m) + h0, MS, 0.3).reshape(-1)
        v = _unit(n, g).view(-1, 3)
        return _exact_newton(ex, lin, m, v, h0, 0.3)
    if kind in ("matvec", "matmat", "build"):
        ex._boundary()
        shape = (8, nb) if kind == "matmat" else (nb,)
        return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g) @ ex.B.T
    m = _start(c, n, g).view(-1, 3)
    if kind == "field":
        return ex.demag(m).reshape(-1)
    if kind == "steps":
        h0 = _vec([-0.025 / MU0 * math.cos(math.radians(10.0)), 0.025 / MU0 * math.sin(math.radians(10.0)), 0.0])
        for _ in range(c["nsteps"]):
            m = _rk4(lambda q: _rate(q, ex.exchange(q, AEX) + ex.demag(q) + h0, MS, c["alpha"]), m, c["dt"])
        return m.reshape(-1)
    lam = 1e-2 * torch.randn(3 * n, dtype=torch.float64, device="cuda", generator=g)
    s = X / X.max(axis=0)
    ku = _vec(2e5 + 5e4 * np.cos(2 * math.pi * s[:, 0]) * np.sin(4 * math.pi * s[:, 1])).requires_grad_(True)
    h0 = _vec([0.0, 0.05 / MU0, 0.0]).requires_grad_(True)
    m = m.clone().requires_grad_(True)
    out = _rk4(lambda q: _rate(q, ex.exchange(q, AEX) + ex.demag(q) + _uniaxial(q, ku[:, None], MS) + h0, MS, 0.1), m,
               c["dt"])
    gm, gk, gh = torch.autograd.grad((out.reshape(-1) * lam).sum(), (m, ku, h0))
    return gm.reshape(-1), gk, gh


def _exact_newton(ex, lin, m, v, h0, alpha):
    """shift v - J v and the preconditioner's inverse 3x3 blocks applied to it (the linear field's
    mean absolute diagonal kappa stands for its derivative)."""
    H = lin(m) + h0
    k = GAMMA / (1.0 + alpha * alpha)
    stab = 0.5 * MS * k
    Hv = lin(v)

    def dot(a, b):
        return (a * b).sum(1, keepdim=True)

    cr = torch.linalg.cross
    damp = v * dot(m, H) - 2.0 * H * dot(m, v) + m * (dot(v, H) + dot(m, Hv)) - Hv * dot(m, m)
    jv = -k * (cr(v, H) + cr(m, Hv) + alpha * damp) + stab * ((1.0 - dot(m, m)) * v - 2.0 * m * dot(m, v))
    y = SHIFT * v - jv
    diag = -2.0 * AEX / (MU0 * MS) * 1e18 / ex.vol * ex.nodal(ex.tv[:, None] * (ex.g * ex.g).sum(2))
    d = torch.stack([diag, diag, diag + 2.0 * 5e5 / (MU0 * MS)], 1)
    kap = (d.abs().sum(1) / 3.0)[:, None]
    cols = []
    for q in range(3):
        e = torch.zeros_like(m)
        e[:, q] = 1.0
        # precession and damping for the local field H_e = kappa e, in the sign that the
        # preconditioner's definition gives them (the reference's block kernel)
        prec = cr(e, H) + kap * cr(m, e)
        damp = e * dot(m, H) - 2.0 * H * dot(m, e) + m * dot(e, H) + kap * (m * dot(m, e) - e * dot(m, m))
        cols.append(k * prec + k * alpha * damp + stab * ((1.0 - dot(m, m)) * e - 2.0 * m * dot(m, e)))
    J = torch.stack(cols, 2)
    A = (SHIFT + 1e-14) * torch.eye(3, dtype=torch.float64, device="cuda") - J
    return y.reshape(-1), torch.linalg.solve(A, y).reshape(-1)


def _exact_ensemble(c, seed):
    boxes = _boxes(c["samples"], c["draw"])
    counts = [_counts(*b)[0] for b in boxes]
    if sum(float(n) ** 3 for n in counts) > 3e13:
        return None
    Bz = np.random.default_rng(c["draw"] + 100).uniform(-0.5, 0.5, size=c["samples"])
    m0 = _unit(sum(counts), _gen(seed)).view(-1, 3).split(counts)
    out = []
    for box, b, m in zip(boxes, Bz, m0):
        X, T = _mesh(*box, 2.0, 0.0)
        ex = _Exact(X, T, 1.1e6)
        h0 = _vec([0.0, 0.0, b / MU0])
        for _ in range(c["nsteps"]):
            m = _rk4(lambda q: _rate(q, ex.exchange(q, 1.6e-11) + ex.dmi(q, 3e-3) + _uniaxial(q, 8e5, 1.1e6)
                                     + ex.demag(q) + h0, 1.1e6, 0.3), m, c["dt"])
        out.append(m)
    return torch.cat(out).reshape(-1)
