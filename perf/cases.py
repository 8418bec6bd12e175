"""The work a user of this framework has it do, as timed cases.

Two layers are called.  The interaction product (AProductCore.Aproduct and its device and
FP32 forms) is the one operation that every solver step repeats; users with their own Krylov
method call it directly.  The solves (DDAModel.bicgstab / solve_mixed, solve_batch,
solve_multi, the topology step, one wavelength of a spectrum) are the whole calls.

Sizes are the repository's own: the lattices of ``lattice.config`` and the tests, and the
range of the served stream (16 to 128 cells in x and y, up to 32 in z, any length between).
Solves run to 1e-11: the iterates of a Krylov method carry rounding differences up to the
level of the tolerance, so only solutions converged well past single precision are the same
numbers from one build, batch or wavelength grid to the next.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "topo-dda-forwin64_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import tdda  # noqa: E402
from tdda import lattice, topo  # noqa: E402

TOL = 1e-11
MAX_IT = 10000


def listed():
    return [
        # The smallest calls: one product of a particle of a few hundred dipoles on host
        # arrays, as a program that steps its own solver over small particles makes them.
        dict(name="product64 host 8x7x5 holes", kind="product", Nx=8, Ny=7, Nz=5, fill=0.7, fp32=False, host=True),
        # FP64 products on device vectors: a thin film pixel at an ordinary size (the
        # lattice of the single-solve workload), and an odd one with the particle inside
        # its box (a sphere or a ligand shell leaves cells empty).
        dict(name="product64 64x64x16", kind="product", Nx=64, Ny=64, Nz=16, fill=1.0, fp32=False, host=False),
        dict(name="product64 37x51x13 holes", kind="product", Nx=37, Ny=51, Nz=13, fill=0.6, fp32=False, host=False),
        # Single-precision products: error studies and inner steps of a user's own
        # refinement.  An odd lattice of the served range, and the largest of it.
        dict(name="product32 41x90x23", kind="product", Nx=41, Ny=90, Nz=23, fill=1.0, fp32=True, host=False),
        dict(name="product32 128x128x32", kind="product", Nx=128, Ny=128, Nz=32, fill=1.0, fp32=True, host=False),
        # The drop-in FP64 solve of the reference's own small workload (random densities).
        dict(name="solve64 20x20x10", kind="solve", Nx=20, Ny=20, Nz=10, density="uniform", eps=4.0, loss=0.1,
             lam=500.0, d=10.0, precision="fp64", rhs=1),
        # One evaluation of a design: new densities in, refined mixed solve, P and the
        # internal field out (the headline workload's lattice and densities).
        dict(name="solve32 64x64x16 smooth", kind="solve", Nx=64, Ny=64, Nz=16, density="smooth", eps=6.25, loss=0.05,
             lam=600.0, d=10.0, precision="refine", rhs=1),
        # A particle of holes and odd lengths, as a user's geometry file gives it.
        dict(name="solve32 45x33x19 holes", kind="solve", Nx=45, Ny=33, Nz=19, density="holes", eps=4.0, loss=0.1,
             lam=520.0, d=10.0, precision="auto", rhs=2),
        # Eight incidences (two polarisations, four angles) on one binary structure.
        dict(name="batch32 96x96x24 x8", kind="solve", Nx=96, Ny=96, Nz=24, density="binary", eps=4.0, loss=0.1,
             lam=550.0, d=8.0, precision="auto", rhs=8),
        # One evaluation of the topology loop: forward and three adjoint solves in a batch,
        # objective at the focus, gradient back to the design.
        dict(name="topology step 80x80x20", kind="topo", Nx=80, Ny=80, Nz=20, eps=4.0, loss=0.1, lam=500.0, d=10.0),
        # A sweep's structures that share a grid shape, solved together (the served stream).
        dict(name="multi32 4 lattices <=56x60x22", kind="multi", Nx=56, Ny=60, Nz=22, count=4, eps=4.0, loss=0.1,
             lam=560.0, d=10.0),
        # One wavelength of a spectrum: a new operator (its Green spectrum), a model, the
        # solve and the fields (the reference builds a core per wavelength).
        dict(name="spectrum point 40x40x12", kind="spectrum", Nx=40, Ny=40, Nz=12, eps=4.0, loss=0.1, lam=540.0, d=10.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "product", "solve", "solve", "multi", "spectrum", "topo"])
    lam, d = round(rng.uniform(480.0, 700.0), 1), 10.0
    eps, loss = rng.choice([(2.25, 0.0), (4.0, 0.1), (6.25, 0.05)])
    if kind == "product":
        fp32 = rng.random() < 0.5
        host = not fp32 and rng.random() < 0.3
        hi = 24 if host else 128
        lo = 4 if not fp32 else 16
        return dict(kind=kind, Nx=_log_int(rng, lo, hi), Ny=_log_int(rng, lo, hi), Nz=_log_int(rng, lo, min(hi, 32)),
                    fill=rng.choice([1.0, 1.0, 0.6]), fp32=fp32, host=host)
    Nx, Ny, Nz = _log_int(rng, 16, 80), _log_int(rng, 16, 80), _log_int(rng, 8, 20)
    if kind == "solve":
        precision = rng.choice(["refine", "auto", "auto", "fp64"])
        if precision == "fp64":  # the drop-in solve at its usual sizes
            Nx, Ny, Nz = _log_int(rng, 8, 32), _log_int(rng, 8, 32), _log_int(rng, 6, 12)
        density = "smooth" if precision == "refine" else rng.choice(["uniform", "binary", "holes"])
        return dict(kind=kind, Nx=Nx, Ny=Ny, Nz=Nz, density=density, eps=4.0, loss=0.1, lam=lam, d=d,
                    precision=precision, rhs=1 if precision == "fp64" else rng.choice([1, 2, 4]))
    if kind == "topo":
        return dict(kind=kind, Nx=Nx, Ny=Ny, Nz=Nz, eps=4.0, loss=0.1, lam=lam, d=d)
    if kind == "multi":
        return dict(kind=kind, Nx=max(24, Nx), Ny=max(24, Ny), Nz=max(16, Nz), count=rng.choice([2, 4]), eps=4.0,
                    loss=0.1, lam=lam, d=d)
    return dict(kind=kind, Nx=Nx, Ny=Ny, Nz=Nz, eps=eps, loss=loss, lam=lam, d=d)


# ------------------------------------------------------------------ inputs from a seed
def _rng(seed, salt):
    return np.random.Generator(np.random.PCG64([int(seed), salt]))


def _sites(Nx, Ny, Nz, fill, rng):
    """The lattice sites (3N int32): the full box, or a random part of it listed in x, y, z order."""
    R = lattice.bulk(Nx, Ny, Nz)
    if fill >= 1.0:
        return R
    n = Nx * Ny * Nz
    keep = np.sort(rng.permutation(n)[:max(1, int(fill * n))])
    return np.ascontiguousarray(R.reshape(-1, 3)[keep].ravel())


def _densities(kind, Nx, Ny, Nz, R, rng):
    """Densities of the dipoles, one each: U[0,1], its 3x3x3 mean, 0/1, or U[0,1] on a part of the box."""
    full = rng.random((Nx, Ny, Nz))
    if kind == "smooth":
        full = np.clip(lattice.box_filter3(full), 0.0, 1.0)
    elif kind == "binary":
        full = (full < 0.4).astype(np.float64)
    r = R.reshape(-1, 3)
    return np.repeat(full[r[:, 0], r[:, 1], r[:, 2]], 3)


def _incidences(n):
    """n of the eight incidences: x/y polarisation at 0, 15, 30, 45 degrees in the xz plane."""
    return lattice.config(3).incidences[:n]


def _solve_setup(case, seed):
    rng = _rng(seed, 11)
    Nx, Ny, Nz = case["Nx"], case["Ny"], case["Nz"]
    R = _sites(Nx, Ny, Nz, 0.7 if case["density"] == "holes" else 1.0, rng)
    diel = _densities("uniform" if case["density"] == "holes" else case["density"], Nx, Ny, Nz, R, rng)
    return R, diel, np.array([1.0 + 0j, complex(case["eps"], case["loss"])])


def _multi_setup(case, seed):
    """The lattices of a cross-lattice batch: boxes at most 3 cells smaller than the case's on
    each axis that share its FFT grid, with their own wavelength, material and densities."""
    rng = _rng(seed, 12)
    top = (case["Nx"], case["Ny"], case["Nz"])
    out = []
    for k in range(case["count"]):
        box = []
        for a, n in enumerate(top):
            m = max(1, n - (k * (a + 1)) % 4)
            while lattice.fft_length(m, a == 2) != lattice.fft_length(n, a == 2):
                m += 1
            box.append(m)
        lam = case["lam"] * (1.0 + 0.05 * k)
        eps = complex(case["eps"], case["loss"]) * (1.0 - 0.1 * (k % 2))
        out.append((tuple(box), lattice.bulk(*box), lam, np.array([1.0 + 0j, eps]),
                    np.repeat(rng.random(box[0] * box[1] * box[2]), 3)))
    return out


def _spectrum_workload(case, seed):
    rng = _rng(seed, 13)
    Nx, Ny, Nz = case["Nx"], case["Ny"], case["Nz"]
    rho = np.clip(lattice.box_filter3(rng.random((Nx, Ny, Nz))), 0.0, 1.0).ravel()
    return lattice.Workload(name="spectrum", Nx=Nx, Ny=Ny, Nz=Nz, d=case["d"], lam=case["lam"],
                            material=np.array([1.0 + 0j, complex(case["eps"], case["loss"])]), rho=rho,
                            R=lattice.bulk(Nx, Ny, Nz), incidences=[lattice.XPOL_Z], tol=TOL, max_it=MAX_IT)


def _topo_theta(case, seed):
    return 0.4 + 0.2 * _rng(seed, 14).random(((case["Nx"] + 1) // 2, (case["Ny"] + 1) // 2))


def _topo_focus(case):
    d = case["d"]
    return (0.5 * d * (case["Nx"] - 1), 0.5 * d * (case["Ny"] - 1), d * (case["Nz"] + 5))


def _pinned(a):
    """Host densities in page-locked memory, as a program that sends new ones every step keeps them."""
    return torch.from_numpy(a).pin_memory().numpy()


def _fields(n3):
    """Where a program that goes on with the fields on the GPU has them: P and the internal field."""
    return tuple(torch.empty(n3, dtype=torch.complex128, device="cuda") for _ in range(2))


def _read_fields(model, out):
    """P and the internal field into the caller's device tensors, through the C interface."""
    model.update_E_in_structure()
    for field, t in zip((tdda.FIELD_P, tdda.FIELD_EINTERNAL), out):
        if tdda.load().tdda_model_get(model.h, field, t.data_ptr(), tdda.MEM_DEVICE) != tdda.OK:
            raise RuntimeError(tdda.load().tdda_last_error().decode())
    return out


PRECISION = {"fp64": tdda.FP64, "refine": tdda.FP32_REFINE, "auto": tdda.FP32_AUTO}


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "product":
        rng = _rng(seed, 10)
        R = _sites(case["Nx"], case["Ny"], case["Nz"], case["fill"], rng)
        core = tdda.AProductCore(case["Nx"], case["Ny"], case["Nz"], R, 10.0, 550.0, np.array([1.0, 4.0 + 0.1j]))
        b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
        state.update(core=core, R=R, b=b)
        if not case["host"]:
            state["db"] = torch.from_numpy(b).cuda()
            state["dy"] = torch.empty_like(state["db"])
            torch.cuda.synchronize()
    elif kind == "solve":
        R, diel, mat = _solve_setup(case, seed)
        core = tdda.AProductCore(case["Nx"], case["Ny"], case["Nz"], R, case["d"], case["lam"], mat,
                                 max_rhs=case["rhs"])
        first = np.full(R.size, 0.5)  # the structure the models were created with
        models = [tdda.DDAModel(core, i.nK, i.E0, i.nE0, first) for i in _incidences(case["rhs"])]
        state.update(core=core, models=models, diel=_pinned(diel))
        state["out"] = [_fields(R.size) for _ in models] if case["precision"] != "fp64" else None
    elif kind == "multi":
        cores, models, diels = [], [], []
        for box, R, lam, mat, diel in _multi_setup(case, seed):
            cores.append(tdda.AProductCore(*box, R, case["d"], lam, mat))
            models.append(tdda.DDAModel(cores[-1], (0.0, 0.0, 1.0), 1.0, (1.0, 0.0, 0.0), np.full(R.size, 0.5)))
            diels.append(_pinned(diel))
        state.update(cores=cores, models=models, diels=diels, out=[_fields(m.n3) for m in models])
    elif kind == "topo":
        state["loop"] = topo.TopoLoop(case["Nx"], case["Ny"], case["Nz"], case["d"], case["lam"],
                                      np.array([1.0 + 0j, complex(case["eps"], case["loss"])]), _topo_theta(case, seed),
                                      _topo_focus(case), precision=tdda.FP32_AUTO, tol=TOL, max_it=MAX_IT)
    else:
        state["w"] = _spectrum_workload(case, seed)
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "product":
        precision = tdda.FP32_REFINE if state["case"]["fp32"] else tdda.FP64
        if state["case"]["host"]:
            return state["core"].Aproduct(state["b"], precision)
        state["core"].Aproduct_device(state["db"].data_ptr(), state["dy"].data_ptr(), precision)
        # a single-precision product is kept in single precision
        return state["dy"].to(torch.complex64) if state["case"]["fp32"] else state["dy"]
    if kind == "solve":
        models = state["models"]
        for m in models:
            m.UpdateAlpha(state["diel"])
            m.InitializeP()
        if state["case"]["precision"] == "fp64":
            models[0].bicgstab(MAX_IT, TOL)
            models[0].update_E_in_structure()
            return [(models[0].get_P(), models[0].get_Einternal())]
        tdda.solve_batch(models, PRECISION[state["case"]["precision"]], MAX_IT, TOL)
        return [_read_fields(m, out) for m, out in zip(models, state["out"])]
    if kind == "multi":
        for m, diel in zip(state["models"], state["diels"]):
            m.UpdateAlpha(diel)
            m.InitializeP()
        tdda.solve_multi(state["models"], MAX_IT, TOL, precision=tdda.FP32_AUTO)
        return [_read_fields(m, out) for m, out in zip(state["models"], state["out"])]
    if kind == "topo":
        r = state["loop"].evaluate()
        return r.objective, r.grad_theta
    s = tdda.solve_workload(state["w"], tdda.FP32_REFINE)
    return s.P, s.Einternal


# ------------------------------------------------------------------ the least work
def _product_work(Nx, Ny, Nz, N, item):
    """One product on the padded grid of 2N points an axis: the vector in and out, the folded
    spectrum of the six tensor components once, and the pruned transforms (only lines that
    hold data forward, only lines that are kept back) at 5 M log2 M a line."""
    Mx, My, Mz = (max(1, 2 * n) for n in (Nx, Ny, Nz))
    green = 6 * (Nx + 1) * (Ny + 1) * (Nz + 1) * item
    lines = Nx * Ny * _fft(Mz) + Nx * Mz * _fft(My) + My * Mz * _fft(Mx)
    return 2 * 3 * N * item, green, 2 * 3 * lines + 72.0 * Mx * My * Mz


def _fft(M):
    return 5.0 * M * math.log2(M) if M > 1 else 0.0


def _solve_work(Nx, Ny, Nz, N, rhs, item, steps):
    """`steps` steps of two products: the operator is read once (it fits on chip across the
    steps only in part, so once is the least), each right-hand side's field and densities are
    read and its solution and field written."""
    _, green, flops = _product_work(Nx, Ny, Nz, N, item)
    return {"bytes": green + rhs * 3.0 * N * (8 + 16 + 16 + 16), "flops": 2.0 * steps * rhs * flops}


def work(case):
    Nx, Ny, Nz = case["Nx"], case["Ny"], case["Nz"]
    N = Nx * Ny * Nz
    kind = case["kind"]
    if kind == "product":
        n = max(1, int(N * case["fill"]))
        vec, green, flops = _product_work(Nx, Ny, Nz, n, 8 if case["fp32"] else 16)
        return {"bytes": float(vec + green), "flops": flops}
    if kind == "solve":  # steps of a well-conditioned lattice at this tolerance
        steps = 60 if case["precision"] == "refine" else 100 if case["precision"] == "fp64" else 25
        n = int(N * 0.7) if case["density"] == "holes" else N
        return _solve_work(Nx, Ny, Nz, n, case["rhs"], 16 if case["precision"] == "fp64" else 8, steps)
    if kind == "multi":
        w = _solve_work(Nx, Ny, Nz, N, 1, 8, 25)
        return {k: v * case["count"] for k, v in w.items()}
    if kind == "topo":
        return _solve_work(Nx, Ny, Nz, N, 4, 8, 60)
    w = _solve_work(Nx, Ny, Nz, N, 1, 8, 60)
    Mx, My, Mz = 2 * Nx, 2 * Ny, 2 * Nz
    w["flops"] += 6.0 * (Mx * My * _fft(Mz) + Mx * Mz * _fft(My) / 2 + My * Mz * _fft(Mx) / 4)
    return w


# ------------------------------------------------------------------ the same in 64 bits
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tensor(K, x, y, z):
    """The LDR interaction tensor at offsets x, y, z: xx, xy, xz, yy, yz, zz, zero at the origin."""
    r2 = x * x + y * y + z * z
    zero = r2 == 0
    r = torch.sqrt(torch.where(zero, torch.ones_like(r2), r2))
    c1 = torch.exp(1j * K * r) / r ** 3
    c2 = (1.0 - 1j * K * r) / r ** 2
    c3 = K * K - 3.0 * c2
    xs, ys, zs = x * x, y * y, z * z
    t = [c1 * (c2 * (r * r - 3 * xs) - K * K * (ys + zs)), c1 * (x * y * c3), c1 * (z * x * c3),
         c1 * (c2 * (r * r - 3 * ys) - K * K * (zs + xs)), c1 * (y * z * c3),
         c1 * (c2 * (r * r - 3 * zs) - K * K * (xs + ys))]
    return [torch.where(zero, torch.zeros_like(v), v) for v in t]


class _Operator:
    """y = A_offdiag b in complex128 by torch.fft on the grid of 2N points an axis."""

    def __init__(self, Nx, Ny, Nz, R, d, K):
        self.dev = _dev()
        self.box = (Nx, Ny, Nz)
        self.M = tuple(2 * n for n in self.box)
        ax = []
        for n in self.box:
            k = torch.arange(2 * n, dtype=torch.float64, device=self.dev)
            ax.append(torch.where(k < n, k, k - 2 * n) * d)
        x, y, z = torch.meshgrid(*ax, indexing="ij")
        keep = (x > -Nx * d) & (y > -Ny * d) & (z > -Nz * d)  # the offset -N is never used
        self.G = [torch.fft.fftn(torch.where(keep, t, torch.zeros_like(t))) for t in _tensor(K, x, y, z)]
        r = torch.from_numpy(np.asarray(R, np.int64).reshape(-1, 3)).to(self.dev)
        self.cell = (r[:, 0] * Ny + r[:, 1]) * Nz + r[:, 2]

    def __call__(self, b):
        Nx, Ny, Nz = self.box
        X = []
        for c in range(3):
            g = torch.zeros(Nx * Ny * Nz, dtype=torch.complex128, device=self.dev)
            g[self.cell] = b.reshape(-1, 3)[:, c]
            X.append(torch.fft.fftn(g.reshape(self.box), s=self.M))
        G = self.G
        Y = (G[0] * X[0] + G[1] * X[1] + G[2] * X[2], G[1] * X[0] + G[3] * X[1] + G[4] * X[2],
             G[2] * X[0] + G[4] * X[1] + G[5] * X[2])
        out = [torch.fft.ifftn(v)[:Nx, :Ny, :Nz].reshape(-1)[self.cell] for v in Y]
        return torch.stack(out, dim=1).reshape(-1)


def _material(mat):
    return [m + 0.01 if abs(m) <= 1.01 else m for m in mat]


def _alpha_inverse(diel, mat, K, d, nK, nE0):
    """eps of the densities in [0, 1] and 1 / alpha of the lattice dispersion relation."""
    m = _material([complex(v) for v in mat])
    rho = (diel if isinstance(diel, torch.Tensor) else torch.from_numpy(diel)).to(_dev())
    eps = m[0] + rho * (m[1] - m[0])
    b1, b2, b3 = -1.891531, 0.1648469, -1.7700004
    S = float(np.sum((np.asarray(nE0) * np.asarray(nK)) ** 2))
    a1 = (3 * d ** 3 / (4 * math.pi)) * (eps - 1) / (eps + 2)
    res = 1 + (a1 / d ** 3) * ((b1 + eps * b2 + eps * b3 * S) * (K * d) ** 2 - 1j * (2.0 / 3.0) * (K * d) ** 3)
    return eps, res / a1


def _incident(R, d, K, inc):
    r = torch.from_numpy(np.asarray(R, np.float64).reshape(-1, 3)).to(_dev()) * d
    k = torch.tensor(np.asarray(inc.nK, np.float64), device=r.device)
    e = torch.tensor(np.asarray(inc.nE0, np.float64) * inc.E0, device=r.device)
    return (torch.exp(1j * K * (r @ k))[:, None] * e[None, :]).reshape(-1)


def _bicgstab(A, b, tol, limit):
    x = torch.zeros_like(b)
    r = b.clone()
    r0, p, rho = r.clone(), r.clone(), torch.vdot(r, r)
    nb = torch.linalg.norm(b)
    for it in range(limit):
        v = A(p)
        alpha = rho / torch.vdot(r0, v)
        s = r - alpha * v
        t = A(s)
        w = torch.vdot(t, s) / torch.vdot(t, t)
        x = x + alpha * p + w * s
        r = s - w * t
        if it % 4 == 3 and float(torch.linalg.norm(r)) <= tol * float(nb):
            break
        rho, old = torch.vdot(r0, r), rho
        p = r + (rho / old) * (alpha / w) * (p - w * v)
    return x


def _solve_exact(op, al, E):
    """P of (A + al) P = E to about 1e-14 of |E|: diagonal right preconditioning, refined."""
    P = torch.zeros_like(E)
    for _ in range(6):
        r = E - (op(P) + al * P)
        if float(torch.linalg.norm(r)) <= 3e-15 * float(torch.linalg.norm(E)):
            break
        P = P + _bicgstab(lambda v: op(v / al) + v, r, 1e-7, 600) / al
    return P


def _design(theta, Nx, Ny, Nz):
    """Densities (three a dipole) of the design parameters on one quadrant: mirrored in x and y, cone
    filter of radius 2 in the plane, extruded along z."""
    ix = torch.minimum(torch.arange(Nx), Nx - 1 - torch.arange(Nx)).to(theta.device)
    iy = torch.minimum(torch.arange(Ny), Ny - 1 - torch.arange(Ny)).to(theta.device)
    k = torch.zeros(5, 5, dtype=torch.float64, device=theta.device)
    for a in range(-2, 3):
        for b in range(-2, 3):
            if a * a + b * b <= 4.0 - 0.01:
                k[a + 2, b + 2] = 2.0 - math.hypot(a, b)
    full = theta[ix][:, iy][None, None]
    conv = torch.nn.functional.conv2d
    rho = conv(full, k[None, None], padding=2) / conv(torch.ones_like(full), k[None, None], padding=2)
    return rho[0, 0].reshape(-1).repeat_interleave(3 * Nz)


def _topo_exact(case, seed, K):
    """|E|^2 at the focus and its gradient by the adjoint method."""
    Nx, Ny, Nz, d = case["Nx"], case["Ny"], case["Nz"], case["d"]
    R = lattice.bulk(Nx, Ny, Nz)
    mat = [1.0, complex(case["eps"], case["loss"])]
    theta = torch.from_numpy(_topo_theta(case, seed)).to(_dev()).requires_grad_(True)
    inc = lattice.XPOL_Z
    _, al = _alpha_inverse(_design(theta, Nx, Ny, Nz), mat, K, d, inc.nK, inc.nE0)
    fixed = al.detach()
    op = _Operator(Nx, Ny, Nz, R, d, K)
    P = _solve_exact(op, fixed, _incident(R, d, K, inc))
    r = torch.from_numpy(R.astype(np.float64).reshape(-1, 3)).to(_dev()) * d
    o = torch.tensor(_topo_focus(case), dtype=torch.float64, device=r.device)
    t = _tensor(K, *(o[a] - r[:, a] for a in range(3)))
    rows = [torch.stack([t[i] for i in row], dim=1).reshape(-1) for row in ((0, 1, 2), (1, 3, 4), (2, 4, 5))]
    phase = torch.exp(1j * K * (o @ torch.tensor(np.asarray(inc.nK), device=r.device)))
    E = [float(inc.nE0[k]) * inc.E0 * phase - torch.sum(rows[k] * P) for k in range(3)]
    lam = sum(torch.conj(E[k]) * _solve_exact(op, fixed, -rows[k]) for k in range(3))
    (-2.0 * torch.sum((lam * P * al).real)).backward()
    return float(sum(abs(complex(e)) ** 2 for e in E)), theta.grad


def _wave_number(lam):
    return 2 * math.pi / lam


def exact(case, seed):
    kind = case["kind"]
    box = (case["Nx"], case["Ny"], case["Nz"])
    if kind == "product":
        rng = _rng(seed, 10)
        R = _sites(*box, case["fill"], rng)
        b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
        y = _Operator(*box, R, 10.0, _wave_number(550.0))(torch.from_numpy(b).to(_dev()))
        return y.cpu().numpy() if case["host"] else y
    K = _wave_number(case["lam"])
    d = case["d"]
    if kind == "solve":
        R, diel, mat = _solve_setup(case, seed)
        op = _Operator(*box, R, d, K)
        out = []
        for inc in _incidences(case["rhs"]):
            eps, al = _alpha_inverse(diel, mat, K, d, inc.nK, inc.nE0)
            P = _solve_exact(op, al, _incident(R, d, K, inc))
            out.append((P, al * P / ((2 + eps) / 3)))
        return out
    if kind == "multi":
        out = []
        inc = lattice.XPOL_Z
        for b, R, lam, mat, diel in _multi_setup(case, seed):
            Kl = _wave_number(lam)
            eps, al = _alpha_inverse(diel, mat, Kl, d, inc.nK, inc.nE0)
            P = _solve_exact(_Operator(*b, R, d, Kl), al, _incident(R, d, Kl, inc))
            out.append((P, al * P / ((2 + eps) / 3)))
        return out
    if kind == "spectrum":
        w = _spectrum_workload(case, seed)
        inc = w.incidences[0]
        eps, al = _alpha_inverse(w.diel_old, w.material, K, d, inc.nK, inc.nE0)
        P = _solve_exact(_Operator(*box, w.R, d, K), al, _incident(w.R, d, K, inc))
        return P, al * P / ((2 + eps) / 3)
    return _topo_exact(case, seed, K)
