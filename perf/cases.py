"""The work a user of this framework has it do: runs of a few time steps from
an initial state, through the Solver interface, over the models, cell kinds,
solver forms and mesh sizes that the package's workloads, tests and benchmark
use.

A pass sets the initial state and advances it by the case's time steps; its
results are the face traces and cell averages, viewed on the device (as a
model's hook or a coupled GPU program reads them).  A learned-form pass also
returns the network's parameters after its online training.
"""
import math
import sys
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "tnl-mhfem_gb300"))

from mhfem import _lib as L  # noqa: E402
from mhfem import problems  # noqa: E402

FORMS = {"fp64": L.FORM_FP64, "mixed": L.FORM_MIXED, "learned": L.FORM_LEARNED}


def _case(name, model, N, form="fp64", solver="bicgstab", steps=1, tol=1e-13):
    c = {"model": model, "N": N, "form": form, "solver": solver, "steps": steps, "tol": tol}
    return dict(c, name=name) if name else c


def listed():
    # The model tolerances: 1e-12 for the heat equation (its workload's own);
    # 1e-13 for the others, the tolerance at which the tests and the benchmark
    # compare the forms with one another.
    return [
        # the smallest run: a teaching or regression mesh, where a step is launch latency
        _case("heat_tri_16", "heat_tri", 16, steps=4, tol=1e-12),
        # the plain FP64 heat equation on 128^2 squares split into triangles
        _case("heat_tri_128", "heat_tri", 128, steps=4, tol=1e-12),
        # the same equation with the reference example's solver, GMRES with restart length 3 to 30
        _case("heat_tri_100_gmres", "heat_tri", 100, solver="gmres", steps=2, tol=1e-12),
        # rectangles, an odd grid
        _case("heat_rect_211", "heat_rect", 211, steps=2, tol=1e-12),
        # two-component advection-diffusion-reaction: a parameter study's mesh, and the full workload's
        _case("adr_tri_90", "adr_tri", 90, steps=4),
        _case("adr_tri_512", "adr_tri", 512, steps=2),
        # heterogeneous diffusion on tetrahedra: a coarse mesh, a medium one, the full workload
        _case("diffusion_tet_21", "diffusion_tet", 21, steps=2),
        _case("diffusion_tet_37", "diffusion_tet", 37, steps=2),
        _case("diffusion_tet_64", "diffusion_tet", 64, steps=2),
        # the same in mixed precision
        _case("diffusion_tet_64_mixed", "diffusion_tet", 64, form="mixed", steps=2),
        # heterogeneous diffusion on cuboids
        _case("diffusion_box_56", "diffusion_box", 56, steps=2),
        # the time-varying source with the learned warm start, trained online
        _case("diffusion_tet_40_learned", "diffusion_tet", 40, form="learned", steps=4),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    steps = rng.randint(1, 4)
    kind = rng.randrange(9)
    if kind == 0:
        return _case(None, "heat_tri", size(8, 384), steps=steps, tol=1e-12)
    if kind == 1:
        return _case(None, "heat_rect", size(8, 384), steps=steps, tol=1e-12)
    if kind == 2:
        return _case(None, "heat_tri", size(8, 160), solver="gmres", steps=steps, tol=1e-12)
    if kind == 3:
        return _case(None, "adr_tri", size(8, 512), steps=steps)
    if kind == 4:
        return _case(None, "diffusion_tet", size(5, 60), steps=min(steps, 2))
    if kind == 5:
        return _case(None, "diffusion_tet", size(5, 60), form="mixed", steps=min(steps, 2))
    if kind == 6:
        return _case(None, "diffusion_box", size(6, 64), steps=min(steps, 2))
    if kind == 7:
        return _case(None, "diffusion_tet", size(8, 40), form="learned", steps=max(steps, 3))
    return _case(None, "diffusion_tet", size(5, 24), solver="gmres", steps=min(steps, 2))


# ---- inputs ---------------------------------------------------------------------


def _bump(p, N, seed):
    """A Gaussian bump at a seeded place as the initial cell values."""
    rng = np.random.default_rng(seed)
    at = rng.uniform(0.35, 0.65, 2)
    cen = p.coords[p.cells].mean(axis=1)
    return np.exp(-50.0 * ((cen - at) ** 2).sum(axis=1))


@lru_cache(maxsize=2)
def _problem(model, N, form, tol, seed):
    f = FORMS[form]
    if model == "heat_tri":
        p = problems.heat2d(N=N, tol=tol, seed=seed, form=f)
        p.Z0 = _bump(p, N, seed)
    elif model == "heat_rect":
        p = problems.heat2d_rect(N=N, tol=tol, form=f)
        p.Z0 = _bump(p, N, seed)
    elif model == "adr_tri":
        p = problems.adr2d(N=N, tol=tol, seed=seed, field_seed=seed + 1, form=f)
    elif model == "diffusion_box":
        p = problems.diffusion3d_box(N=N, tol=tol, field_seed=seed + 1, form=f)
    elif form == "learned":
        # period 1000 dt, the online-training workload's
        p = problems.diffusion3d_source(N=N, tol=tol, seed=seed, field_seed=seed + 1, psi_seed=seed + 2, form=f)
    else:
        p = problems.diffusion3d(N=N, tol=tol, seed=seed, field_seed=seed + 1, form=f)
    return p


def _make(case, seed):
    return _problem(case["model"], case["N"], case["form"], case["tol"], 3 * int(seed) + 11)


def prepare(case, seed):
    p = _make(case, seed)
    s = problems.make_solver(p)
    if case["solver"] == "gmres":
        s.setup(tol=p.tol, max_iter=20000, linear_solver="gmres", gmres_restart=30, gmres_restart_min=3,
                gmres_restart_step_min=3, gmres_restart_step_max=3)
    params = None
    if case["form"] == "learned":
        # every step trains (two Adam iterations) and tries the guess
        s.learned_options(train_steps=1 << 30, train_iters=2, learning_rate=3e-3, use_during_training=True,
                          seed=int(seed) + 1)
        params = s.learned_params()
    views = {}
    for name in ("Z_iF", "Z_iK"):
        a = s.array_device(name)
        a.solver = s  # the view keeps its owner alive
        views[name] = torch.as_tensor(a, device="cuda")
    return {"solver": s, "Z0": p.Z0, "dt": p.dt, "steps": case["steps"], "params": params, "views": views}


def run(state):
    s, dt = state["solver"], state["dt"]
    s.setInitialCondition(state["Z0"])
    if state["params"] is not None:
        s.set_learned_params(state["params"])
    for k in range(state["steps"]):
        s.step(k * dt, dt, stats=False)
    out = dict(state["views"])
    if state["params"] is not None:
        out["params"] = s.learned_params()
    return out


# ---- sizes ----------------------------------------------------------------------


def _sizes(case):
    """Cells, faces, equations, faces and vertices per cell."""
    N, m = case["N"], case["model"]
    if m in ("heat_tri", "adr_tri"):
        return 2 * N * N, 3 * N * N + 2 * N, 2 if m == "adr_tri" else 1, 3, 3
    if m == "heat_rect":
        return N * N, 2 * N * (N + 1), 1, 4, 4
    if m == "diffusion_box":
        return N ** 3, 3 * N * N * (N + 1), 1, 6, 8
    return 6 * N ** 3, 12 * N ** 3 + 6 * N * N, 1, 4, 4


def work(case):
    """Per step: the mesh and the coefficients read, the state read and written, the face system (values,
    columns, right-hand side) written and read once.  The Krylov iterations' own traffic depends on their
    number and is left out."""
    C, F, n, nf, nv = _sizes(case)
    rows, width = n * F, (2 * nf - 1) * n
    coef = (2 * n * n + n * n * (nf if case["model"] == "adr_tri" else 0)) * 8 * C
    system = rows * (12 * width + 8)
    b = 4 * (nv + nf) * C + coef + 2 * 8 * (n * C + rows) + 2 * system
    fl = C * (n * nf) ** 2 * 6 + 2 * rows * width
    if case["form"] == "learned":  # two Adam iterations: the layers' products, forward and backward
        fl += 2 * 3 * 2 * F * (16 * 64 + 3 * 128 * 64)
        b += 2 * 2 * F * 64 * 2 * 4
    return {"bytes": b * case["steps"], "flops": fl * case["steps"]}


# ---- the same steps in 64 bits, in plain torch ------------------------------------

_BOX_FACES = {2: [[0, 1], [1, 2], [2, 3], [3, 0]],
              3: [[0, 1, 2, 3], [0, 1, 5, 4], [1, 2, 6, 5], [2, 3, 7, 6], [3, 0, 4, 7], [4, 5, 6, 7]]}
_BOX_AXIS = {2: [1, 0, 1, 0], 3: [2, 1, 0, 1, 0, 2]}  # the axis each face is normal to


def _faces(cells, V, box, dim):
    """cell -> face numbers (order of first appearance over cells and local faces), face -> its two (cell, local face)
    slots (-1: none), face -> its vertices."""
    C, nv = cells.shape
    local = _BOX_FACES[dim] if box else [[v for v in range(nv) if v != e] for e in range(nv)]
    nf = len(local)
    f = torch.stack([cells[:, q] for q in local], dim=1).reshape(C * nf, -1)
    f = f.sort(dim=1).values
    key = torch.zeros(C * nf, dtype=torch.int64, device=cells.device)
    for k in range(min(f.shape[1], 3)):  # three vertices identify a face
        key = key * V + f[:, k]
    uniq, inv = torch.unique(key, return_inverse=True)
    F = uniq.numel()
    slot = torch.arange(C * nf, device=cells.device)
    first = torch.full((F,), C * nf, dtype=torch.int64, device=cells.device).scatter_reduce(0, inv, slot, "amin")
    last = torch.full((F,), -1, dtype=torch.int64, device=cells.device).scatter_reduce(0, inv, slot, "amax")
    order = first.argsort()
    rank = torch.empty_like(order)
    rank[order] = torch.arange(F, device=cells.device)
    first, last = first[order], last[order]
    return rank[inv].reshape(C, nf), first, torch.where(last == first, torch.full_like(last, -1), last), f[first]


def _local_inverse(X, box, dim, lumped):
    """The inverse RT0 mass matrix of every cell (coefficient 1), and the cells' measures."""
    if box:
        h = X[:, 2 if dim == 2 else 6] - X[:, 0]
        meas = h.prod(dim=1)
        ax = _BOX_AXIS[dim]
        B = X.new_zeros(X.shape[0], 2 * dim, 2 * dim)
        for e, a in enumerate(ax):
            for g, c in enumerate(ax):
                if a == c:
                    B[:, e, g] = (4 if e == g else 2) * meas / h[:, a] ** 2
        return B, meas
    edges = X[:, 1:] - X[:, :1]
    meas = torch.linalg.det(edges).abs() / math.factorial(dim)
    d = X.unsqueeze(1) - X.unsqueeze(2)  # d[K, e, v] = X_v - X_e
    G = torch.einsum("kevx,kfvx->kef", d, d)
    if lumped:
        M = G / (dim + 1)
    else:
        s = d.sum(dim=2)
        M = (G + torch.einsum("kex,kfx->kef", s, s)) / ((dim + 1) * (dim + 2))
    M = M / (dim * dim * meas.reshape(-1, 1, 1))
    return torch.linalg.inv(M), meas


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p = _make(case, seed)
    n, dim, box = p.config.n_eq, p.config.dim, p.config.cell == L.CELL_BOX
    coords = torch.from_numpy(p.coords).to(dev)
    cells = torch.from_numpy(p.cells.astype(np.int64)).to(dev)
    C = cells.shape[0]
    cf, s0, s1, fverts = _faces(cells, coords.shape[0], box, dim)
    nf, F = cf.shape[1], s0.numel()
    interior = s1 >= 0

    def coef(name, shape):
        v = np.asarray(p.coeffs[name], np.float64)
        return torch.from_numpy(v.reshape(shape)).to(dev) if v.size > 1 else None if v == 0 else torch.full(shape, float(v), dtype=torch.float64, device=dev)

    def mat(name):  # (i, j, K) -> [K, i, j]; a uniform value of a one-equation model
        v = coef(name, (n, n, C))
        return torch.zeros(C, n, n, dtype=torch.float64, device=dev) if v is None else v.permute(2, 0, 1)

    B, meas = _local_inverse(coords[cells], box, dim, p.config.mass_lumping)
    D, Nc, r = mat("D"), mat("N"), mat("r")
    a = coef("a", (n, n, nf, C))
    fb = coef("f", (n, C))
    psi = coef("psi", (1, C)) if p.source else None
    be = B.sum(dim=2)
    tau = p.dt
    mt = meas.reshape(-1, 1, 1)
    Qi = torch.linalg.inv(D * be.sum(dim=1).reshape(-1, 1, 1) + mt / tau * Nc + mt * r)
    DQ = D @ Qi
    # per-cell block of the face system, [K, (e, i), (f, j)]
    S = torch.einsum("kij,kef->keifj", D, B) - torch.einsum("kij,ke,kf->keifj", DQ @ D, be, be)
    S = S.reshape(C, nf * n, nf * n)
    rows = (cf.reshape(C, nf, 1) * n + torch.arange(n, device=dev)).reshape(C, nf * n)
    slots = torch.stack([s0, torch.where(interior, s1, s0)], dim=1)  # a face's slots in the per-cell products
    two = interior.to(torch.float64).reshape(F, 1)

    def gather(loc):  # sum of the per-cell face values [K, e, i] over a face's cells -> rows
        loc = loc.reshape(C * nf, n)
        return (loc[slots[:, 0]] + two * loc[slots[:, 1]]).reshape(-1)

    fc = torch.stack([s0 // nf, torch.where(interior, s1 // nf, -torch.ones_like(s1))], dim=1).cpu().numpy()
    tags, _, dval = p.bc_fn(fverts.cpu().numpy(), fc)
    tags = torch.from_numpy(np.asarray(tags).reshape(n, F).T.copy()).to(dev)
    dval = torch.from_numpy(np.asarray(dval, np.float64).reshape(n, F).T.copy()).to(dev)
    fixed = ((~interior).reshape(F, 1) & (tags == 0)).reshape(-1)
    free = (~fixed).to(torch.float64)
    xd = torch.where(fixed, dval.reshape(-1), torch.zeros_like(free))
    outflow = ((~interior).reshape(F, 1) & (tags == 2))

    def A(x):
        return gather(torch.bmm(S, x[rows].unsqueeze(2)))

    diag = gather(torch.diagonal(S, dim1=1, dim2=2).contiguous())
    Zk = torch.from_numpy(p.Z0.reshape(n, C).T.copy()).to(dev)
    zk0 = Zk[s0 // nf]
    Zf = torch.where(interior.reshape(F, 1), 0.5 * (zk0 + Zk[slots[:, 1] // nf]), zk0).reshape(-1)

    def cg(b, x):  # Jacobi CG on the free rows (the blocks are symmetric), restarted from the true residual
        bn = b.norm()
        for _ in range(3):
            res = (b - A(x)) * free
            if float(res.norm()) <= 1e-15 * float(bn):
                break
            z = res / diag
            q, rz = z.clone(), res @ z
            for it in range(4000):
                v = A(q) * free
                al = rz / (q @ v)
                x = x + al * q
                res = res - al * v
                if it % 20 == 19 and float(res.norm()) <= 1e-15 * float(bn):
                    break
                z = res / diag
                rz, old = res @ z, rz
                q = z + (rz / old) * q
        return x

    for k in range(case["steps"]):
        R = meas.reshape(-1, 1) / tau * torch.einsum("kij,kj->ki", Nc, Zk)
        src = None if fb is None else fb.T
        if p.source:
            src = src + p.source[0] * math.sin(2 * math.pi * (k * tau) / p.source[1]) * psi.T
        if src is not None:
            R = R + meas.reshape(-1, 1) * src
        bc = torch.zeros(C, nf, n, dtype=torch.float64, device=dev)
        if a is not None:
            # upwind values on a face, by the sign of its first cell's flux
            af = a.permute(3, 2, 0, 1).reshape(C * nf, n, n)  # [slot, i, j]
            a0 = af[s0]
            zf = Zf.reshape(F, n)
            up = torch.where(interior.reshape(F, 1), Zk[slots[:, 1] // nf], zf)
            Zu = torch.where(a0 > 0, Zk[s0 // nf].unsqueeze(1), torch.where(a0 < 0, up.unsqueeze(1), torch.zeros_like(a0)))
            adv = (af.reshape(C, nf, n, n) * Zu[cf]).sum(dim=3)  # [K, e, i]
            R = R - adv.sum(dim=1)
            # zero total flux through the walls: their rows carry the advective flux
            wall = ((~interior).reshape(F, 1) & (tags == 1) & ~outflow).to(torch.float64)
            bc = adv * wall[cf]
        QR = torch.einsum("kij,kj->ki", Qi, R)
        rhs = gather(be.unsqueeze(2) * torch.einsum("kij,kj->ki", D, QR).unsqueeze(1) + bc)
        b = (rhs - A(xd)) * free
        Zf = cg(b, Zf * free) + xd
        zl = Zf[rows].reshape(C, nf, n)
        Zk = QR + torch.einsum("kij,kj->ki", Qi @ D, (be.unsqueeze(2) * zl).sum(dim=1))
    out = {"Z_iF": Zf, "Z_iK": Zk.T.contiguous().reshape(-1)}
    if case["form"] == "learned":
        out["params"] = None
    return out
