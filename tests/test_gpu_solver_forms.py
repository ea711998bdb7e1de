"""Every form of the linear solve at the ELL widths it is compiled for and at the run-time width,
against the oracle: the FP64 solve with the ELL words streamed and x in memory, the FP32 inner solve
of the mixed form, the five-kernel iterations above both (with rows that are a multiple of four and
not) and the two-kernel GMRES.  test_resident_plan.py holds the form that each of these sizes takes.

The bar is the parity tests': both sides solve to 1e-13, the states agree within 1e-10.
"""
import numpy as np
import pytest

from helpers import diffusion3d_n2, rel_err, variant
from mhfem import _lib as L
from mhfem import problems
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu


def box_n2(N):
    """Two components on cuboids (ELL width 21): coupled diffusion and reaction."""
    p = problems.diffusion3d_box(N=N, steps=1)
    C = p.C
    Nc = np.zeros((2, 2, C)); Nc[0, 0] = 1.0; Nc[1, 1] = 2.0
    D = np.zeros((2, 2, C)); D[0, 0] = p.coeffs["D"]; D[1, 1] = 0.5 * p.coeffs["D"]; D[0, 1] = 0.1
    r = np.zeros((2, 2, C)); r[0, 0] = 0.3; r[0, 1] = r[1, 0] = -0.1; r[1, 1] = 0.2
    base_bc = p.bc_fn

    def bc2(fv, fc):
        t, v, d = base_bc(fv, fc)
        return np.concatenate([t, t]), np.concatenate([v, v + 0.1 * (t == 1)]), np.concatenate([d + 0.2, d])

    q = variant(p, n_eq=2, coeffs={"N": Nc.ravel(), "D": D.ravel(), "r": r.ravel(), "f": 0.5})
    q.bc_fn = bc2
    q.Z0 = np.random.default_rng(17).uniform(0, 1, 2 * C)
    return q


def _check(name, N, rows, form=L.FORM_FP64, **opts):
    make = {"diffusion3d_n2": diffusion3d_n2, "box_n2": box_n2}.get(name) or (
        lambda N: problems.WORKLOADS[name](N=N, steps=1))
    p = make(N)
    p.tol = 1e-13
    p.config.form = form
    s = problems.make_solver(p)
    assert s.F * p.n == rows
    s.setup(tol=1e-13, max_iter=20000, **opts)
    st = s.step(0.0, p.dt)
    assert st["residual"] < 1e-13
    m = OracleModel.from_problem(p)
    m.step(0.0, p.dt, 1e-13)
    zf, zk = s.state()
    s.close()
    assert rel_err(zf, m.Z_iF) < 1e-10
    assert rel_err(zk, m.Z_iK) < 1e-10


@pytest.mark.parametrize("name,N,rows", [
    ("heat2d", 475, 677_825),          # x in memory, its update in the waiting warps
    ("diffusion3d", 40, 777_600),      # x in memory
    ("adr2d", 338, 686_816),
    ("adr2d", 350, 736_400),           # five kernels, width 9
    ("diffusion3d_box", 60, 658_800),  # width 10
    ("diffusion3d_n2", 28, 536_256),   # width 13
    ("box_n2", 37, 312_132),           # the run-time width (21)
])
def test_fp64(name, N, rows):
    _check(name, N, rows)


@pytest.mark.parametrize("name,N,rows", [
    ("heat2d", 430, 555_560),          # streamed, x in shared memory
    ("heat2d", 680, 1_388_560),        # x in memory, its update in the waiting warps
    ("heat2d", 736, 1_626_560),        # five kernels, four rows per thread, 24-bit columns
    ("heat2d", 741, 1_648_725),        # an odd number of rows
    ("adr2d", 200, 240_800),           # width 9: the ELL words in shared memory, streamed, five kernels
    ("adr2d", 240, 346_560),
    ("adr2d", 420, 1_060_080),
    ("diffusion3d_box", 42, 227_556),  # width 10
    ("diffusion3d_box", 50, 382_500),
    ("diffusion3d_box", 68, 957_168),
    ("diffusion3d_n2", 18, 143_856),   # width 13
    ("diffusion3d_n2", 22, 261_360),
    ("diffusion3d_n2", 31, 726_516),
    ("box_n2", 43, 488_136),           # the run-time width
])
def test_mixed(name, N, rows):
    _check(name, N, rows, L.FORM_MIXED)


@pytest.mark.parametrize("variant", ["cgs", "cgsr"])
@pytest.mark.parametrize("name,N,rows", [
    ("heat2d", 515, 796_705),
    ("adr2d", 360, 779_040),
    ("diffusion3d_n2", 31, 726_516),
    ("box_n2", 42, 455_112),
])
def test_gmres_of_two_kernels(name, N, rows, variant):
    _check(name, N, rows, linear_solver="gmres", gmres_restart=30, gmres_variant=variant)
