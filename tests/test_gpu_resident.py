"""The FP64 BiCGStab resident on the SMs (csrc/resident.cuh, resident_two.cuh) at the edges of
its forms, against the oracle: one CTA, clusters of 2 to 16 with a partial
last block of rows, the largest cluster and the first grid, both sides of the
sizes where an iteration goes from two reductions to three and where phase B
stops forming the neighbours' s, the sizes where the ELL words and then x
leave shared memory, and the last resident system and the first one above it;
run-time and compile-time widths.

The bar is the parity tests': both sides solve to 1e-13, the states agree
within 1e-10.
"""
import numpy as np
import pytest

from helpers import diffusion3d_n2, rel_err
from mhfem import _lib as L
from mhfem import problems
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu

TOL_STATE = 1e-10

# (model, N): the row count in the comment
SIZES = [
    ("heat2d", 2),           # 16: one CTA
    ("heat2d", 6),           # 120
    ("heat2d", 7),           # 161: a cluster of 2
    ("heat2d", 17),          # 901: 8, the last block partial
    ("heat2d", 36),          # 3,960: the largest cluster
    ("heat2d", 37),          # 4,181: the smallest grid
    ("heat2d", 53),          # 8,533
    ("heat2d", 162),         # 79,056
    ("heat2d", 203),         # 124,033: two reductions per iteration
    ("heat2d", 205),         # 126,485: three, the neighbours' s recomputed
    ("heat2d", 288),         # 249,408
    ("heat2d", 290),         # 252,880: s published
    ("heat2d", 345),         # 357,765: ELL words streamed
    ("heat2d", 520),         # 812,240: x in memory, the largest resident system
    ("heat2d", 523),         # 821,633: five kernels
    ("diffusion3d", 3),      # width 6: 378
    ("diffusion3d", 7),      # 4,410
    ("diffusion3d", 13),     # 27,378
    ("diffusion3d", 19),     # 84,474
    ("diffusion3d", 29),     # 297,714: streamed
    ("diffusion3d_box", 9),  # width 10: 2,430
    ("diffusion3d_box", 24),  # 43,200
    ("diffusion3d_box", 36),  # 143,856
    ("diffusion3d_box", 50),  # 382,500: streamed
    ("adr2d", 15),           # width 9: 1,410
    ("adr2d", 60),           # 21,840
    ("adr2d", 120),          # 86,880
    ("adr2d", 240),          # 346,560: streamed
    ("diffusion3d_n2", 6),   # width 13: 5,616
    ("diffusion3d_n2", 20),  # 196,800
    ("box3d_lumped", 10),    # a lumped cuboid system
]


def _problem(name, N):
    if name == "diffusion3d_n2":
        p = diffusion3d_n2(N)
    elif name == "box3d_lumped":
        p = problems.diffusion3d_box(N=N, steps=2, lumping=True)
    else:
        p = problems.WORKLOADS[name](N=N, steps=2)
    p.tol = 1e-13
    return p


@pytest.mark.parametrize("name,N", SIZES)
def test_resident_solve_against_oracle(name, N):
    p = _problem(name, N)
    s = problems.make_solver(p)
    m = OracleModel.from_problem(p)
    t = 0.0
    for _ in range(1 if s.F * p.n > 100000 else 2):
        st = s.step(t, p.dt)
        m.step(t, p.dt, 1e-13)
        assert st["residual"] < 1e-13
        t += p.dt
    zf, zk = s.state()
    assert rel_err(zf, m.Z_iF) < TOL_STATE
    assert rel_err(zk, m.Z_iK) < TOL_STATE
    s.close()


@pytest.mark.parametrize("name,N", [("heat2d", 30), ("heat2d", 40), ("heat2d", 100), ("diffusion3d", 29)])
def test_resident_solve_continues_after_a_chunk(name, N):
    """A time step 400 times as long takes more iterations than one launch
    runs (256): the solve goes on from the state the launch left, in the
    cluster, the grid and the streamed form."""
    p = _problem(name, N)
    p.dt *= 400.0
    s = problems.make_solver(p)
    m = OracleModel.from_problem(p)
    s.step(0.0, p.dt)
    m.step(0.0, p.dt, 1e-13)
    # two solutions with residuals of 1e-13 differ by at most 2e-13 times the
    # condition number, which is below 24 N^2 dt (heat) and 5e4 here
    assert rel_err(s.state()[0], m.Z_iF) < 1e-8
    s.close()


@pytest.mark.parametrize("name,N", [
    ("heat2d", 6),            # one CTA
    ("heat2d", 36),           # the largest cluster
    ("heat2d", 37),           # the smallest grid
    ("heat2d", 200),          # 120,400: two reductions per iteration
    ("heat2d", 391),          # 459,425: the ELL words still in shared memory
    ("heat2d", 405),          # 492,885: streamed
    ("diffusion3d", 13),
    ("diffusion3d", 33),      # 437,778: streamed
    ("diffusion3d", 50),      # 1,515,000: x in shared memory, the largest width-6 system below
    ("diffusion3d", 52),      # 1,703,520: five kernels
    ("diffusion3d_box", 30),  # width 10
    ("adr2d", 30),            # width 9
])
def test_resident_inner_solve_against_oracle(name, N):
    """The mixed form, whose FP32 inner solve runs resident."""
    p = _problem(name, N)
    p.config.form = L.FORM_MIXED
    s = problems.make_solver(p)
    m = OracleModel.from_problem(p)
    st = s.step(0.0, p.dt)
    m.step(0.0, p.dt, 1e-13)
    assert st["residual"] < 1e-13 and st["sweeps"] > 1
    zf, zk = s.state()
    assert rel_err(zf, m.Z_iF) < TOL_STATE
    assert rel_err(zk, m.Z_iK) < TOL_STATE
    s.close()


@pytest.mark.parametrize("variant", ["cgs", "cgsr"])
@pytest.mark.parametrize("name,N", [
    ("heat2d", 2),             # one CTA, the Krylov space as large as the system
    ("heat2d", 17),            # a cluster, the last block partial
    ("heat2d", 36),            # the largest cluster
    ("heat2d", 37),            # the smallest grid
    ("heat2d", 150),           # 67,800: the basis in shared memory
    ("heat2d", 200),           # 120,400: the basis in memory
    ("heat2d", 300),           # 270,600
    ("diffusion3d", 6),        # width 6
    ("adr2d", 40),             # width 9
    ("diffusion3d_box", 12),   # width 10
    ("diffusion3d_n2", 5),     # width 13
])
def test_resident_gmres_against_oracle(name, N, variant):
    p = _problem(name, N)
    s = problems.make_solver(p)
    s.setup(tol=1e-13, max_iter=20000, linear_solver="gmres", gmres_restart=30, gmres_variant=variant,
            gmres_restart_min=3, gmres_restart_step_min=2, gmres_restart_step_max=4)
    m = OracleModel.from_problem(p)
    st = s.step(0.0, p.dt)
    m.step(0.0, p.dt, 1e-13)
    assert st["residual"] < 1e-13
    zf, zk = s.state()
    assert rel_err(zf, m.Z_iF) < TOL_STATE
    assert rel_err(zk, m.Z_iK) < TOL_STATE
    s.close()


def test_resident_solve_iteration_cap():
    p = _problem("heat2d", 64)
    s = problems.make_solver(p, max_iter=7)
    with pytest.raises(Exception, match="7 iterations"):
        s.step(0.0, p.dt)
    s.setup(tol=1e-12, max_iter=1000)
    s.setInitialCondition(p.Z0)
    assert s.step(0.0, p.dt)["residual"] < 1e-12
    assert np.isfinite(s.state()[0]).all()
    s.close()


@pytest.mark.parametrize("form,solver", [(L.FORM_FP64, "bicgstab"), (L.FORM_FP64, "gmres"), (L.FORM_MIXED, "bicgstab")])
@pytest.mark.parametrize("N", [8, 64])
def test_failed_assembly_leaves_the_state(form, solver, N):
    """A non-positive diagonal is found by the solve's first kernel: the error
    is reported, the traces stay as they were, and the next step works."""
    p = _problem("heat2d", N)
    p.config.form = form
    s = problems.make_solver(p)
    s.setup(tol=1e-13, max_iter=20000, linear_solver=solver)
    before = s.state()[0]
    s.set_coeff("D", -1e-3)
    with pytest.raises(Exception, match="not positive"):
        s.step(0.0, p.dt)
    assert np.array_equal(s.state()[0], before)
    s.set_coeff("D", 1.0)
    m = OracleModel.from_problem(p)
    s.step(0.0, p.dt)
    m.step(0.0, p.dt, 1e-13)
    assert rel_err(s.state()[0], m.Z_iF) < TOL_STATE
    s.close()
