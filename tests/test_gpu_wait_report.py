"""A wait between the CTAs of a resident solve that gives up is reported,
whichever wait it was and whatever the first CTA wrote.

mhfem_check_wait_report makes one CTA give its waits up: it has
arrived, so the others pass that wait and fail the next one within a few
polls.  Nothing hangs: every wait is bounded, and a CTA that gave up returns.
"""
import pytest

from helpers import rel_err
from mhfem import _lib as L
from mhfem import problems
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu

# (model, N): grids of more than one CTA
SYSTEMS = [
    ("heat2d", 40),    # two reductions per iteration
    ("heat2d", 210),   # three, the ELL words in shared memory
    ("heat2d", 350),   # the ELL words streamed
]


def _solver(name, N, form=L.FORM_FP64, **opts):
    p = problems.WORKLOADS[name](N=N, steps=2)
    p.tol = 1e-13
    p.config.form = form
    s = problems.make_solver(p)
    if opts:
        s.setup(tol=p.tol, max_iter=20000, **opts)
    return p, s


@pytest.mark.parametrize("cta", [1, 3])
@pytest.mark.parametrize("name,N", SYSTEMS)
def test_last_wait_that_gives_up_is_reported(name, N, cta):
    """The traces solve the system already, so the solve ends at its first and
    only wait; the first CTA passes it and writes a converged result."""
    p, s = _solver(name, N)
    s.step(0.0, p.dt)
    s.setup(tol=1e-9, max_iter=20000)
    assert s.solveLinearSystem()["iterations"] == 0
    s.lib.mhfem_check_wait_report(s._h, cta)
    with pytest.raises(Exception, match="gave up"):
        s.solveLinearSystem()
    s.lib.mhfem_check_wait_report(s._h, -1)
    assert s.solveLinearSystem()["iterations"] == 0
    s.close()


@pytest.mark.parametrize("name,N,form,opts", [
    ("heat2d", 40, L.FORM_FP64, {}),
    ("heat2d", 210, L.FORM_FP64, {}),
    ("heat2d", 350, L.FORM_FP64, {}),
    ("heat2d", 100, L.FORM_MIXED, {}),
    ("heat2d", 420, L.FORM_MIXED, {}),
    ("heat2d", 100, L.FORM_FP64, {"linear_solver": "gmres"}),
    ("heat2d", 250, L.FORM_FP64, {"linear_solver": "gmres"}),
])
def test_solve_works_again_after_a_wait_gave_up(name, N, form, opts):
    p, s = _solver(name, N, form, **opts)
    s.lib.mhfem_check_wait_report(s._h, 2)
    with pytest.raises(Exception, match="gave up"):
        s.step(0.0, p.dt)
    s.lib.mhfem_check_wait_report(s._h, -1)
    s.setInitialCondition(p.Z0)
    m = OracleModel.from_problem(p)
    assert s.step(0.0, p.dt)["residual"] < 1e-13
    m.step(0.0, p.dt, 1e-13)
    assert rel_err(s.state()[0], m.Z_iF) < 1e-10
    s.close()
