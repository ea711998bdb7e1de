"""A resident solve that takes more iterations than one launch runs (256) goes on from the state the
launch left, in every form: each case asserts that it does take more."""
import ctypes as ct

import numpy as np
import pytest

from helpers import rel_err
from mhfem import _lib as L
from mhfem import problems
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu

CHUNK = 256


@pytest.mark.parametrize("rows,width", [
    (100, 4),        # one CTA
    (4096, 6),       # a cluster
    (12287, 4),      # the grid, two reductions
    (131072, 4),     # three reductions, phase B forms the neighbours' s
    (131072, 9),     # three reductions, s published
    (262144, 10),    # the ELL words streamed
])
def test_bicgstab(rows, width):
    """A chain with unit diagonal and neighbours -(0.5 - 1e-4), against the direct solution.  The
    eigenvalues lie in [2e-4, 2], so a residual of 1e-12 leaves a relative error of 1e-8 at most; the
    bound is twice that.  (A chain of 100 takes fewer iterations than unknowns.)"""
    import torch
    from scipy.linalg import solve_banded

    off = -(0.5 - 1e-4)
    r = np.arange(rows)
    cols = np.tile(r.astype(np.int32), (width, 1))
    vals = np.zeros((width, rows))
    cols[0, 1:], vals[0, 1:] = r[:-1], off
    cols[1, :-1], vals[1, :-1] = r[1:], off
    b = np.random.default_rng(rows).standard_normal(rows)
    dev = [torch.from_numpy(a).cuda() for a in (cols, vals, b)]
    x = torch.zeros(rows, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    it, res = ct.c_int32(), ct.c_double()
    st = L.load().mhfem_bicgstab_noalloc(dev[0].data_ptr(), dev[1].data_ptr(), width, rows, dev[2].data_ptr(),
                                         x.data_ptr(), 1e-12, 20000, 60.0, ct.byref(it), ct.byref(res), None)
    assert st == L.OK and res.value < 1e-12
    if rows > 100:
        assert it.value > CHUNK
    ref = solve_banded((1, 1), np.array([np.full(rows, off), np.ones(rows), np.full(rows, off)]), b)
    assert np.linalg.norm(x.cpu().numpy() - ref) < 2e-8 * np.linalg.norm(ref)


def _step(name, N, factor, form=L.FORM_FP64, **opts):
    """A time step `factor` times as long.  Two solutions with residuals of 1e-13 differ by at most
    2e-13 times the condition number, which is below 24 N^2 dt (heat) and 5e4 (diffusion) here."""
    p = problems.WORKLOADS[name](N=N, steps=1)
    p.dt *= factor
    p.config.form = form
    s = problems.make_solver(p)
    s.setup(tol=1e-13, max_iter=20000, **opts)
    st = s.step(0.0, p.dt)
    m = OracleModel.from_problem(p)
    m.step(0.0, p.dt, 1e-13)
    assert rel_err(s.state()[0], m.Z_iF) < 1e-8
    s.close()
    return st


@pytest.mark.parametrize("N,factor", [(205, 20), (290, 20), (345, 10), (475, 5)])
def test_time_step(N, factor):
    """The three-reduction forms, the streamed one and x in memory."""
    assert _step("heat2d", N, factor)["iterations"] > CHUNK


@pytest.mark.parametrize("N,factor", [(26, 100), (30, 10), (36, 10), (50, 4)])
def test_mixed_inner_solve(N, factor):
    """Two reductions, three, streamed, x in memory: all sweeps to the same inner tolerance, so that
    the mean of the sweeps' counts above 256 means that one of them is."""
    st = _step("diffusion3d", N, factor, L.FORM_MIXED, inner_tol=1e-6, inner_adaptive=False)
    assert st["iterations"] > CHUNK * st["sweeps"]


@pytest.mark.parametrize("variant", ["cgs", "cgsr"])
@pytest.mark.parametrize("N,factor", [(36, 100), (100, 20), (200, 20)])
def test_gmres(N, factor, variant):
    """A cluster, the basis in shared memory, the basis in memory."""
    assert _step("heat2d", N, factor, linear_solver="gmres", gmres_variant=variant)["iterations"] > CHUNK
