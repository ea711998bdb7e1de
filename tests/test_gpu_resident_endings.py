"""How a resident BiCGStab solve ends or restarts when a scalar of the iteration vanishes, in every
form it runs in: systems of equal small blocks of dyadic numbers, as many as a power of two, through
mhfem_bicgstab_noalloc.  Every sum, quotient and update below is exact in FP64, so each branch is
taken for certain.
"""
import ctypes as ct

import numpy as np
import pytest

from mhfem import _lib as L

pytestmark = pytest.mark.gpu

# (rows, ELL width): the form that the plan gives them
FORMS = [
    (64, 4),        # one CTA
    (2048, 6),      # a cluster
    (16384, 4),     # the grid, two reductions
    (131072, 4),    # three reductions, phase B forms the neighbours' s
    (131072, 9),    # three reductions, s published
    (262144, 10),   # the ELL words streamed
    (262144, 13),
]


def solve_blocks(block, b, rows, width, tol=1e-12, max_iter=100):
    """A x = b from x = 0, A = rows / len(b) copies of `block` (unit diagonal) on the diagonal."""
    import torch

    lib = L.load()
    block = np.asarray(block, np.float64)
    n = block.shape[0]
    assert rows % n == 0 and np.all(np.diag(block) == 1) and width >= n - 1
    r = np.arange(rows)
    cols = np.tile(r.astype(np.int32), (width, 1))  # padding: the own row, value 0
    vals = np.zeros((width, rows))
    for i in range(n):
        for k, j in enumerate(j for j in range(n) if j != i):
            cols[k, i::n] = r[i::n] - i + j
            vals[k, i::n] = block[i, j]
    dev = [torch.from_numpy(a).cuda() for a in (cols, vals, np.tile(np.asarray(b, np.float64), rows // n))]
    x = torch.zeros(rows, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    it, res = ct.c_int32(), ct.c_double()
    st = lib.mhfem_bicgstab_noalloc(dev[0].data_ptr(), dev[1].data_ptr(), width, rows, dev[2].data_ptr(),
                                    x.data_ptr(), tol, max_iter, 60.0, ct.byref(it), ct.byref(res), None)
    return st, it.value, res.value, x.cpu().numpy().reshape(-1, n)


@pytest.mark.parametrize("rows,width", FORMS)
def test_residual_that_vanishes(rows, width):
    """One unknown of a pair depends on the other: alpha = 1, s = (-a, 0) is not zero, omega = 1 and
    r = 0 after the first iteration, with (rh, r) = 0 and nothing left to restart from."""
    st, it, res, x = solve_blocks([[1.0, -0.5], [0.0, 1.0]], [0.0, 1.0], rows, width)
    assert st == L.OK and it == 1 and res == 0
    assert np.array_equal(x, np.tile([0.5, 1.0], (rows // 2, 1)))


@pytest.mark.parametrize("rows,width", FORMS)
def test_right_hand_side_near_the_smallest_numbers(rows, width):
    """The same system with (rh, v) = 2^-1026: its reciprocal is beyond the largest number, the
    quotient rho / (rh, v) = 1 is not."""
    n = rows // 2
    w = 2.0 ** ((-1026 - int(np.log2(n))) // 2)
    scale = n * w * w
    assert scale in (2.0**-1026, 2.0**-1027)
    st, it, res, x = solve_blocks([[1.0, -0.5], [0.0, 1.0]], [0.0, w], rows, width)
    assert st == L.OK and it == 1 and res == 0
    assert np.array_equal(x, np.tile([0.5 * w, w], (n, 1)))


@pytest.mark.parametrize("rows,width", FORMS)
def test_half_step_that_does_not_solve(rows, width):
    """A singular system: alpha = 1/2, s = (-6, 3) and A s = 0.  There is no omega, and ||s|| is three
    quarters of ||b||: a breakdown, not a solution."""
    st, it, res, x = solve_blocks([[1.0, 2.0], [0.5, 1.0]], [4.0, 8.0], rows, width)
    assert st == L.ERR_BREAKDOWN


@pytest.mark.parametrize("rows,width", FORMS)
def test_half_step_that_solves(rows, width):
    """The identity: alpha = 1 and s = 0, so the first half step solves the system."""
    st, it, res, x = solve_blocks([[1.0, 0.0], [0.0, 1.0]], [1.0, -1.0], rows, width)
    assert st == L.OK and it == 1 and res == 0
    assert np.array_equal(x, np.tile([1.0, -1.0], (rows // 2, 1)))


@pytest.mark.parametrize("rows,width", FORMS)
def test_breakdown(rows, width):
    """(rh, A rh) = 0 in the first iteration: no alpha."""
    st, it, res, x = solve_blocks([[1.0, -3.0], [1.0, 1.0]], [1.0, 1.0], rows, width)
    assert st == L.ERR_BREAKDOWN and it == 0 and res == 1
    assert not x.any()


# rows of three times a power of two, the forms as above
@pytest.mark.parametrize("rows,width", [(48, 4), (1536, 6), (12288, 4), (196608, 4), (196608, 6), (196608, 13)])
def test_restart(rows, width):
    """The columns of the block sum to 2, so (rh, A s) = 2 (rh, s) = 0 and rho' = 0 after the first
    iteration (alpha = 1/2, omega = 5, r = (2, -1, -1) / 16): rh = p = r, and the solve goes on.  It
    could not without the restart: rho = 0 ends it."""
    block = np.array([[1.0, 0.5, 0.25], [1.0, 1.0, 0.75], [0.0, 0.5, 1.0]])
    st, it, res, x = solve_blocks(block, [1.0, 1.0, 1.0], rows, width)
    assert st == L.OK and 2 <= it <= 8 and res < 1e-12
    # the block's condition number is below 100
    assert np.abs(x - np.linalg.solve(block, np.ones(3))).max() < 1e-9
