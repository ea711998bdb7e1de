"""mhfem_bicgstab_noalloc keeps its promise at every width: the solve tests its convergence in every
iteration.  One system of the largest size, its ELL words padded to wider and wider ones (value 0 on
the own row): the padding takes the solve from the form with the words in shared memory (width 4) to
the streamed one, at 25 and 40 beyond the matrix size up to which larger systems run resident, and
changes neither the products nor the order of any sum."""
import ctypes as ct

import numpy as np
import pytest

from mhfem import _lib as L

pytestmark = pytest.mark.gpu

ROWS = L.NOALLOC_MAX_ROWS


def _solve(width, tol):
    import torch

    lib = L.load()
    r = np.arange(ROWS, dtype=np.int64)
    cols = np.tile(r.astype(np.int32), (width, 1))
    vals = np.zeros((width, ROWS))
    rng = np.random.default_rng(4)
    for k, d in enumerate((-512, -1, 1, 512)):
        cols[k] = (r + d) % ROWS
        vals[k] = rng.uniform(-0.24, -0.2, ROWS)
    b = rng.standard_normal(ROWS)
    dev = [torch.from_numpy(a).cuda() for a in (cols, vals, b)]
    x = torch.zeros(ROWS, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    it, res = ct.c_int32(), ct.c_double()
    st = lib.mhfem_bicgstab_noalloc(dev[0].data_ptr(), dev[1].data_ptr(), width, ROWS, dev[2].data_ptr(),
                                    x.data_ptr(), tol, 1000, 60.0, ct.byref(it), ct.byref(res), None)
    return st, it.value, res.value, x.cpu().numpy()


@pytest.mark.parametrize("width", [10, 13, 25, 40])
def test_convergence_is_tested_in_every_iteration(width):
    counts = set()
    for tol in (1e-2, 1e-3, 1e-4, 1e-6, 1e-8):
        st0, it0, res0, x0 = _solve(4, tol)
        st, it, res, x = _solve(width, tol)
        assert st0 == L.OK and st == L.OK
        assert it == it0 and res == pytest.approx(res0, rel=1e-6)
        assert np.abs(x - x0).max() <= 1e-12 * np.abs(x0).max()
        counts.add(it0 % 4)
    assert counts - {0}  # not only counts that a test in every fourth iteration gives too
