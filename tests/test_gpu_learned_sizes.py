"""Gradients of the learned warm start at face counts around the edges of the training kernels'
splits: the decoder takes 32 rows per block pass, the GEMM kernels 128 faces per tile, and the
partial sums of the tiles are added in slices of 8.  Compared with the CPU oracle, which rounds to
BF16 at the same points.

The loss, the decoder's gradients and the top layer's weight gradient, which the decoder and the
two reductions form directly: below the top layer a BF16 step of an activation can flip a ReLU,
which on a mesh of a few faces moves those layers' gradients by several percent.  Tolerance 2^-8
relative per tensor: one BF16 step in every value."""
import numpy as np
import pytest

from mhfem import _lib as L
from mhfem import problems
from oracle import mpnn_oracle as mo
from test_gpu_learned import flatten, graph_from_solver, unflatten

pytestmark = pytest.mark.gpu


# 18, 120, 378, 2808 and 4410 faces: less than one decoder pass, one tile not quite full, three
# tiles, 22 tiles (the slices of the reduction uneven), 35 tiles with a short last one
@pytest.mark.parametrize("N", [1, 2, 3, 6, 7])
def test_gradients_at_the_edges_of_the_splits(N):
    p = problems.diffusion3d(N=N, steps=1, form=L.FORM_LEARNED)
    s = problems.make_solver(p)
    nbr, deg = graph_from_solver(s)
    fv, fc, _ = s.topology()
    tags, _, _ = p.bc_fn(fv, fc)
    fixed = (fc[:, 1] < 0) & (tags == 0)
    assert s.F == 12 * N**3 + 6 * N**2
    rng = np.random.default_rng(100 + N)
    x = rng.standard_normal((s.F, 16)).astype(np.float32)
    y = rng.standard_normal(s.F)
    params = mo.init_params(5)
    for k in params:
        params[k] = params[k] + 0.05 * rng.standard_normal(params[k].shape)
    params = unflatten(flatten(params))
    s.set_learned_params(flatten(params))
    loss, g = s.learned_gradients(x, y)
    s.close()
    ref, gr, _ = mo.loss_and_grads(params, x.astype(np.float64), nbr, deg, y, (~fixed).astype(np.float64), bf=True)
    assert abs(loss - ref) < 2.0**-8 * ref
    gg = unflatten(g)
    top = f"W{mo.LAYERS}"
    for k in ("wd", "bd", top):
        err = np.linalg.norm(gg[k] - gr[k]) / max(np.linalg.norm(gr[k]), 1e-30)
        assert err < 2.0**-8, f"gradient {k}: relative error {err:.3e}"
