"""The training decoder's weight gradient on a mesh of several passes over the grid (777,600 faces),
against 64 bits.

With zero weights above the encoder's bias every face has the same hidden values c (BF16 numbers
between 1 and 2) and output 0, and with one target value every training face the same dout, so that
the exact gradient is c times the sum of dout.

Tolerance: a run of four FP32 products and sums is off by at most (1 + 1 + 2 + 3 + 4) / 4 units of
2^-24, the three levels of pair sums and the result's own rounding by one each; the sums behind are
FP64."""
import numpy as np
import pytest

from mhfem import _lib as L
from mhfem import problems
from oracle import mpnn_oracle as mo
from test_gpu_learned import flatten, unflatten

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("target", [-0.5, -0.15, -0.35])
def test_decoder_weight_gradient_sums(target):
    p = problems.diffusion3d(N=40, steps=1, form=L.FORM_LEARNED)
    s = problems.make_solver(p)
    fv, fc, _ = s.topology()
    tags, _, _ = p.bc_fn(fv, fc)
    fixed = (fc[:, 1] < 0) & (tags == 0)
    assert s.F == 777_600
    params = {k: np.zeros_like(v) for k, v in mo.init_params(0).items()}
    c = (129 + 2 * np.arange(mo.H)) / 128.0  # 129/128 .. 255/128
    params["b0"] = c
    s.set_learned_params(flatten(params))
    loss, g = s.learned_gradients(np.zeros((s.F, 16), np.float32), np.full(s.F, target))
    s.close()
    gg = unflatten(g)
    n = int((~fixed).sum())
    dout = float(np.float32(2.0 * -target / n))
    assert abs(loss - target**2) <= 1e-12 * target**2
    err = np.abs(gg["wd"] / (c * dout * n) - 1.0)
    assert err.max() <= (11 / 4 + 4) * 2.0**-24
    assert abs(gg["bd"][0] / (dout * n) - 1.0) <= 2.0**-24
