"""GPU: the training GEMM at tile remainders and unaligned strides, against
the float64 network oracle (the bars of test_gpu_learn: outputs 3e-3,
gradients 1e-2, loss 1e-3 relative)."""
import numpy as np
import pytest

from oracle import mlp_oracle as M
from test_gpu_learn import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("din,hidden,dout,rows", [(1, 16, 1, 1), (37, 16, 35, 77), (33, 48, 65, 31), (32, 64, 64, 32),
                                                  (129, 80, 63, 257)])
def test_gemm_remainders(din, hidden, dout, rows):
    from letkf_gb300 import mlp_debug, mlp_param_shapes
    rng = np.random.default_rng(7 * din + rows)
    shapes = mlp_param_shapes(din, hidden, dout)
    p = np.concatenate([rng.uniform(-1, 1, size=s).ravel() * (np.sqrt(6.0 / sum(s)) if len(s) == 2 else 0.1)
                        for s in shapes]).astype(np.float32)
    x = rng.standard_normal((rows, din)).astype(np.float32)
    t = rng.standard_normal((rows, dout)).astype(np.float32)
    g = mlp_debug(p, x, t, hidden=hidden)
    loss, grad, y = M.loss_grad(p, x, t, hidden, dout)
    assert rel(g["y_simt"], y) <= 3e-3
    assert abs(g["loss"] - loss) <= 1e-3 * loss
    o = 0
    for s in shapes:
        n = int(np.prod(s))
        assert rel(g["grad"][o:o + n], grad[o:o + n]) <= 1e-2, s
        o += n
