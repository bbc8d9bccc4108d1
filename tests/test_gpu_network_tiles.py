"""The network's tensor-core kernels where their tiling can go wrong: one tile
in all, rows at both image edges, two tiles per row, fewer tiles than CTAs, and
several tiles per CTA with a remainder (the ring of stages wraps, the
accumulators run over tiles).  The oracle rounds to bfloat16 where the kernels
do and sums in float64; the bars are those of test_nn.py (another order of the
sums can move a value across a bfloat16 rounding)."""
import numpy as np
import pytest
from conftest import rel_l2

pytestmark = pytest.mark.gpu


# 1; 2; 42; 297 (one more than two CTAs per SM); 645 (3 tiles in some CTAs, 2 in others)
@pytest.mark.parametrize("shape", [(1, 1, 128), (1, 1, 256), (3, 7, 256), (3, 99, 128),
                                   (5, 129, 128)])
def test_forward_and_gradient(shape):
    import nn_oracle as N
    import qpgpu

    nb, h, w = shape
    rng = np.random.default_rng(11)
    p = []
    for ci, co in zip(N.CIN, N.COUT):
        p += [rng.normal(0, np.sqrt(2.0 / (9 * ci)), 9 * ci * co), rng.normal(0, 0.05, co)]
    p = np.concatenate(p).astype(np.float32)
    x = rng.normal(0, 1, (nb, 16, h, w)).astype(np.float32)
    t = rng.normal(0, 1, (nb, 2, h, w)).astype(np.float32)
    net = qpgpu.Predictor(seed=1)
    net.set_params(p)
    for _ in range(2):  # the second pass runs on the kept work buffers
        assert rel_l2(net.forward(x), N.forward(p, x)[0]) < 5e-3
        loss, g = net.loss_grad(x, t)
    eloss, eg = N.loss_grad(p, x, t)
    assert abs(loss - eloss) < 1e-3 * eloss
    o = 0
    for ci, co in zip(N.CIN, N.COUT):
        n = 9 * ci * co
        used = slice(None) if co == 32 else slice(0, 2)  # 2 of the last layer's outputs
        assert rel_l2(g[o:o + n].reshape(9, ci, co)[..., used],
                      eg[o:o + n].reshape(9, ci, co)[..., used]) < 3e-2
        assert rel_l2(g[o + n:o + n + co][used], eg[o + n:o + n + co][used]) < 3e-2
        o += n + co
    net.close()
