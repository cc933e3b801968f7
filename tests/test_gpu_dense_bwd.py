"""Both gradients of a dense layer by the warp-tile kernel (csrc/snntc_bwd_dense.cu) against the register-tile kernels it takes
over from: the same sums in the same order, hence the same bits. Sizes around the edges of its tiles (32, 16, 8), chunks (16)
and row slices (64 and more), fan-in and fan-out that 16-byte copies cannot take, and values outside the range of the
scaled dW loop."""
import numpy as np
import pytest

import oracle as O
from tests import parity as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,I,J,bv", [(1, 1, 1, 1.0), (1, 33, 10, 0.0), (7, 64, 16, 1.0), (32, 784, 400, 1.0), (33, 257, 130, 0.0),
                                      (64, 31, 17, 1.0), (65, 300, 44, 1.0), (129, 100, 260, 0.0), (640, 36, 10, 1.0),
                                      (1000, 500, 77, 1.0), (2047, 40, 12, 1.0), (2048, 96, 100, 1.0)])
@pytest.mark.parametrize("odd", [False, True])
def test_dense_backward_matches_the_register_tiles_bit_for_bit(B, I, J, bv, odd):
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(B + 7 * I + J)
    x, w = P.make_inputs(B + I + J, (B, I), (I + (bv > 0), J), "ref", bias=bv > 0)
    if odd:   # an input below 2^-60 sends every dW kernel through its unscaled loop
        x[rng.integers(B), rng.integers(I)] = 1e-30
    params = O.fc_params(biasvolt=bv)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    out = ops.snn_fc(xd, wd, params)
    g = rng.standard_normal((B, J)).astype(np.float32)
    g[rng.random(g.shape) < 0.4] = 0
    gd = torch.from_numpy(g).cuda()
    dx, dw, _ = ops.snn_fc_grad(gd, xd, wd, params, out)
    dx1, dw1, _ = ops.snn_fc_grad(gd, xd, wd, params, out, opts=_lib.options(dx_kernel=1, dw_kernel=1))
    assert torch.equal(dx, dx1) and torch.equal(dw, dw1)
    _, only, _ = ops.snn_fc_grad(gd, xd, wd, params, out, need_input_grad=False)
    assert torch.equal(only, dw)
    outc = out.cpu().numpy()
    ref = O.fc_backward(g, x, w, params, outc[:B], outc[B:], "f64")
    P.check_close(dx.cpu().numpy(), ref["dx"], "dense dX", abs_sum=ref["dx_abs"])
    P.check_close(dw.cpu().numpy(), ref["dw"], "dense dW", abs_sum=ref["dw_abs"])
