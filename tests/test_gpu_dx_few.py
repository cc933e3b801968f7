"""dX of convolutions on few channels, or a channel count that is no multiple of four (csrc/snntc_dx_few.cu), against the float64
oracle and the register-tile kernel: every register width, strides, windows larger than the stride and smaller, fields that drop
trailing rows, fan-out below, at and above a warp."""
import numpy as np
import pytest

import oracle as O
from tests import parity as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,C,Kh,Kw,Sh,Sw,Kc,padding", [
    (1, 5, 7, 1, 1, 1, 1, 1, 1, "SAME"), (2, 9, 8, 1, 5, 5, 2, 2, 40, "SAME"), (3, 12, 11, 3, 7, 7, 2, 2, 64, "SAME"),
    (2, 10, 13, 4, 3, 3, 1, 1, 33, "VALID"), (1, 11, 10, 5, 2, 3, 3, 1, 31, "VALID"), (2, 8, 9, 9, 3, 3, 2, 1, 100, "SAME"),
    (1, 9, 9, 15, 5, 3, 1, 2, 8, "SAME"), (2, 6, 6, 17, 5, 5, 1, 1, 128, "SAME"), (1, 8, 8, 18, 3, 3, 1, 1, 24, "SAME"), (2, 7, 7, 37, 3, 3, 2, 2, 36, "VALID")])
def test_conv_dx_with_lanes_over_the_outputs(B, H, W, C, Kh, Kw, Sh, Sw, Kc, padding):
    import torch
    from snntc_2023_b200 import _lib, ops
    x, w = P.make_inputs(B * H + C, (B, H, W, C), (Kh * Kw * C + 1, Kc), "ref", bias=True)
    params = O.cv_params(Kh, Kw, Sh, Sw, padding, 1.0)
    pt, pl, Nh, Nw = ops.conv_geometry(H, W, Kh, Kw, Sh, Sw, padding)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    out = ops.snn_cv(xd, wd, params, pt, pl, Nh, Nw)
    g = np.random.default_rng(C).standard_normal((B, Nh, Nw, Kc)).astype(np.float32)
    gd = torch.from_numpy(g).cuda()
    oc = out.cpu().numpy()
    ref = O.cv_backward(g, x, w, params, oc[:B], oc[B:], "f64")
    for kernel in (3, 1, 0):
        dx, dw, _ = ops.snn_cv_grad(gd, xd, wd, params, out, pt, pl, opts=_lib.options(dx_kernel=kernel))
        P.check_close(dx.cpu().numpy(), ref["dx"], "dX kernel %d" % kernel, abs_sum=ref["dx_abs"])
        P.check_close(dw.cpu().numpy(), ref["dw"], "dW beside it", abs_sum=ref["dw_abs"])
