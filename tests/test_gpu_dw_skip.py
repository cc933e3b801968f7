"""dW of convolutions whose channels or outputs are no multiple of four (csrc/snntc_dw_skip.cu, single-column copies) against the
float64 oracle and the register-tile kernel: every compiled tile width, several tiles, remainders of columns, rows and outputs."""
import numpy as np
import pytest

import oracle as O
from tests import parity as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,C,Kh,Kw,Sh,Sw,Kc,padding,bias", [
    (1, 5, 7, 1, 1, 1, 1, 1, 1, "SAME", True), (3, 12, 11, 3, 7, 7, 2, 2, 33, "SAME", True),     # 1 and 148 rows (3 units)
    (2, 10, 13, 7, 3, 3, 1, 1, 30, "VALID", True), (2, 11, 10, 14, 4, 4, 3, 1, 31, "VALID", False),  # 64 (1), 224 (4)
    (2, 9, 8, 5, 5, 5, 2, 2, 40, "SAME", True), (1, 9, 9, 38, 3, 3, 1, 2, 65, "SAME", True),     # 126 (2), 343 (6)
    (1, 8, 8, 53, 3, 3, 1, 1, 24, "SAME", True), (2, 7, 7, 71, 3, 3, 2, 2, 36, "VALID", True),   # 478 (8), 640 (10)
    (1, 8, 9, 90, 3, 3, 1, 1, 6, "SAME", True), (2, 6, 6, 32, 3, 3, 1, 1, 27, "SAME", True)])    # two tiles; x aligned, J not
def test_conv_dw_with_single_column_copies(B, H, W, C, Kh, Kw, Sh, Sw, Kc, padding, bias):
    import torch
    from snntc_2023_b200 import _lib, ops
    x, w = P.make_inputs(B * H + C, (B, H, W, C), (Kh * Kw * C + bias, Kc), "ref", bias=bias)
    params = O.cv_params(Kh, Kw, Sh, Sw, padding, 1.0 if bias else -1.0)
    pt, pl, Nh, Nw = ops.conv_geometry(H, W, Kh, Kw, Sh, Sw, padding)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    out = ops.snn_cv(xd, wd, params, pt, pl, Nh, Nw)
    rng = np.random.default_rng(C)
    g = (rng.standard_normal((B, Nh, Nw, Kc)) * (rng.random((B, Nh, Nw, Kc)) < 0.5)).astype(np.float32)
    gd = torch.from_numpy(g).cuda()
    oc = out.cpu().numpy()
    ref = O.cv_backward(g, x, w, params, oc[:B], oc[B:], "f64")
    for kernel in (2, 1, 0):
        _, dw, _ = ops.snn_cv_grad(gd, xd, wd, params, out, pt, pl, opts=_lib.options(dw_kernel=kernel))
        P.check_close(dw.cpu().numpy(), ref["dw"], "dW kernel %d" % kernel, abs_sum=ref["dw_abs"])


@pytest.mark.parametrize("C,J,k", [(64, 64, 3), (32, 96, 3), (128, 52, 3), (16, 128, 1), (256, 40, 2), (8, 36, 5)])
@pytest.mark.parametrize("pattern", ["hot", "late", "none", "all"])
def test_channels_dealt_out_by_activity(C, J, k, pattern):
    """dW through tensor maps with output channels that differ in how often they carry a gradient: a few always and the rest never, only
    in images that the first stages do not see, none at all, all: against the register tile."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(C + J + k)
    B, H, W = 5, 19, 17
    x, w = P.make_inputs(C + J + k, (B, H, W, C), (k * k * C + 1, J), "ref", bias=True)
    params = O.cv_params(k, k, 1, 1, "SAME")
    pt, pl, Nh, Nw = ops.conv_geometry(H, W, k, k, 1, 1, "SAME")
    gr = rng.standard_normal((B, Nh, Nw, J)).astype(np.float32)
    if pattern == "hot":
        gr[..., rng.permutation(J)[J // 8:]] = 0
    elif pattern == "late":
        gr[:3] = 0
        gr[..., ::3] = 0
    elif pattern == "none":
        gr[:] = 0
    xd, wd, gd = (torch.from_numpy(a).cuda() for a in (x, w, gr))
    out = ops.snn_cv(xd, wd, params, pt, pl, Nh, Nw)
    _, dw1, _ = ops.snn_cv_grad(gd, xd, wd, params, out, pt, pl, opts=_lib.options(dw_kernel=1))
    _, dw4, _ = ops.snn_cv_grad(gd, xd, wd, params, out, pt, pl, opts=_lib.options(dw_kernel=4))
    assert float((dw4 - dw1).norm()) <= 1e-5 * float(dw1.norm())     # sums of 32-bit floats in another order
    _, dw5, _ = ops.snn_cv_grad(gd, xd, wd, params, out, pt, pl, opts=_lib.options(dw_kernel=4))
    assert torch.equal(dw4, dw5)
    assert _lib.load_measure().snntc_copy_timeouts() == 0


@pytest.mark.parametrize("C,J,k,stride", [(64, 64, 3, 1), (32, 96, 3, 2), (20, 52, 5, 2), (128, 40, 3, 1), (16, 24, 3, 2),   # 16-byte copies
                                          (19, 64, 3, 1), (3, 33, 7, 2), (53, 70, 3, 2), (7, 30, 5, 1), (90, 9, 3, 1)])       # single columns
@pytest.mark.parametrize("pattern", ["hot", "late", "none", "all"])
def test_channels_dealt_out_by_activity_with_copies_per_thread(C, J, k, stride, pattern):
    """The same patterns in the row-skipping kernel with copies per thread: strides, channel and output counts that are no multiple of
    four, 32 and 64 outputs to a CTA with ragged last ones."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(C + J + k + stride)
    B, H, W = 5, 19, 17
    x, w = P.make_inputs(C + J + k, (B, H, W, C), (k * k * C + 1, J), "ref", bias=True)
    params = O.cv_params(k, k, stride, stride, "SAME")
    pt, pl, Nh, Nw = ops.conv_geometry(H, W, k, k, stride, stride, "SAME")
    gr = rng.standard_normal((B, Nh, Nw, J)).astype(np.float32)
    if pattern == "hot":
        gr[..., rng.permutation(J)[max(1, J // 8):]] = 0
    elif pattern == "late":
        gr[:3] = 0
        gr[..., ::3] = 0
    elif pattern == "none":
        gr[:] = 0
    xd, wd, gd = (torch.from_numpy(a).cuda() for a in (x, w, gr))
    out = ops.snn_cv(xd, wd, params, pt, pl, Nh, Nw)
    _, dw1, _ = ops.snn_cv_grad(gd, xd, wd, params, out, pt, pl, opts=_lib.options(dw_kernel=1))
    _, dw2, _ = ops.snn_cv_grad(gd, xd, wd, params, out, pt, pl, opts=_lib.options(dw_kernel=2))
    assert float((dw2 - dw1).norm()) <= 1e-5 * float(dw1.norm())     # sums of 32-bit floats in another order
    _, dw3, _ = ops.snn_cv_grad(gd, xd, wd, params, out, pt, pl, opts=_lib.options(dw_kernel=2))
    assert torch.equal(dw2, dw3)
