"""The sorted lists of the per-row bucket sort (csrc/snntc_sort.cu), read back from the workspace, against numpy: ascending in
(value, source index), inputs that never spike left out. Row lengths on both sides of every change of launch shape, rows of
equal inputs (one bucket holds everything), of few distinct values, with outliers, and receptive fields with taps outside
the image."""
import numpy as np
import pytest

import oracle as O
from tests import parity as P

pytestmark = pytest.mark.gpu


def _values(rng, shape, kind):
    if kind == "spread":
        x = np.exp(1.5 * rng.random(shape))
        x[rng.random(shape) < 0.4] = 1e5
    elif kind == "equal":
        x = np.full(shape, np.e)
    elif kind == "few":
        x = rng.integers(-3, 9, shape) / 4.0
    else:   # one far outlier among close values
        x = 1.0 + 1e-3 * rng.random(shape)
        x.reshape(shape[0], -1)[:, 0] = 9e4
    return x.astype(np.float32)


def _check(ws, rows, J, what):
    R, I = rows.shape
    stride = (I + 3) // 4 * 4
    raw = ws.cpu().numpy().view(np.uint8)
    lists = raw[:R * stride * 8].view(np.uint32).reshape(R, stride, 2)
    counts = raw[R * stride * 8:R * stride * 8 + 4 * R].view(np.int32)
    for r in range(R):
        keep = np.flatnonzero(~(rows[r] > np.float32(1e5) - np.float32(0.1)))
        order = keep[np.lexsort((keep, rows[r][keep]))]
        assert counts[r] == len(order), "%s row %d" % (what, r)
        assert np.array_equal(lists[r, :len(order), 0].view(np.float32), rows[r][order]), "%s row %d values" % (what, r)
        assert np.array_equal(lists[r, :len(order), 1], (order * J).astype(np.uint32)), "%s row %d indices" % (what, r)


@pytest.mark.parametrize("I", [1, 40, 257, 1000, 1024, 1025, 4096, 4097, 8192, 8193, 20000, 28900])
@pytest.mark.parametrize("kind", ["spread", "equal", "few", "outlier"])
def test_dense_rows(I, kind):
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(I)
    x = _values(rng, (3, I), kind)
    w = torch.zeros((I + 1, 8), device="cuda")
    ws = ops.fc_forward_workspace(3, I, 8, "cuda")
    ops.snn_fc(torch.from_numpy(x).cuda(), w, O.fc_params(biasvolt=1.0), opts=_lib.options(forward_parts=1, list_builder=1), workspace=ws)
    _check(ws, x, 8, "dense %d %s" % (I, kind))


@pytest.mark.parametrize("I", [300, 1024])
@pytest.mark.parametrize("kind", ["spread", "equal", "few"])
def test_many_dense_rows(I, kind):
    """More rows than 16 per SM: a warp per row."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(I + 1)
    x = _values(rng, (2500, I), kind)
    w = torch.zeros((I + 1, 4), device="cuda")
    ws = ops.fc_forward_workspace(2500, I, 4, "cuda")
    ops.snn_fc(torch.from_numpy(x).cuda(), w, O.fc_params(biasvolt=1.0), opts=_lib.options(forward_parts=1, list_builder=1), workspace=ws)
    _check(ws, x, 4, "many rows %d %s" % (I, kind))


@pytest.mark.parametrize("B,H,W,C,K,S", [(2, 11, 9, 20, 5, 2), (1, 9, 9, 64, 7, 2), (40, 12, 13, 12, 5, 1)])
def test_receptive_fields(B, H, W, C, K, S):
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(C)
    x = _values(rng, (B, H, W, C), "spread")
    params = O.cv_params(K, K, S, S, "SAME", 1.0)
    pt, pl, Nh, Nw = ops.conv_geometry(H, W, K, K, S, S, "SAME")
    w = torch.zeros((K * K * C + 1, 4), device="cuda")
    xd = torch.from_numpy(x).cuda()
    ws = ops.cv_forward_workspace(xd, w, params, Nh, Nw)
    ops.snn_cv(xd, w, params, pt, pl, Nh, Nw, opts=_lib.options(forward_parts=1, list_builder=1), workspace=ws)
    _check(ws, P.im2col_rows(x, K, K, S, S, "SAME"), 4, "fields")


@pytest.mark.parametrize("R,I", [(7, 65), (5, 70), (3, 147), (6, 200), (9, 256), (2500, 65), (2400, 147), (2400, 256), (2400, 511),
                                 (5, 1), (2500, 31), (11, 33), (2500, 64)])
@pytest.mark.parametrize("kind", ["spread", "equal", "few", "outlier"])
def test_short_dense_rows(R, I, kind):
    """65 to 256 inputs, a CTA per row and (from 16 rows per SM on) a warp per row; up to 64, the register network, which is the
    library's own choice there."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(R + I)
    x = _values(rng, (R, I), kind)
    w = torch.zeros((I + 1, 4), device="cuda")
    for builder in (0, 1) if I > 64 else (0, 1, 3):
        ws = ops.fc_forward_workspace(R, I, 4, "cuda")
        ops.snn_fc(torch.from_numpy(x).cuda(), w, O.fc_params(biasvolt=1.0), opts=_lib.options(forward_parts=1, list_builder=builder), workspace=ws)
        _check(ws, x, 4, "short rows %d %s, builder %d" % (I, kind, builder))


@pytest.mark.parametrize("B,H,W,C,K,S", [(3, 31, 30, 70, 3, 1), (10, 32, 31, 16, 7, 2), (3, 29, 30, 7, 9, 1)])
def test_many_receptive_fields(B, H, W, C, K, S):
    """A warp per row of more than 512 inputs, which only receptive fields get (630, 784 and 567 inputs, at least 2368 rows)."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(C + K)
    x = _values(rng, (B, H, W, C), "spread")
    params = O.cv_params(K, K, S, S, "SAME", 1.0)
    pt, pl, Nh, Nw = ops.conv_geometry(H, W, K, K, S, S, "SAME")
    assert 512 < K * K * C <= 1024 and B * Nh * Nw >= 2368
    w = torch.zeros((K * K * C + 1, 4), device="cuda")
    xd = torch.from_numpy(x).cuda()
    ws = ops.cv_forward_workspace(xd, w, params, Nh, Nw)
    ops.snn_cv(xd, w, params, pt, pl, Nh, Nw, opts=_lib.options(forward_parts=1, list_builder=1), workspace=ws)
    _check(ws, P.im2col_rows(x, K, K, S, S, "SAME"), 4, "fields")
