"""The walk that copies its weight rows ahead into shared memory (csrc/snntc_walk_ring.cu) and the one with several rows per warp
(csrc/snntc_walk_rows.cu), against the oracle's protocol and bit for bit against the walk from global memory: fan-in around the
edges of groups (4, 8 entries), blocks (16, 32) and the ring of weight blocks, ragged fan-out, rows of unequal length, ties,
inputs below the bias input, rows whose every output fires early. And fan-outs whose weights are copied with padded rows."""
import numpy as np
import pytest

import oracle as O
from tests import parity as P

pytestmark = pytest.mark.gpu

LAYOUTS = (16, 32, 64)   # walk_layout of the measurement build: copied ahead; rows per warp, weights global / in shared memory


def _checked(x, w, params):
    import torch
    from snntc_2023_b200 import _lib, ops
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    a = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=1 if w.shape[1] % 2 == 0 else 2))
    for layout in LAYOUTS:   # (the last two need a fan-out up to 64 that is a multiple of four)
        b = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=layout))
        assert torch.equal(a, b), "layout %d" % layout
    return b


@pytest.mark.parametrize("I", [1, 7, 8, 9, 63, 64, 65, 127, 129, 257, 384, 385, 784, 1500])
@pytest.mark.parametrize("J", [1, 4, 10, 20, 36, 63, 64, 100, 130])
def test_walks_agree_with_the_walk_from_global_memory(I, J):
    bv = 1.0 if (I + J) % 3 else 0.0
    x, w = P.make_inputs(1000 * I + J, (5, I), (I + (bv > 0), J), "ref" if I > 8 else "test", bias=bv > 0)
    params = O.fc_params(biasvolt=bv)
    bc = _checked(x, w, params).cpu().numpy()
    P.check_forward(bc[:5], bc[5:], O.fc_forward(x, w, params, "f32"), O.fc_forward(x, w, params, "f64"), rows=x,
                    what="ring walk I=%d J=%d" % (I, J), max_flagged=0.2)


@pytest.mark.parametrize("bv", [0.0, 1.0])
@pytest.mark.parametrize("lo,hi", [(4, 40), (1, 12), (-8, 12)])
def test_walks_on_exact_ties_and_inputs_below_the_bias_input(bv, lo, hi):
    rng = np.random.default_rng(10 * abs(lo) + hi)
    x = (rng.integers(lo, hi, size=(9, 300)) / 4.0).astype(np.float32)
    x[::2, ::3] = 1e5
    w = (rng.integers(-12, 13, size=(300 + (bv > 0), 96)) / 4.0).astype(np.float32)
    _checked(x, w, O.fc_params(biasvolt=bv))


def test_walks_stop_when_every_output_has_fired():
    rng = np.random.default_rng(3)
    x = np.exp(rng.random((4, 2000))).astype(np.float32)
    w = np.abs(rng.standard_normal((2001, 70))).astype(np.float32)     # positive weights: everything fires within a few entries
    assert float(_checked(x, w, O.fc_params(biasvolt=1.0))[:4].max()) < 1e5


@pytest.mark.parametrize("R,I,J", [(1300, 40, 3), (1300, 90, 10), (2500, 70, 33), (700, 130, 77), (300, 257, 215)])
def test_padded_weight_rows(R, I, J):
    """Enough items that a fan-out that is no multiple of four gets padded weights: the same bits as without (layout 2)."""
    import torch
    from snntc_2023_b200 import _lib, ops
    x, w = P.make_inputs(R + I + J, (R, I), (I + 1, J), "ref", bias=True)
    params = O.fc_params(biasvolt=1.0)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    assert torch.equal(ops.snn_fc(xd, wd, params), ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2)))
    assert torch.equal(ops.snn_fc_infer(xd, wd, params), ops.snn_fc(xd, wd, params)[:R])


@pytest.mark.parametrize("R,I,J", [(8000, 80, 10), (9000, 90, 27), (15000, 70, 50), (33000, 66, 61), (33000, 66, 63), (2500, 130, 77),
                                   (1500, 260, 215), (2500, 70, 33)])
@pytest.mark.parametrize("bv,sentinels,positive", [(1.0, True, False), (0.0, False, False), (1.0, False, True)])
def test_padded_weight_rows_of_every_walk(R, I, J, bv, sentinels, positive):
    """Padded weight rows in the several-rows walk (J up to 64) and the walks from global memory: training and inference, with and
    without inputs that never spike and a bias row; positive weights: every output fires early, so that the padding, which
    never does, decides when a row is done."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(R + J)
    x = np.exp(1.5 * rng.random((R, I))).astype(np.float32)
    if sentinels:
        x[rng.random((R, I)) < 0.4] = 1e5
    w = (rng.standard_normal((I + (bv > 0), J)) * np.sqrt(15.0 / I)).astype(np.float32)
    if positive:
        w = np.abs(w)
        w[I:] = 0.0      # (a bias weight of 1 or more would put the spike in front of the bias input: none)
    params = O.fc_params(biasvolt=bv)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    out = ops.snn_fc(xd, wd, params)
    assert torch.equal(out, ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2)))
    assert torch.equal(ops.snn_fc_infer(xd, wd, params), out[:R])
    # (a decision within rounding of a tie can leave an output without a spike: 1 of 243 000 of the fp32 oracle at 9000 x 90 x 27)
    assert not positive or float((out[:R] >= 1e5).float().mean()) < 1e-4


@pytest.mark.parametrize("R,I,J", [(1400, 40, 200), (1500, 33, 200), (2600, 30, 128), (4900, 30, 128), (9400, 21, 160), (700, 50, 512),
                                   (1300, 64, 66), (5000, 20, 68), (2500, 90, 1000)])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_choice_among_the_walks_from_global_memory(R, I, J, offset):
    """Both sides of the lines between output pairs and four outputs per lane (33 to 70 warps of 64 outputs per SM and beyond,
    narrow last blocks), with weights that start on a 16-, 4- or 8-byte boundary: the bits of one output per lane."""
    import torch
    from snntc_2023_b200 import _lib, ops
    x, w = P.make_inputs(R + I + J, (R, I), (I + 1, J), "ref", bias=True)
    params = O.fc_params(biasvolt=1.0)
    xd = torch.from_numpy(x).cuda()
    flat = torch.zeros(w.size + 4, device="cuda")
    wd = flat[offset:offset + w.size].view(w.shape).copy_(torch.from_numpy(w))
    assert wd.data_ptr() % 16 == 4 * offset
    out = ops.snn_fc(xd, wd, params)
    ref = ops.snn_fc(xd, torch.from_numpy(w).cuda(), params, opts=_lib.options(walk_layout=2, walk_outputs=1))
    assert torch.equal(out, ref)
    assert torch.equal(ops.snn_fc_infer(xd, wd, params), out[:R])


@pytest.mark.parametrize("J", [16, 64, 96, 132])
@pytest.mark.parametrize("band,scale", [(1e-4, 3e4), (1e-3, 3e3), (3e-3, 1e3)])
def test_spikes_that_rounding_hides_and_negative_denominators(J, band, scale):
    """Inputs so close together that rounding decides many steps: outputs cross their threshold without a spike, stay behind it
    (the walks turn their sums' sign), and some spike on the way back, with a negative denominator. Every layout: the bits of one
    output per lane, which takes every such step through the reference's comparisons."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(J)
    I, R = 300, 600
    x = np.exp(band * rng.random((R, I))).astype(np.float32)
    w = (rng.standard_normal((I + 1, J)) * np.sqrt(15.0 / I) * scale).astype(np.float32)
    w[I] = 0.0
    params = O.fc_params(biasvolt=1.0)
    o32, o64 = O.fc_forward(x[:64], w, params, "f32"), O.fc_forward(x[:64], w, params, "f64")
    assert ((o32["y"] < 9e4) != (o64["y"] < 9e4)).sum() > 0 or J == 16
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    ref = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2, walk_outputs=1))
    assert band > 1e-4 or int((ref[R:] < 0).sum()) > 0
    for layout in (0, 1, 3, 8, 16, 32, 64):
        assert torch.equal(ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=layout)), ref), "layout %d" % layout
    got = ref[:64].cpu().numpy()
    assert np.array_equal(got < 9e4, o32["y"] < 9e4)


@pytest.mark.parametrize("R,I,J", [(37, 33, 100), (37, 64, 128), (75, 97, 36), (290, 70, 256), (290, 31, 200), (148, 65, 500), (900, 40, 64),
                                   (600, 200, 12)])
@pytest.mark.parametrize("bv", [0.0, 1.0])
def test_walk_with_a_copying_warp(R, I, J, bv):
    """One, two and four warps beside the one that copies (chosen by the number of CTAs), ragged slices, lists that end anywhere in a
    block, an empty row, a row of ties: the bits of one output per lane from global memory."""
    import torch
    from snntc_2023_b200 import _lib, ops
    x, w = P.make_inputs(R + I + J, (R, I), (I + (bv > 0), J), "ref", bias=bv > 0)
    x[3] = 1e5
    x[5] = 2.0
    params = O.fc_params(biasvolt=bv)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    ref = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2, walk_outputs=1))
    assert torch.equal(ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=16)), ref)
    assert torch.equal(ops.snn_fc(xd, wd, params), ref)


@pytest.mark.parametrize("R,I,J", [(1481, 15, 17), (1600, 16, 32), (2500, 47, 20), (3552, 70, 27), (3553, 40, 32), (1480, 300, 24)])
@pytest.mark.parametrize("bv", [0.0, 1.0])
def test_walk_whose_warps_copy_for_themselves(R, I, J, bv):
    """Fan-outs of 17 to 32 at 10 to 24 rows per SM and one row either side, padded and whole, lists that end anywhere in a block of 16,
    an empty row, a row of ties: the bits of one output per lane from global memory."""
    import torch
    from snntc_2023_b200 import _lib, ops
    x, w = P.make_inputs(R + I + J, (R, I), (I + (bv > 0), J), "ref", bias=bv > 0)
    x[np.arange(R) % 7 == 0, :I // 2] = 1e5
    x[3] = 1e5
    x[5] = 2.0
    params = O.fc_params(biasvolt=bv)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    ref = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2, walk_outputs=1))
    assert torch.equal(ops.snn_fc(xd, wd, params), ref)
    assert torch.equal(ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=16)), ref)


@pytest.mark.parametrize("J", [64, 128, 40])
def test_rows_without_inputs_beside_long_ones(J):
    """Every third row has no input that can spike, so that the bias input alone decides (weights above one: the spike, below: none);
    the rows around it end at inputs above that spike, and with 6000 rows every warp of the staged walk takes several."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(J)
    R, I = 6000, 100
    x = np.exp(2 + rng.random((R, I))).astype(np.float32)
    x[::3] = 1e5
    w = (rng.standard_normal((I + 1, J)) * 0.3).astype(np.float32)
    w[I] = np.where(np.arange(J) % 2 == 0, 2.0, 0.5)
    params = O.fc_params(biasvolt=1.0)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    want = np.where(np.arange(J) % 2 == 0, np.float32(2.0), np.float32(1e5))
    for layout in (0, 1, 2, 3, 8, 16, 32, 64):
        y = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=layout))[:R].cpu().numpy()
        assert np.abs(y[::3] - want).max() == 0.0, "layout %d" % layout


@pytest.mark.parametrize("J", [16, 64, 96, 128, 132])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("bv", [0.0, 1.0])
def test_spikes_in_front_of_weights_that_are_no_numbers(J, bad, bv):
    """One infinite or NaN weight in every column, anywhere from the first input to the last: an output that fired in front of it keeps
    its spike, in every layout, and what had not fired by then stays without one. The bits of one output per lane, which keeps a
    flag per output, and the oracle's spikes."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(J)
    R, I = 400, 120
    x = np.exp(1.5 * rng.random((R, I))).astype(np.float32)
    w = (rng.standard_normal((I + (bv > 0), J)) * np.sqrt(15.0 / I)).astype(np.float32)
    w[I:] = 0.0
    w[rng.integers(0, I, J), np.arange(J)] = bad
    x[0, :6] = [1.0, 1.1, 1.2, 1.3, 1.4, 1.5]      # fires at 1.21667 in column 0, then meets `bad`
    x[0, 6:] = 1e5
    w[:6, 0] = [5.0, 1.0, 1.0, 0.1, bad, 0.1]
    w[6:I, 0] = 0.1
    params = O.fc_params(biasvolt=bv)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    ref = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2, walk_outputs=1))
    for layout in (0, 1, 3, 8, 16, 32, 64):
        assert torch.equal(ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=layout)), ref), "layout %d" % layout
    o32 = O.fc_forward(x, w, params, "f32")
    got = ref[:R].cpu().numpy()
    assert np.array_equal(got < 9e4, o32["y"] < 9e4)
    assert abs(got[0, 0] - 1.21667) < 1e-4 and 0.1 < (got < 9e4).mean() < 0.95
    assert np.allclose(got, o32["y"], rtol=1e-5)


@pytest.mark.parametrize("J,layout", [(128, 3), (64, 1), (64, 8), (32, 32)])
def test_rows_with_an_input_below_zero_take_the_comparisons_near_zero_only(J, layout):
    """Where no proof holds that a sum below the margin has fired, the reference's comparisons are taken near zero, not at every step:
    rows with one small negative input against the same rows without it (median of interleaved runs, graph replays of ten calls). The
    comparisons at every spike take 1.12 to 1.37 times as long, those at every step 3.7 to 4.6 times."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(J)
    R, I = 16384, 576
    x = np.exp(1.5 * rng.random((R, I))).astype(np.float32)
    x[rng.random((R, I)) < 0.5] = 1e5
    w = (rng.standard_normal((I + 1, J)) * np.sqrt(15.0 / I)).astype(np.float32)
    w[I] = 1.2                                      # (a spike of the bias input alone would lie at 6, behind every input)
    w[0] = 0.0
    params = O.fc_params(biasvolt=1.0)
    opts = _lib.options(walk_layout=layout)
    times, graphs, outs = ([], []), [], []
    for first in (0.5, -0.5):
        x[:, 0] = first                             # (weight zero: changes no sum)
        xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
        ws = ops.fc_forward_workspace(R, I, J, xd.device)
        outs.append(ops.snn_fc(xd, wd, params, opts=opts, workspace=ws))
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(10):                     # (the walk alone: a negative input widens the range over which the lists are sorted)
                ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=layout, forward_parts=2), workspace=ws)
        graphs.append((g, xd, wd, ws))
    assert torch.equal(outs[0], outs[1])
    for _ in range(7):
        for t, (g, _, _, _) in zip(times, graphs):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.replay()
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
    plain, below = (sorted(t)[3] for t in times)
    assert below < 1.8 * plain, "%.3f ms against %.3f" % (below, plain)


@pytest.mark.parametrize("J", [20, 32])
@pytest.mark.parametrize("R", [600, 1600, 3500])
@pytest.mark.parametrize("band,scale", [(1e-4, 3e4), (1e-3, 3e3), (3e-3, 1e3)])
def test_hidden_spikes_in_the_walk_whose_warps_copy_for_themselves(R, J, band, scale):
    """As above at fan-outs of 17 to 32: by name at any number of rows (128), and as the library chooses it at 1600 and 3500."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(R + J)
    I = 300
    x = np.exp(band * rng.random((R, I))).astype(np.float32)
    w = (rng.standard_normal((I + 1, J)) * np.sqrt(15.0 / I) * scale).astype(np.float32)
    w[I] = 0.0
    params = O.fc_params(biasvolt=1.0)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    ref = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2, walk_outputs=1))
    assert band > 1e-4 or int((ref[R:] < 0).sum()) > 0
    for layout in (0, 16, 128, 256):
        assert torch.equal(ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=layout)), ref), "layout %d" % layout


@pytest.mark.parametrize("J", [4, 16, 20, 32, 36, 100, 256])
@pytest.mark.parametrize("I", [1, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 64, 65, 300])
def test_warps_that_copy_for_themselves_by_name(I, J):
    """Lists that end at every edge of a group of 8 or 16 and a block of 16 or 32, one and several slices of 32 outputs with ragged last ones,
    inputs below zero and below the bias input, empty rows."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(40 * I + J)
    x = np.exp(1.5 * rng.random((70, I))).astype(np.float32)
    x[rng.random((70, I)) < 0.3] = 1e5
    x[2] = 1e5
    x[4, 0] = -0.25
    x[6] = 0.5
    w = (rng.standard_normal((I + 1, J)) * np.sqrt(15.0 / I)).astype(np.float32)
    params = O.fc_params(biasvolt=1.0)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    ref = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2, walk_outputs=1))
    for layout in (128, 256):
        assert torch.equal(ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=layout)), ref), "layout %d" % layout


@pytest.mark.parametrize("J", [32, 64, 128])
@pytest.mark.parametrize("first", [0, 16, 128])
def test_lists_of_one_call_walked_by_the_next(J, first):
    """Lists built without a walk (by a call whose own walk would need no bound on the weight sums), then walked in every layout from the
    same workspace, with inputs so close together that many steps need the bound: the bits of both in one call."""
    import torch
    from snntc_2023_b200 import _lib, ops
    rng = np.random.default_rng(J)
    R, I = 600, 300
    x = np.exp(1e-3 * rng.random((R, I))).astype(np.float32)
    w = (rng.standard_normal((I + 1, J)) * np.sqrt(15.0 / I) * 3e3).astype(np.float32)
    w[I] = 0.0
    params = O.fc_params(biasvolt=1.0)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    ref = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2, walk_outputs=1))
    ws = ops.fc_forward_workspace(R, I, J, xd.device)
    ws.view(torch.int32).fill_(0)                     # a bound of zero, were none formed
    ops.snn_fc(xd, wd, params, opts=_lib.options(forward_parts=1, walk_layout=first), workspace=ws)
    for layout in (1, 2, 3, 8, 16, 32, 64, 128, 256):
        got = ops.snn_fc(xd, wd, params, opts=_lib.options(forward_parts=2, walk_layout=layout), workspace=ws)
        assert torch.equal(got, ref), "layout %d" % layout


@pytest.mark.parametrize("R,I,J", [(590, 64, 12), (595, 64, 12), (889, 257, 24), (1700, 400, 10), (2372, 70, 9), (2400, 300, 16), (3552, 65, 12),
                                   (3553, 65, 12), (886, 60, 10), (900, 70, 64), (890, 300, 96), (1000, 300, 64), (400, 90, 200), (300, 784, 200)])
@pytest.mark.parametrize("bv", [0.0, 1.0])
def test_lines_between_the_walks_that_copy(R, I, J, bv):
    """Either side of the lines between the walk with a copying warp, those whose warps copy for themselves (blocks of 32 and 16 entries) and
    the pairs walk, padded and whole rows: the bits of one output per lane, training and inference."""
    import torch
    from snntc_2023_b200 import _lib, ops
    x, w = P.make_inputs(R + I + J, (R, I), (I + (bv > 0), J), "ref", bias=bv > 0)
    x[np.arange(R) % 5 == 0, :I // 3] = 1e5
    x[3] = 1e5
    params = O.fc_params(biasvolt=bv)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    ref = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2, walk_outputs=1))
    assert torch.equal(ops.snn_fc(xd, wd, params), ref)
    assert torch.equal(ops.snn_fc_infer(xd, wd, params), ref[:R])


@pytest.mark.parametrize("I", [768, 784, 801, 802, 810, 830, 836, 837, 850])
def test_staged_weights_up_to_what_fits(I):
    """The staged walk with 32 warps, with fewer where the weights leave less room, and behind its limit (then the pairs walk)."""
    import torch
    from snntc_2023_b200 import _lib, ops
    x, w = P.make_inputs(I, (5200, I), (I + 1, 64), "ref", bias=True)
    x[::3, ::2] = 1e5
    params = O.fc_params(biasvolt=1.0)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    ref = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=2, walk_outputs=1))
    assert torch.equal(ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=8)), ref)
