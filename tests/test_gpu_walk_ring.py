"""The walk that copies its weight rows ahead into shared memory (csrc/snntc_walk_ring.cu), against the oracle's protocol and
bit for bit against the walk from global memory: fan-in around the edges of groups (4 entries), blocks (32) and the ring of
weight blocks, ragged fan-out, ties, inputs below the bias input, rows whose every output fires early."""
import numpy as np
import pytest

import oracle as O
from tests import parity as P

pytestmark = pytest.mark.gpu

RING = 16   # walk_layout of the measurement build


def _checked(x, w, params):
    import torch
    from snntc_2023_b200 import _lib, ops
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    a = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=1 if w.shape[1] % 2 == 0 else 2))
    b = ops.snn_fc(xd, wd, params, opts=_lib.options(walk_layout=RING))
    assert torch.equal(a, b)
    return b


@pytest.mark.parametrize("I", [1, 7, 8, 9, 63, 64, 65, 127, 129, 257, 384, 385, 784, 1500])
@pytest.mark.parametrize("J", [1, 10, 63, 64, 100, 130])
def test_ring_walk_agrees_with_the_walk_from_global_memory(I, J):
    bv = 1.0 if (I + J) % 3 else 0.0
    x, w = P.make_inputs(1000 * I + J, (5, I), (I + (bv > 0), J), "ref" if I > 8 else "test", bias=bv > 0)
    params = O.fc_params(biasvolt=bv)
    bc = _checked(x, w, params).cpu().numpy()
    P.check_forward(bc[:5], bc[5:], O.fc_forward(x, w, params, "f32"), O.fc_forward(x, w, params, "f64"), rows=x,
                    what="ring walk I=%d J=%d" % (I, J), max_flagged=0.2)


@pytest.mark.parametrize("bv", [0.0, 1.0])
@pytest.mark.parametrize("lo,hi", [(4, 40), (1, 12), (-8, 12)])
def test_ring_walk_on_exact_ties_and_inputs_below_the_bias_input(bv, lo, hi):
    rng = np.random.default_rng(10 * abs(lo) + hi)
    x = (rng.integers(lo, hi, size=(9, 300)) / 4.0).astype(np.float32)
    w = (rng.integers(-12, 13, size=(300 + (bv > 0), 96)) / 4.0).astype(np.float32)
    _checked(x, w, O.fc_params(biasvolt=bv))


def test_ring_walk_stops_when_every_output_has_fired():
    rng = np.random.default_rng(3)
    x = np.exp(rng.random((4, 2000))).astype(np.float32)
    w = np.abs(rng.standard_normal((2001, 70))).astype(np.float32)     # positive weights: everything fires within a few entries
    assert float(_checked(x, w, O.fc_params(biasvolt=1.0))[:4].max()) < 1e5
