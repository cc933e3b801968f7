"""SnnNet.backward adds the constraint cost's gradient straight to the flat bucket instead of sending it through autograd.
Whatever else goes on in the process, the result has to be what autograd's own way gives."""
import threading

import pytest

pytestmark = pytest.mark.gpu

K, K2 = 100.0, 1e-2


def _net_and_batch(seed=0):
    import torch
    from snntc_2023_b200 import nets
    specs = [("dense", 20, 16), ("dense", 16, 5)]
    net = nets.SnnNet(specs, weights=nets.spec_weights(specs, seed))
    g = torch.Generator("cuda").manual_seed(seed)
    x = torch.exp(torch.rand(12, 20, device="cuda", generator=g))
    return net, x, torch.randint(0, 5, (12,), device="cuda", generator=g)


def _expected(net, x, labels):
    """flat gradient of loss + cost: the loss by SnnNet.backward alone, the cost by autograd."""
    import torch
    net.backward(net.loss(x, labels))
    loss_only = net.flat_grad.clone()
    weights = [l.weight for l in net.weighted_layers()]
    cost = torch.autograd.grad(net.constraint_cost(K, K2), weights)
    return loss_only, loss_only + torch.cat([c.reshape(-1) for c in cost]), cost


def test_a_cost_differentiated_on_another_thread_keeps_its_gradient():
    """While one thread is inside SnnNet.backward, another asks autograd for the gradient of a cost on the same weights:
    each gets its own."""
    import torch
    net, x, labels = _net_and_batch()
    _, want, want_cost = _expected(net, x, labels)
    weights = [l.weight for l in net.weighted_layers()]
    inside, other_done, got, errors = threading.Event(), threading.Event(), [], []

    class Hold(torch.autograd.Function):     # a host node: it runs on the thread that called backward
        @staticmethod
        def forward(ctx, t):
            return t.clone()

        @staticmethod
        def backward(ctx, g):
            inside.set()
            other_done.wait(60)
            return g

    def other():
        try:
            inside.wait(60)
            got.extend(torch.autograd.grad(net.constraint_cost(K, K2), weights))
        except Exception as e:   # pragma: no cover
            errors.append(e)
        finally:
            other_done.set()

    t = threading.Thread(target=other)
    t.start()
    held = Hold.apply(torch.zeros((), requires_grad=True)).to("cuda")
    net.backward(net.loss(x, labels) + net.constraint_cost(K, K2) + held)
    t.join()
    assert not errors and inside.is_set(), errors
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want_cost))
    assert torch.equal(net.flat_grad, want)
