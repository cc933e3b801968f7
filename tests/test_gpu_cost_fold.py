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


def test_a_frozen_weight_gets_no_cost():
    """autograd gives a weight with requires_grad=False nothing, so the bucket's slice of it holds what the operators wrote
    there and no cost; the other slices hold both."""
    import torch
    net, x, labels = _net_and_batch(1)
    loss_only, want, _ = _expected(net, x, labels)
    frozen, free = net.weighted_layers()
    frozen.weight.requires_grad_(False)
    net.backward(net.loss(x, labels) + net.constraint_cost(K, K2))
    n = frozen.weight.numel()
    assert torch.equal(net.flat_grad[n:], want[n:])
    assert not torch.equal(want[:n], loss_only[:n])          # (there is a cost to leave out)
    assert torch.equal(net.flat_grad[:n], loss_only[:n])


@pytest.mark.parametrize("kind", ["tensor", "post_accumulate", "node"])
def test_a_hook_on_a_weight_sees_the_cost(kind):
    """Every kind of hook that autograd calls when a gradient reaches a weight sees the cost's gradient, and the bucket holds
    the whole objective's all the same."""
    import torch
    net, x, labels = _net_and_batch(2)
    _, want, cost = _expected(net, x, labels)
    w = net.weighted_layers()[0].weight
    seen = []
    if kind == "tensor":
        w.register_hook(lambda g: seen.append(g.clone()))
    elif kind == "post_accumulate":
        w.register_post_accumulate_grad_hook(lambda p: seen.append(p.grad.clone()))
    else:
        node = w.view_as(w).grad_fn.next_functions[0][0]
        node.register_prehook(lambda gs: seen.append(gs[0].clone()) if gs[0] is not None else None)
    net.backward(net.loss(x, labels) + net.constraint_cost(K, K2))
    assert len(seen) >= 1 and torch.equal(seen[-1], cost[0])
    assert torch.equal(net.flat_grad, want)


def test_a_cost_formed_on_another_stream_is_waited_for():
    """A term whose backward runs on another stream than the caller's goes autograd's way, which orders the streams."""
    import torch
    net, x, labels = _net_and_batch(3)
    _, want, _ = _expected(net, x, labels)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    big = torch.randn(4096, 4096, device="cuda")
    with torch.cuda.stream(side):
        scale = (big @ big @ big).mean() * 0 + 1.0           # keeps the side stream busy in front of the cost
        cost = net.constraint_cost(K, K2) * scale
    torch.cuda.current_stream().wait_stream(side)
    net.backward(net.loss(x, labels) + cost)
    assert torch.equal(net.flat_grad, want)
