"""Small layers are chains of kernels launched as programmatic dependents, on workspaces that the allocator hands out again at once:
calls queued back to back, with other inputs each time, give the bits of the same calls waited for one by one."""
import pytest

pytestmark = pytest.mark.gpu

MLP = [("dense", 200, 96), ("dense", 96, 70), ("dense", 70, 10)]
CONV = [("conv", 3, 16, 3, 1), ("conv", 16, 24, 3, 1), ("pool", 2), ("conv", 24, 27, 5, 2), ("flatten",), ("dense", 4 * 3 * 27, 10)]


@pytest.mark.parametrize("specs,shape", [(MLP, (200,)), (CONV, (14, 10, 3))])
@pytest.mark.parametrize("batch", [1, 3, 33])
def test_back_to_back_steps_match_waited_for_steps(specs, shape, batch):
    import torch
    from snntc_2023_b200 import nets, train
    net = nets.SnnNet(specs, weights=nets.spec_weights(specs, 3))
    g = torch.Generator("cuda").manual_seed(batch)
    inputs = [(torch.rand((batch,) + shape, device="cuda", generator=g), torch.randint(0, 10, (batch,), device="cuda", generator=g))
              for _ in range(6)]

    def step(t, labels, wait):
        x = train.encode(t, one_minus=False)
        for layer in net.layers:
            wait()
            x = layer(x)
        wait()
        loss = train.loss_func(x, labels)
        wait()
        net.backward(loss + net.constraint_cost(100.0, 1e-2))
        wait()
        with torch.no_grad():
            y = net(train.encode(t, one_minus=False))
        return loss.detach().clone(), net.flat_grad.clone(), y

    want = [step(*i, torch.cuda.synchronize) for i in inputs]
    torch.cuda.synchronize()
    got = [step(*inputs[k % 6], lambda: None) for k in range(60)]
    torch.cuda.synchronize()
    for k, result in enumerate(got):
        for a, b in zip(result, want[k % 6]):
            assert torch.equal(a, b), "step %d" % k


def test_loss_of_a_large_batch_in_a_captured_graph():
    """The workspace of the two-launch loss lives in the capture's pool: replays with other inputs give the eager bits."""
    import torch
    from snntc_2023_b200 import train
    from snntc_2023_b200.graph import GraphedStep
    g = torch.Generator("cuda").manual_seed(5)
    batches = [(torch.rand(3000, 300, device="cuda", generator=g) + 1, torch.randint(0, 300, (3000,), device="cuda", generator=g)) for _ in range(4)]
    graphed = GraphedStep(lambda y, lab: train.loss_func(y, lab), list(batches[0]))
    for y, lab in batches:
        assert torch.equal(graphed(y, lab).clone(), train.loss_func(y, lab))
