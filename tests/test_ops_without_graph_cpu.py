"""Ops whose gradients are off run their forward without an autograd node, except where something looks at the node."""
import pytest
import torch
from torch.autograd import forward_ad

from uttt_b200.ops.functional import _run


class _Double(torch.autograd.Function):
    nodes = 0

    @staticmethod
    def forward(ctx, x, k):
        _Double.nodes += type(ctx).__name__ != "_NoGraph"
        ctx.save_for_backward(x)
        ctx.set_materialize_grads(False)
        ctx.k = k
        return x * k

    @staticmethod
    def backward(ctx, g):
        return g * ctx.k, None


@pytest.mark.parametrize("grad,needs,nodes", [(True, True, 1), (True, False, 1), (False, True, 0), (False, False, 0)])
def test_values_and_nodes(grad, needs, nodes):
    x = torch.arange(3.0).requires_grad_(needs)
    _Double.nodes = 0
    with torch.set_grad_enabled(grad):
        y = _run(_Double, x, 2.0)
    assert torch.equal(y, torch.tensor([0.0, 2.0, 4.0])) and y.requires_grad == (grad and needs) and _Double.nodes == nodes


def test_what_the_node_refuses_stays_refused():
    x = torch.arange(3.0)
    with torch.no_grad():
        with pytest.raises(RuntimeError):                        # no vmap rule
            torch.func.vmap(lambda t: _run(_Double, t, 2.0))(x)
        with forward_ad.dual_level(), pytest.raises(RuntimeError):      # no jvp
            _run(_Double, forward_ad.make_dual(x, torch.ones(3)), 2.0)


def test_saved_tensor_hooks_see_what_is_saved():
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t) or t, lambda t: t):
        y = _run(_Double, torch.ones(2, requires_grad=True), 3.0)
    y.sum().backward()
    assert len(seen) == 1
