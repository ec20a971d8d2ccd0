"""The native host path of the autograd entry points: what the parity tests do not reach -- arguments that have to be
laid out first, states that must not be changed behind a pending backward, and calls without gradients."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu
DEV = 'cuda:0'


def ins(dtype=torch.float32):
    return [t.to(DEV) for t in util.delta_inputs(5, 2, 3, 19, 16, dtype=dtype)]


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
def test_inner_strided_streams_are_laid_out_and_their_gradients_flow_back(fwp, dtype):
    *x, gy = ins(dtype)
    x = x[:3] + [x[3]]
    flat = [t.clone().requires_grad_() for t in x]
    tall = [t.transpose(2, 3).contiguous().requires_grad_() for t in x[:3]] + [x[3].clone().requires_grad_()]
    W1, W2 = (torch.zeros(2, 3, 16, 16, device=DEV) for _ in range(2))
    y1 = fwp.fast_weight_delta(*flat, W1)
    y2 = fwp.fast_weight_delta(*[t.transpose(2, 3) for t in tall[:3]], tall[3], W2)
    assert torch.equal(y1, y2) and torch.equal(W1, W2)
    y1.backward(gy)
    y2.backward(gy.expand_as(gy))
    for a, b in zip(flat[:3], tall[:3]):
        assert torch.equal(a.grad, b.grad.transpose(2, 3))


def test_states_and_inputs_are_version_checked_and_graphs_are_freed(fwp):
    *x, gy = ins()
    x = [t.requires_grad_() for t in x]
    W = torch.zeros(2, 3, 16, 16, device=DEV)
    y = fwp.fast_weight_delta(*x, W)
    W.zero_()
    with pytest.raises(RuntimeError, match='modified by an inplace operation'):
        y.backward(gy)
    y = fwp.fast_weight_delta(*x, torch.zeros_like(W))
    y.backward(gy)
    with pytest.raises(RuntimeError, match='second time'):
        y.backward(gy)


def test_calls_without_gradients_give_the_same_outputs(fwp):
    *x, _ = ins()
    W1, W2 = (torch.randn(2, 3, 16, 16, device=DEV, generator=torch.Generator(DEV).manual_seed(1)) for _ in range(2))
    with torch.no_grad():
        y1 = fwp.fast_weight_delta(*x, W1)
    y2 = fwp.fast_weight_delta(*[t.clone().requires_grad_() for t in x], W2)
    assert not y1.requires_grad and y2.requires_grad and torch.equal(y1, y2) and torch.equal(W1, W2)
