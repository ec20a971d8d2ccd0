"""The native autograd nodes among torch's own: saved-tensor hooks reach everything they keep for their backward (activation
checkpointing and offloading free it all, and give the gradients of the plain call), and undefined gradients are zeros."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint

from tests import util

pytestmark = pytest.mark.gpu
DEV = 'cuda:0'
B, H, L, d = 2, 4, 130, 16
STEP = B * H * L * d * 4        # bytes of one (B, H, L, d) tensor


def cases(fwp, start=None):
    """name -> (leaves, call, how many (B, H, L, d) tensors the node keeps besides inputs and outputs); every call starts
    from multiples of start['W'], start['h']"""
    from recurrent_fwp_b200.delta_layer_io import delta_attention
    if start is None:
        start = {'W': torch.zeros(B, H, d, d, device=DEV), 'h': torch.zeros(B, H, 1, d, device=DEV)}
    # factors, none of them 1: tensors of their own, also for a tracer that merges equal nodes
    W, h = lambda f=3: start['W'] * f, lambda f=3: start['h'] * f
    q, k, v, b, _ = (t.to(DEV) for t in util.delta_inputs(81, B, H, L, d))
    qkvb = torch.randn(L, B, H, 3 * d + 1, generator=util.gen(82)).to(DEV)
    rec = [t.to(DEV) for t in util.rec_inputs(83, B, H, L, d)[:8]]
    rnn = [t.to(DEV) for t in util.rnn_inputs(84, B, H, L, d)[:4]]
    lstm = [t.to(DEV) for g in util.lstm_inputs(85, B, H, L, d)[0] for t in g]
    call_lstm = lambda f: lambda *x: f(*x[0:4], W(), *x[4:8], W(2), *x[8:12], W(4), h(), h(2))[0]
    return {'delta': ([q, k, v, b], lambda *x: fwp.fast_weight_delta(*x, W()), 1),
            'layer': ([qkvb], lambda x: delta_attention(x, W(), 0.25), 4),
            'sum': ([q, k, v], lambda *x: fwp.fast_weight_sum(*x, W()), 0),
            'rec': (rec, lambda *x: fwp.rec_update_fwm_tanh(*x, W(), h()), 4),
            'rnn1': (rnn, lambda z_, k_, v_, b_: fwp.fast_rnn(z_, k_, v_, W(), b_, h()), 1),
            'rnn2': (rnn, lambda z_, k_, v_, b_: fwp.fast_rnn_v2(z_, k_, v_, W(), b_, h()), 2),
            'lstm1': (lstm, call_lstm(fwp.fast_lstm), 6),
            'lstm4': (lstm, call_lstm(fwp.fast_lstm_v4), 7)}


@pytest.mark.parametrize('name', ['delta', 'layer', 'sum', 'rec', 'rnn1', 'rnn2', 'lstm1', 'lstm4'])
def test_hooks_see_every_kept_buffer(fwp, name):
    leaves, call, kept = cases(fwp)[name]
    plain = [t.clone().requires_grad_() for t in leaves]
    y = call(*plain)
    gy = torch.randn(y.shape, generator=util.gen(86)).to(DEV)
    y.backward(gy)

    def run(wrapped):
        x = [t.clone().requires_grad_() for t in leaves]
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        out = wrapped(*x)
        held = torch.cuda.memory_allocated() - before - out.numel() * 4
        out.backward(gy)
        for a, r in zip(x, plain):
            assert torch.equal(a.grad, r.grad)
        return held

    def offloaded(*x):
        with torch.autograd.graph.save_on_cpu():
            return call(*x)

    own = run(call)
    assert own >= kept * STEP
    # with its tensors elsewhere a call holds no more than small change (states and the like)
    assert run(offloaded) < STEP
    assert run(lambda *x: checkpoint(call, *x, use_reentrant=False)) < STEP


class Cut(torch.autograd.Function):
    """Passes a tensor on and hands no gradient back: the node before it gets an undefined one."""

    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, g):
        return None


@pytest.mark.parametrize('name', ['delta', 'layer', 'sum', 'rec', 'rnn1', 'rnn2', 'lstm1', 'lstm4'])
def test_an_undefined_incoming_gradient_counts_as_zeros(fwp, name):
    leaves, call, _ = cases(fwp)[name]
    x = [t.clone().requires_grad_() for t in leaves]
    Cut.apply(call(*x)).sum().backward()
    for t in x:
        assert t.grad is not None and not t.grad.any()


def test_fault_check_covers_both_rules_and_directions(fwp):
    """With the check on, a wait that ran out (the library's bounded probe raises the flag) fails the next call."""
    from recurrent_fwp_b200 import _lib

    def ran_out():
        stream, dev = _lib.stream_and_device(torch.zeros(1, device=DEV))
        _lib.check(_lib.lib.fwp_debug_bounded_wait_probe(64, stream, dev), 'probe')

    try:
        _lib.native.check_device_fault(True)
        for name in ('delta', 'layer', 'sum'):
            leaves, call, _ = cases(fwp)[name]
            x = [t.clone().requires_grad_() for t in leaves]
            y = call(*x)
            ran_out()
            with pytest.raises(RuntimeError, match='bounded wait'):
                call(*x)
            ran_out()
            with pytest.raises(RuntimeError, match='bounded wait'):
                y.sum().backward()
    finally:
        _lib.native.check_device_fault(False)
        _lib.device_fault()


@pytest.mark.parametrize('name', ['delta', 'layer', 'sum', 'rec', 'rnn1', 'rnn2', 'lstm1', 'lstm4'])
def test_tracing_records_the_call(fwp, name):
    """torch.jit.trace: the traced function computes, and differentiates, on new inputs what the plain one does."""
    W, h = torch.full((B, H, d, d), 0.1, device=DEV), torch.full((B, H, 1, d), 0.1, device=DEV)
    start = {}
    leaves, call, _ = cases(fwp, start)[name]

    def f(W0, h0, *x):
        start.update(W=W0, h=h0)
        return call(*x) * 2

    traced = torch.jit.trace(f, (W * 0, h * 0, *(t.flip(0) for t in leaves)))
    x, r = ([t.clone().requires_grad_() for t in leaves] for _ in range(2))
    y, ref = traced(W, h, *x), f(W, h, *r)
    assert torch.equal(y, ref)
    gy = torch.randn(y.shape, generator=util.gen(87)).to(DEV)
    y.backward(gy)
    ref.backward(gy)
    for a, b in zip(x, r):
        assert torch.equal(a.grad, b.grad)


@pytest.mark.parametrize('name', ['delta', 'layer', 'sum', 'rec', 'rnn1', 'lstm1'])
def test_forward_mode_and_function_transforms_are_refused(fwp, name):
    """The ops have a backward only: a tangent or a transform raises, as from any autograd.Function without them."""
    import torch.autograd.forward_ad as fw
    leaves, call, _ = cases(fwp)[name]
    with fw.dual_level():
        x = [fw.make_dual(leaves[0], torch.ones_like(leaves[0]))] + leaves[1:]
        with pytest.raises(RuntimeError):
            call(*x)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: call(t, *leaves[1:]))(torch.stack([leaves[0]] * 2))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: call(t, *leaves[1:]).sum())(leaves[0])
    assert call(*leaves).isfinite().all()
