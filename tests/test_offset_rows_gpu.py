"""Long calls whose rows do not start on 16-byte boundaries (slices of a wider projection) through the d = 32 role
kernels, which then stage word by word, against the general kernels on aligned copies; sequence counts and lengths on
both sides of a chunk."""
import pytest
import torch

from tests import util
from tests.test_family_plans_gpu import D, DEV, close, misalign, note_backward_kernel, run_lstm, run_rnn

pytestmark = pytest.mark.gpu
SHAPES = [(1, 2, 64), (1, 3, 71)]


def state(seed, B, H, rows):
    return torch.randn(B, H, rows, D, generator=util.gen(seed)) * 0.1


def both(run, keys):
    from recurrent_fwp_b200 import _lib
    off = run(True)
    try:
        for key in keys:
            _lib.tune(key, 0)
        ref = run(False)
    finally:
        for key in keys:
            _lib.tune(key, 1)
    return off, ref


@pytest.mark.parametrize('ver', [2, 1])
@pytest.mark.parametrize('B,H,L', SHAPES)
def test_rnn(fwp, ver, B, H, L):
    z, k, v, b, gy = util.rnn_inputs(51, B, H, L, D)
    args = (z, k, v, b, state(52, B, H, D), state(53, B, H, 1), gy)
    off, ref = both(lambda mis: run_rnn(ver, *args, mis=mis), ['rnn_bwd.32.roles'])
    assert off['kb'] == 'rnn_bwd_roles32_kernel' and ref['kb'] == 'rnn_bwd_kernel'
    assert close(off['W_back'], ref['W_back'])
    for a, r in zip(off['g'], ref['g']):
        assert close(a, r)


@pytest.mark.parametrize('variant', [1, 3])
@pytest.mark.parametrize('B,H,L', SHAPES)
def test_lstm(fwp, variant, B, H, L):
    gates, gy = util.lstm_inputs(61, B, H, L, D)
    Ws = [state(62 + i, B, H, D) for i in range(3)]
    args = (gates, Ws, state(65, B, H, 1), state(66, B, H, 1), gy)
    off, ref = both(lambda mis: run_lstm(variant, *args, mis=mis), ['lstm_fwd.32.gates', 'lstm_bwd.32.roles'])
    assert off['kf'] == 'lstm_fwd_gates32_kernel' and off['kb'] == 'lstm_bwd_roles32_kernel'
    assert ref['kf'] == 'lstm_fwd_kernel' and ref['kb'] == 'lstm_bwd_kernel'
    assert close(off['y'], ref['y']) and close(off['cell'], ref['cell'])
    for a, r in zip(off['W_end'] + off['W_back'] + off['g'], ref['W_end'] + ref['W_back'] + ref['g']):
        assert close(a, r)


@pytest.mark.parametrize('B,H,L', SHAPES)
def test_recurrent_delta(fwp, B, H, L):
    from recurrent_fwp_b200.rec_update_fwm_tanh import rec_update_fwm_tanh
    *ins, gy = util.rec_inputs(71, B, H, L, D)
    W0, h0 = state(72, B, H, D), state(73, B, H, 1)

    def run(mis):
        leaves = [(misalign(t.to(DEV)) if mis and i < 3 else t.clone().to(DEV)).requires_grad_() for i, t in enumerate(ins)]
        W, hs, kb = W0.clone().to(DEV), h0.clone().to(DEV), []
        y = rec_update_fwm_tanh(*leaves, W, hs)
        note_backward_kernel(leaves[0], kb)
        y.backward(gy.to(DEV))
        return dict(y=y.detach(), W_back=W, g=[l.grad for l in leaves], kb=kb[0])
    off, ref = both(run, ['rec_bwd.32.roles'])
    assert off['kb'] == 'rec_bwd_roles32_kernel' and ref['kb'] == 'rec_bwd_kernel'
    assert close(off['y'], ref['y']) and close(off['W_back'], ref['W_back'])
    for a, r in zip(off['g'], ref['g']):
        assert close(a, r)
