"""Delta LSTM v1: drop-in for the reference's ``fast_lstm`` module.

Mirrors ``FastLSTM`` / ``fast_lstm`` of language_modeling/src/utils/fast_lstm/__init__.py:36-205:
``forward(ctx, Zi,Ki,Vi,bi,Wi, Zu,Ku,Vu,bu,Wu, Zo,Ko,Vo,bo,Wo, h0, c0) -> (rnn_out, cell_out)``.
The three fast matrices and ``h0``/``c0`` are updated in place to the end-of-segment
state; backward rewinds the matrices in place, ignores ``grad_cell`` (as the
reference does) and returns 12 gradients and 5 ``None``.

The sibling modules ``fast_lstm_v2`` / ``_v3`` / ``_v4`` are built from the same
factory below; they differ in where softmax / sigmoid / the skip term sit
(language_modeling/src/utils/fast_lstm_v{2,3,4}/__init__.py).
"""
import torch

from recurrent_fwp_b200 import _lib


def _normalise(Zi, Ki, Vi, bi, Wi, Zu, Ku, Vu, bu, Wu, Zo, Ko, Vo, bo, Wo, h0, c0):
    N, H, L, _ = Zi.shape
    M = Vi.shape[3]
    assert Ki.shape == (N, H, L, M)
    assert Vi.shape == (N, H, L, M)
    assert h0.shape == (N, H, 1, M)
    assert Wi.shape == (N, H, M, M)
    if Zi.dtype != torch.float32:
        raise TypeError('the recurrent fast-weight kernels take float32 tensors')
    gates = ((Zi, Ki, Vi, bi, Wi), (Zu, Ku, Vu, bu, Wu), (Zo, Ko, Vo, bo, Wo))
    args = []
    for g, (z, k, v, b, w) in zip('iuo', gates):
        _lib.require_streams(Zi, {'Z' + g: (z, (N, H, L, M)), 'K' + g: (k, (N, H, L, M)),
                                  'V' + g: (v, (N, H, L, M)), 'b' + g: (b, (N, H, L, 1))})
        _lib.require_f32(Zi, {'W' + g: (w, (N, H, M, M))})
        if w.stride(3) != 1:
            raise RuntimeError('the fast matrices must have a unit innermost stride (they are updated in place)')
        args += [_lib.unit_inner(t) for t in (z, k, v, b)] + [w]
    _lib.require_f32(Zi, {'h0': (h0, (N, H, 1, M)), 'c0': (c0, (N, H, 1, M))})
    _lib.require_cuda(*args, h0, c0)
    if M > 1 and (h0.stride(3) != 1 or c0.stride(3) != 1):
        raise RuntimeError('h0 and c0 must have a unit innermost stride (they are updated in place)')
    return args + [h0, c0]


def make_lstm_function(variant, name):
    entry = 'fast_lstm' if variant == 1 else 'fast_lstm_v%d' % variant
    return type(name, (torch.autograd.Function,), {
        '__doc__': 'Fast LSTM with the FWM update rule (variant %d); native like the delta rule\'s.' % variant,
        'apply': staticmethod(_lib.entry_point(entry, _normalise))})


FastLSTM = make_lstm_function(1, 'FastLSTM')
fast_lstm = FastLSTM.apply
