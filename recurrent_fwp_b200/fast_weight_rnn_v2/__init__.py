"""Delta RNN v2: drop-in for the reference's ``fast_weight_rnn_v2`` module.

Mirrors ``FastRNNv2`` / ``fast_rnn_v2`` of algorithmic/fast_weight_rnn_v2/__init__.py:29-121
(argument order ``Z, K, V, W, beta, h0`` -- W before beta).  Per step the fast
matrix is written by the delta rule from (k, v, beta) and read with the
softmax-normalised previous hidden state: ``h_t = W_t softmax_eps(h_{t-1}) + z_t``.
``W`` [N,H,d,d] and ``h0`` [N,H,1,d] are updated in place to the end-of-segment
state; backward rewinds ``W`` in place and returns no gradient for W and h0.
"""
import torch

from recurrent_fwp_b200 import _lib


def _normalise(Z, K, V, W, beta, h0):
    N, H, L, _ = Z.shape
    M = V.shape[3]
    assert K.shape == (N, H, L, M)
    assert V.shape == (N, H, L, M)
    assert h0.shape == (N, H, 1, M)
    assert W.shape == (N, H, M, M)
    if Z.dtype != torch.float32:
        raise TypeError('the recurrent fast-weight kernels take float32 tensors')
    _lib.require_streams(Z, {'Z': (Z, (N, H, L, M)), 'K': (K, (N, H, L, M)), 'V': (V, (N, H, L, M)),
                             'beta': (beta, (N, H, L, 1))})
    _lib.require_f32(Z, {'W': (W, (N, H, M, M)), 'h0': (h0, (N, H, 1, M))})
    _lib.require_cuda(Z, K, V, W, beta, h0)
    if W.stride(3) != 1 or h0.stride(3) != 1:
        raise RuntimeError('W and h0 must have a unit innermost stride (they are updated in place)')
    Z, K, V, beta = (_lib.unit_inner(t) for t in (Z, K, V, beta))
    return Z, K, V, W, beta, h0


class FastRNNv2(torch.autograd.Function):
    """Fast RNN with the FWM update rule (v2: softmax on the delayed state); native like the delta rule's."""

    apply = staticmethod(_lib.entry_point('fast_rnn_v2', _normalise))


fast_rnn_v2 = FastRNNv2.apply
