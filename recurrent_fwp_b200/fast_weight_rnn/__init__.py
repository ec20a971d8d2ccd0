"""Delta RNN v1: drop-in for the reference's ``fast_weight_rnn`` module.

Mirrors ``FastRNN`` / ``fast_rnn`` of language_modeling/src/utils/fast_weight_rnn/__init__.py:41-118
(argument order ``Z, K, V, W, beta, h0``): ``h_t = softmax(W_t h_{t-1} + z_t)`` with
``W_t`` written by the delta rule.  ``W`` and ``h0`` are updated in place; backward
rewinds ``W`` and returns no gradient for W and h0.
"""
import torch

from recurrent_fwp_b200 import _lib
from recurrent_fwp_b200.fast_weight_rnn_v2 import _normalise


class FastRNN(torch.autograd.Function):
    """Fast RNN with the FWM update rule (v1: softmax on the output); native like the delta rule's."""

    apply = staticmethod(_lib.entry_point('fast_rnn', _normalise))


fast_rnn = FastRNN.apply
