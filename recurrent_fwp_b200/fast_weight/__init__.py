"""Delta-rule fast weight memory: drop-in for the reference's ``fast_weight`` module.

Mirrors ``DeltaFastWeight`` / ``fast_weight_delta`` of
algorithmic/fast_weight/__init__.py:26-96 (also language_modeling/src/utils/fast_fast_weight
and reinforcement_learning/torchbeast/fast_weight): same positional arguments,
same saved tensors, same in-place state semantics --

  * ``W`` [N,H,E,M] enters as the start-of-segment state and is overwritten with
    the end-of-segment state;
  * ``backward`` rewinds that same tensor in place to the start-of-segment state
    (callers that carry the state clone it before backward, as the reference's
    layers do), and returns no gradient for it.

Differences a caller can observe: inputs may be float32 or bfloat16 (the state
and the tensors saved for backward stay float32); the work runs on the current
CUDA stream of the inputs' device instead of the legacy default stream.
"""
import torch

from recurrent_fwp_b200 import _lib


def _normalise(Q, K, V, beta, W):
    N, H, L, E = Q.shape
    M = V.shape[3]
    _lib.io_dtype(Q)
    _lib.require_streams(Q, {'K': (K, (N, H, L, E)), 'V': (V, (N, H, L, M)), 'beta': (beta, (N, H, L, 1))})
    _lib.require_f32(Q, {'W': (W, (N, H, E, M))})
    _lib.require_cuda(Q, K, V, beta, W)
    if W.stride(3) != 1:
        raise RuntimeError('W must have a unit innermost stride (it is updated in place)')
    return [_lib.unit_inner(t) for t in (Q, K, V, beta)] + [W]


class DeltaFastWeight(torch.autograd.Function):
    """Fast weight using the delta update rule.  The forward, the autograd node and the backward are native
    (csrc/binding/fwp_torch.cpp); ``apply`` is the entry point."""

    apply = staticmethod(_lib.entry_point('fast_weight_delta', _normalise))


# Alias the autograd function to the reference's snake-case name
fast_weight_delta = DeltaFastWeight.apply
