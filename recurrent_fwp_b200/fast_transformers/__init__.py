"""Sum-rule causal product with carried state: drop-in for the reference's
``fast_transformers`` module (``FastWeightSum`` / ``fast_weight_sum``,
algorithmic/fast_transformers/__init__.py:25-84).

``W`` [N,H,E,M] is updated in place to the end-of-segment state.  As in the
reference, the backward takes no state: its prefix sums restart from zero, so a
carried non-zero ``W`` contributes nothing to ``grad_Q`` and ``W`` is not rewound.
"""
import torch

from recurrent_fwp_b200 import _lib


def _normalise(Q, K, V, W):
    N, H, L, E = Q.shape
    M = V.shape[3]
    _lib.io_dtype(Q)
    _lib.require_streams(Q, {'K': (K, (N, H, L, E)), 'V': (V, (N, H, L, M))})
    _lib.require_f32(Q, {'W': (W, (N, H, E, M))})
    _lib.require_cuda(Q, K, V, W)
    if M > 1 and W.stride(3) != 1:
        raise RuntimeError('W must have a unit innermost stride (it is updated in place)')
    return [_lib.unit_inner(t) for t in (Q, K, V)] + [W]


class FastWeightSum(torch.autograd.Function):
    """Fast weight using the purely additive (sum) update rule; native like the delta rule's."""

    apply = staticmethod(_lib.entry_point('fast_weight_sum', _normalise))


fast_weight_sum = FastWeightSum.apply
