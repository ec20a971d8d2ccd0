"""Recurrent delta net: drop-in for the reference's ``rec_update_fwm_tanh`` module.

Mirrors ``FastWeightRecUpdateTanh`` / ``rec_update_fwm_tanh`` of
algorithmic/rec_update_fwm_tanh/__init__.py:31-139 (same file in language_modeling/src/utils
and reinforcement_learning/torchbeast): ``forward(ctx, qx, kx, vx, bx, R_q, R_k, R_v, r_b, W, h0)``.
The inputs are *pre-activations*: softmax on query/key, sigmoid on beta and the
``R . tanh(y_{t-1})`` feedback are applied inside the kernel.  ``W`` [N,H,d,d] and
``h0`` [N,H,1,d] are updated in place; backward rewinds ``W`` and returns gradients
for the four streams and the four recurrent parameters, ``None`` for W and h0.
"""
import torch

from recurrent_fwp_b200 import _lib


def _normalise(qx, kx, vx, bx, R_q, R_k, R_v, r_b, W, h0):
    N, H, L, E = qx.shape
    M = vx.shape[3]
    assert E == M, "Current kernel only support this case."
    assert R_q.shape == (1, H, M, M), "Reshape/unsqueeze if needed."
    assert R_k.shape == (1, H, M, M), "Reshape/unsqueeze if needed."
    assert R_v.shape == (1, H, M, M), "Reshape/unsqueeze if needed."
    assert r_b.shape == (1, H, 1, M), "Reshape/unsqueeze if needed."
    if qx.dtype != torch.float32:
        raise TypeError('the recurrent fast-weight kernels take float32 tensors')
    _lib.require_streams(qx, {'kx': (kx, (N, H, L, E)), 'vx': (vx, (N, H, L, M)), 'bx': (bx, (N, H, L, 1))})
    _lib.require_f32(qx, {'R_q': (R_q, (1, H, M, M)), 'R_k': (R_k, (1, H, M, M)), 'R_v': (R_v, (1, H, M, M)),
                          'r_b': (r_b, (1, H, 1, M)), 'W': (W, (N, H, E, M)), 'h0': (h0, (N, H, 1, M))})
    _lib.require_cuda(qx, kx, vx, bx, R_q, R_k, R_v, r_b, W, h0)
    if W.stride(3) != 1 or h0.stride(3) != 1:
        raise RuntimeError('W and h0 must have a unit innermost stride (they are updated in place)')
    return ([_lib.unit_inner(t) for t in (qx, kx, vx, bx)] + [t.contiguous() for t in (R_q, R_k, R_v, r_b)] + [W, h0])


class FastWeightRecUpdateTanh(torch.autograd.Function):
    """Delta-rule fast weight memory with tanh feedback from the previous output; native like the delta rule's."""

    apply = staticmethod(_lib.entry_point('rec_update_fwm_tanh', _normalise))


rec_update_fwm_tanh = FastWeightRecUpdateTanh.apply
