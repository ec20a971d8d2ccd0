"""The four-warp step-by-step backward at E = M = 32 (``delta_bwd_tile32_kernel``) against the per-step kernels and fp64.

Counts that put one, two and four sequences on an SM, lengths on both sides of its chunks of eight steps (it starts at 17), and rows
in every form it accepts: packed, views of a (L, B, H, d) tensor, rows that are not 16-byte aligned.  Both kernels are fp32 and
differ in the order of their sums of 32 terms over at most L steps: 2e-5 of a tensor's scale, the bound of the other plans' tests."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu
DEV = 'cuda:0'
D = 32
TOL = 2e-5


def close(a, b):
    return (a.double() - b.double()).abs().max().item() <= TOL * max(b.abs().max().item(), 1e-6)


def lay_out(t, form):
    if form == 'views':         # (L, B, H, d) underneath
        return t.permute(2, 0, 1, 3).contiguous().permute(1, 2, 0, 3)
    if form == 'offset':        # rows 4 bytes off a 16-byte boundary
        wide = torch.zeros(*t.shape[:-1], t.shape[-1] + 1, device=t.device)
        wide[..., 1:].copy_(t)
        return wide[..., 1:]
    return t.clone()


def run(ins, gy, W0, form):
    from recurrent_fwp_b200 import _lib, fast_weight_delta
    leaves = [lay_out(t.to(DEV), form).requires_grad_() for t in ins]
    W, kb = W0.clone().to(DEV), []
    y = fast_weight_delta(*leaves, W)
    leaves[0].register_hook(lambda g: kb.append(_lib.last_kernel()))
    y.backward(lay_out(gy.to(DEV), form))
    return [t.grad for t in leaves] + [W], kb[0]


@pytest.mark.parametrize('B,H,L,form', [(1, 1, 17, 'packed'), (1, 3, 23, 'offset'), (74, 4, 24, 'packed'), (74, 4, 25, 'views'), (111, 4, 31, 'packed'),
                                        (111, 4, 18, 'offset'), (148, 4, 33, 'views'), (5, 8, 95, 'packed')])
def test_four_warp_backward(fwp, B, H, L, form):
    from recurrent_fwp_b200 import _lib
    *ins, gy = util.delta_inputs(71, B, H, L, D)
    W0 = torch.randn(B, H, D, D, generator=util.gen(72)) * 0.1
    got, kb = run(ins, gy, W0, form)
    try:
        _lib.tune('delta.blocked', 0)
        ref, kr = run(ins, gy, W0, form)
    finally:
        _lib.tune('delta.blocked', -1)
    assert kb == 'delta_bwd_tile32_kernel' and kr == 'delta_bwd_step_kernel'
    for a, r in zip(got, ref):
        assert close(a, r)
    # and the recurrence in fp64 on the first sequences
    q, k, v, b, g64 = (t[:1].double() for t in (*ins, gy))
    W = W0[:1].double()
    leaves = [t.clone().requires_grad_() for t in (q, k, v, b)]
    y, S = [], W
    for t in range(L):
        kt, qt = leaves[1][:, :, t], leaves[0][:, :, t]
        u = leaves[3][:, :, t] * (leaves[2][:, :, t] - torch.einsum('nhem,nhe->nhm', S, kt))
        S = S + torch.einsum('nhe,nhm->nhem', kt, u)
        y.append(torch.einsum('nhem,nhe->nhm', S, qt))
    grads = torch.autograd.grad(torch.stack(y, 2), leaves, g64)
    for a, r in zip(got, grads):
        assert close(a[:1].cpu(), r)


@pytest.mark.parametrize('B,H,L,form,tile', [(1, 4, 88, 'packed', True), (1, 4, 89, 'packed', False), (5, 8, 96, 'packed', False),
                                             (5, 8, 256, 'packed', False), (7, 8, 160, 'packed', True), (1, 4, 72, 'offset', True),
                                             (1, 4, 73, 'offset', False), (9, 8, 112, 'offset', False), (10, 8, 160, 'offset', True)])
def test_few_long_sequences_take_the_three_launches(fwp, B, H, L, form, tile):
    """Up to 3/8 (rows off a 16-byte boundary: half) as many sequences as the SMs of a B200, from the length on where they win."""
    *ins, gy = util.delta_inputs(73, B, H, L, D)
    W0 = torch.randn(B, H, D, D, generator=util.gen(74)) * 0.1
    got, kb = run(ins, gy, W0, form)
    assert kb == ('delta_bwd_tile32_kernel' if tile else 'delta_bwd_finish_kernel')
    assert (got[-1].cpu() - W0).abs().max().item() <= 1e-5      # rewound
