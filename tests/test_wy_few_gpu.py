"""The forward for few sequences (``delta_fwd_wy_few_kernel``) above d = 16 against the per-step or shared-memory kernels.

Row forms that its staging copies tell apart (whole rows, rows of whole 16-byte pieces, rows at odd offsets), head sizes at and
beside its instances, and lengths on both sides of sixteen steps and of its helpers' turns.  Both sides are fp32 with sums in another
order: 2e-6 of the largest value is what the split products are held to elsewhere; the reference adds its own rounding, 1e-5."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu
DEV = 'cuda:0'


def run(ins, W0, grad):
    from recurrent_fwp_b200 import _lib, fast_weight_delta
    leaves = [t.detach().requires_grad_(grad) for t in ins]
    W = W0.clone()
    y = fast_weight_delta(*leaves, W)
    return y.detach(), W, _lib.last_kernel()


@pytest.mark.parametrize('E,M,L,form,few', [(32, 32, 112, 'packed', True), (20, 20, 113, 'views', True), (17, 25, 127, 'packed', True),
                                            (24, 32, 240, 'offset', True), (32, 32, 111, 'packed', False), (96, 32, 144, 'views', 'forced'),
                                            (80, 29, 161, 'packed', 'forced'), (77, 32, 150, 'offset', 'forced'), (65, 16, 145, 'packed', True),
                                            (96, 32, 143, 'packed', False), (97, 32, 160, 'packed', False)])
def test_few_sequences(fwp, E, M, L, form, few):
    from recurrent_fwp_b200 import _lib
    B, H = 2, 3
    *ins, _ = util.delta_inputs(81, B, H, L, E, M)
    W0 = (torch.randn(B, H, E, M, generator=util.gen(82)) * 0.1).to(DEV)

    def lay_out(t):
        t = t.to(DEV)
        if form == 'views':
            return t.permute(2, 0, 1, 3).contiguous().permute(1, 2, 0, 3)
        if form == 'offset':
            wide = torch.zeros(*t.shape[:-1], t.shape[-1] + 1, device=DEV)
            wide[..., 1:].copy_(t)
            return wide[..., 1:]
        return t
    ins = [lay_out(t) for t in ins]
    try:                        # so few sequences take it by themselves up to 16 values only
        _lib.tune('delta.wy.helpers', 6 if few == 'forced' else 0)
        y, W, kf = run(ins, W0, True)
    finally:
        _lib.tune('delta.wy.helpers', 0)
    assert (kf == 'delta_fwd_wy_few_kernel') == bool(few)
    try:
        _lib.tune('delta.wy', 0)
        yr, Wr, kr = run(ins, W0, False)
    finally:
        _lib.tune('delta.wy', -1)
    assert 'wy' not in kr
    for a, r in ((y, yr), (W, Wr)):
        assert (a - r).abs().max().item() <= 1e-5 * r.abs().max().item()


@pytest.mark.parametrize('E,M,n,L,few', [(96, 32, 111, 144, True), (96, 32, 110, 144, False), (77, 20, 6, 384, False), (96, 16, 6, 144, True),
                                         (24, 24, 6, 112, False), (24, 24, 6, 113, True), (32, 32, 149, 160, False)])
def test_where_it_is_taken(fwp, E, M, n, L, few):
    """By the numbers of a B200's SMs (148): up to one sequence each, from three quarters of them on where M is above 16."""
    *ins, _ = (t.to(DEV) for t in util.delta_inputs(83, n, 1, L, E, M))
    _, _, kf = run(ins, torch.zeros(n, 1, E, M, device=DEV), False)
    assert kf == ('delta_fwd_wy_few_kernel' if few else 'delta_fwd_wy_kernel')
