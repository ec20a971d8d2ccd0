"""GPU parity of the recurrent delta net against the fp64 CPU oracle and the golden fixture.
Tolerances: outputs max-abs <= 1e-4; stream and parameter gradients through ``util.check_grads``
(scaled-rel <= 1e-3 vs fp64, strict element-wise measure above 4 x the fp32 CPU recurrence's own
noise floor, all figures recorded).  The reference's own threshold for this op is 1e-2, used on its
golden self-test case."""
import pytest
import torch

from oracle import kernels as K
from tests import util

pytestmark = pytest.mark.gpu
DEV = 'cuda:0'
NAMES = ('qx', 'kx', 'vx', 'bx', 'R_q', 'R_k', 'R_v', 'r_b')


def oracle64(ins, W0, h0, gy, dtype=torch.float64):
    """The explicit recurrences in ``dtype``: fp64 is the ground truth, fp32 the reference's own arithmetic."""
    ins = [t.to(dtype) for t in ins]
    N, H, L, d = ins[0].shape
    W, st = W0.to(dtype).clone(), h0.to(dtype).clone()
    z = lambda *s: torch.zeros(*s, dtype=dtype)
    qo, ko, vo_, out, vold = (z(N, H, L, d) for _ in range(5))
    bo = z(N, H, L, 1)
    K.rec_update_fwm_tanh_forward(*ins, qo, ko, vo_, bo, vold, st, W, out)
    W_end = W.clone()
    od = torch.tanh(torch.cat([h0.to(dtype), out[:, :, :-1]], 2))
    g = [torch.zeros_like(t) for t in ins]
    K.rec_update_fwm_tanh_backward(qo, ko, vo_, bo, vold, od, gy.to(dtype), *ins[4:8], W, *g)
    return out, g, W_end, st


@pytest.mark.parametrize('B,H,L,d', [(2, 3, 29, 32), (2, 2, 21, 16), (1, 2, 9, 64), (2, 2, 1, 32), (1, 2, 7, 18)])
def test_parity_vs_oracle(fwp, B, H, L, d):
    from recurrent_fwp_b200.rec_update_fwm_tanh import rec_update_fwm_tanh
    *ins, gy = util.rec_inputs(7, B, H, L, d)
    W0 = torch.randn(B, H, d, d, generator=util.gen(8)) * 0.1
    h0 = torch.randn(B, H, 1, d, generator=util.gen(9))
    leaves = [t.clone().to(DEV).requires_grad_() for t in ins]
    W, hs = W0.to(DEV), h0.to(DEV)
    y = rec_update_fwm_tanh(*leaves, W, hs)
    W_end = W.clone()
    y.backward(gy.to(DEV))
    out, g, S_end, st = oracle64(ins, W0, h0, gy)
    _, g32, _, _ = oracle64(ins, W0, h0, gy, torch.float32)
    assert util.max_abs(y, out) <= 1e-4
    assert util.max_abs(W_end, S_end) <= 1e-4 and util.max_abs(hs, st) <= 1e-4
    util.check_grads('rec_delta B%d H%d L%d d%d' % (B, H, L, d), NAMES, [l.grad for l in leaves], g32, g)
    assert util.max_abs(W, W0) <= 1e-5


def test_golden_reference_selftest_case(fwp):
    from recurrent_fwp_b200.rec_update_fwm_tanh import rec_update_fwm_tanh
    gd = util.golden('rec_delta')
    ins = [gd['in_' + n] for n in ('q0', 'k0', 'v0', 'beta0', 'R_q0', 'R_k0', 'R_v0', 'r_b0')]
    N, H, L, d = ins[0].shape
    leaves = [t.to(DEV).requires_grad_() for t in ins]
    y = rec_update_fwm_tanh(*leaves, torch.zeros(N, H, d, d, device=DEV), torch.zeros(N, H, 1, d, device=DEV))
    y.sum().backward()
    assert util.max_rel(y, gd['out_LBHd'].permute(1, 2, 0, 3)) < 1e-2
    for leaf, n in zip(leaves, ('q2', 'k2', 'v2', 'beta2', 'Rq2', 'Rk2', 'Rv2', 'rb2')):
        assert util.max_rel(leaf.grad, gd['grad_' + n]) < 1e-2


def test_config3_shape_slice_and_determinism(fwp):
    """configs[2] shape (B=64,H=8,L=256,d=32) on a batch slice; two runs must agree bit for bit
    (parameter gradients are reduced in a fixed order, not with atomics)."""
    from recurrent_fwp_b200.rec_update_fwm_tanh import rec_update_fwm_tanh
    B, H, L, d = 4, 8, 256, 32
    *ins, gy = util.rec_inputs(17, B, H, L, d)
    runs = []
    for _ in range(2):
        leaves = [t.clone().to(DEV).requires_grad_() for t in ins]
        y = rec_update_fwm_tanh(*leaves, torch.zeros(B, H, d, d, device=DEV), torch.zeros(B, H, 1, d, device=DEV))
        y.backward(gy.to(DEV))
        runs.append([y.detach()] + [l.grad for l in leaves])
    for a, b in zip(*runs):
        assert torch.equal(a, b)
    out, g, _, _ = oracle64(ins, torch.zeros(B, H, d, d), torch.zeros(B, H, 1, d), gy)
    out32, g32, _, _ = oracle64(ins, torch.zeros(B, H, d, d), torch.zeros(B, H, 1, d), gy, torch.float32)
    util.record('rec_delta recurrent-delta-net shape slice', y_cuda=util.max_abs(runs[0][0], out),
                y_cpu32=util.max_abs(out32, out))
    assert util.max_abs(runs[0][0], out) <= 1e-4
    util.check_grads('rec_delta recurrent-delta-net shape slice', NAMES, runs[0][1:], g32, g)


@pytest.mark.parametrize('L', [256, 4096])
def test_gradients_through_the_softmax_sum_to_zero(fwp, L):
    """Each step's gradients of q and k before their softmax sum to zero over the features up to the rounding of that sum, however long
    the sequence: the three-warp backward must not put the rewind's rounding there.  The general kernel sums the same 32 products in
    another order, so the largest sum of either is within a factor of two of the other's."""
    from recurrent_fwp_b200 import _lib
    from recurrent_fwp_b200.rec_update_fwm_tanh import rec_update_fwm_tanh
    B, H, d = 2, 4, 32
    *ins, gy = util.rec_inputs(2, B, H, L, d)
    W0 = torch.randn(B, H, d, d, generator=util.gen(52)) * 0.1
    h0 = torch.randn(B, H, 1, d, generator=util.gen(62)) * 0.1
    sums = {}
    try:
        for roles in (1, 0):
            _lib.tune('rec_bwd.32.roles', roles)
            leaves = [t.clone().to(DEV).requires_grad_() for t in ins]
            rec_update_fwm_tanh(*leaves, W0.to(DEV), h0.to(DEV)).backward(gy.to(DEV))
            sums[roles] = [leaf.grad.double().sum(-1).abs().amax().item() for leaf in leaves[:2]]
    finally:
        _lib.tune('rec_bwd.32.roles', 1)
    for fast, general in zip(sums[1], sums[0]):
        assert fast <= 2 * general, sums


@pytest.mark.parametrize('roles', [1, 0])
def test_delayed_output_enters_the_backward_by_an_accurate_tanh(fwp, roles):
    """With one step the gradient of r_b is tanh(h0) times the gradient of beta, one rounded product, so the tanh can be read off:
    2 ulp for tanhf as CUDA documents it and half an ulp for the product, an ulp being 2^-23 of the value at most."""
    from recurrent_fwp_b200 import _lib
    from recurrent_fwp_b200.rec_update_fwm_tanh import rec_update_fwm_tanh
    B, H, L, d = 1, 64, 1, 32
    *ins, gy = util.rec_inputs(3, B, H, L, d)
    W0 = torch.randn(B, H, d, d, generator=util.gen(4)) * 0.1
    h0 = torch.linspace(-3, 3, H * d).view(B, H, 1, d)
    leaves = [t.clone().to(DEV).requires_grad_() for t in ins]
    try:
        _lib.tune('rec_bwd.32.roles', roles)
        rec_update_fwm_tanh(*leaves, W0.to(DEV), h0.to(DEV)).backward(gy.to(DEV))
    finally:
        _lib.tune('rec_bwd.32.roles', 1)
    got = leaves[7].grad.double() / leaves[3].grad.double()
    want = torch.tanh(h0.double()).to(DEV)
    assert ((got - want) / want).abs().max().item() <= 2.5 * 2.0 ** -23
