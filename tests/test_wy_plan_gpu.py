"""The chunkwise split-product plan of the delta and sum rules (csrc/fwp_delta_wy.cuh): every instance, at chunk remainders,
padded head sizes, layer-sliced streams with rows at odd offsets, and both ways of sharing the work between warps."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu
DEV = 'cuda:0'


def run(fwp, rule, x, W, plan):
    from recurrent_fwp_b200 import _lib
    try:
        for key, value in plan.items():
            _lib.tune(key, value)
        f = fwp.fast_weight_delta if rule == 'delta' else fwp.fast_weight_sum
        W = W.clone()
        with torch.no_grad():
            y = f(*x, W)
        return y, W, _lib.last_kernel()
    finally:
        _lib.tune('delta.wy', -1)
        _lib.tune('delta.wy.helpers', 0)


def sliced(x):
    """The same streams as transposed views of one (L, B, H, width) tensor, rows at odd element offsets."""
    p = torch.cat([t.permute(2, 0, 1, 3) for t in x], -1)
    return [t.permute(1, 2, 0, 3) for t in torch.split(p, [t.shape[3] for t in x], -1)]


@pytest.mark.parametrize('E,M', [(16, 16), (9, 14), (32, 32), (20, 31), (48, 48), (64, 64), (50, 33), (32, 97), (96, 16),
                                 (70, 32), (96, 64), (128, 16), (128, 20), (101, 64), (128, 128)])
@pytest.mark.parametrize('L', [1, 17, 130])
def test_forward_meets_the_oracle(fwp, E, M, L):
    B, H = 2, 3
    q, k, v, b, _ = util.delta_inputs(7, B, H, L, E, M)
    W0 = torch.randn(B, H, E, M, generator=util.gen(8)) * 0.1
    for rule in ('delta', 'sum'):
        x = [q, k, v] + ([b] if rule == 'delta' else [])
        S = W0.double().clone()
        ref = torch.empty(B, H, L, M, dtype=torch.float64)
        for t in range(L):
            kt, u = k[:, :, t].double(), v[:, :, t].double()
            if rule == 'delta':
                u = b[:, :, t].double() * (u - torch.einsum('bhem,bhe->bhm', S, kt))
            S = S + kt[..., None] * u[:, :, None]
            ref[:, :, t] = torch.einsum('bhem,bhe->bhm', S, q[:, :, t].double())
        dev = [t.to(DEV) for t in x]
        for streams in (dev, sliced(dev)):
            for helpers in (2, 4, 6):
                y, W, kernel = run(fwp, rule, streams, W0.to(DEV), {'delta.wy': 1, 'delta.wy.helpers': helpers})
                assert kernel == ('delta_fwd_wy_few_kernel' if util.few_form(rule, E, M, q.dtype, helpers) else 'delta_fwd_wy_kernel')
                # fp32 accuracy: three-part products keep every bit of the operands
                assert util.max_abs(y, ref) <= 2e-6 * max(1., ref.abs().max().item()), (rule, helpers)
                assert util.max_abs(W, S) <= 2e-6 * max(1., S.abs().max().item()), (rule, helpers)


@pytest.mark.parametrize('B,H,L,d', [(300, 1, 70, 16), (40, 8, 33, 32), (150, 2, 50, 64)])
def test_forward_with_more_sequences_than_the_gpu_holds(fwp, B, H, L, d):
    q, k, v, b, _ = (t.to(DEV) for t in util.delta_inputs(9, B, H, L, d))
    W0 = torch.randn(B, H, d, d, generator=util.gen(10)).to(DEV) * 0.1
    y, W, _ = run(fwp, 'delta', [q, k, v, b], W0, {'delta.wy': 0})
    for helpers in (0, 2, 4, 6):
        y2, W2, _ = run(fwp, 'delta', [q, k, v, b], W0, {'delta.wy': 1, 'delta.wy.helpers': helpers})
        assert util.max_abs(y, y2) <= 5e-6 and util.max_abs(W, W2) <= 5e-6
    from recurrent_fwp_b200 import _lib
    assert _lib.device_fault() == 0


@pytest.mark.parametrize('E,M', [(16, 16), (9, 14), (32, 32), (20, 31), (48, 48), (64, 64), (50, 33), (32, 97), (96, 16),
                                 (70, 32), (96, 64), (128, 16), (128, 20), (101, 64), (128, 128)])
@pytest.mark.parametrize('L', [5, 17, 130])
def test_three_launch_backward_meets_the_oracle(fwp, E, M, L):
    """csrc/fwp_delta_phases.cuh against autograd through the recurrence in fp64, packed and layer-sliced streams."""
    from recurrent_fwp_b200 import _lib
    B, H = 2, 3
    q, k, v, b, gy = util.delta_inputs(17, B, H, L, E, M)
    W0 = torch.randn(B, H, E, M, generator=util.gen(18)) * 0.1
    leaves = [t.double().requires_grad_() for t in (q, k, v, b)]
    S, ys = W0.double(), []
    for t in range(L):
        kt = leaves[1][:, :, t]
        u = leaves[3][:, :, t] * (leaves[2][:, :, t] - torch.einsum('bhem,bhe->bhm', S, kt))
        S = S + kt[..., None] * u[:, :, None]
        ys.append(torch.einsum('bhem,bhe->bhm', S, leaves[0][:, :, t]))
    torch.stack(ys, 2).backward(gy.double())
    dev = [t.to(DEV) for t in (q, k, v, b)]
    seen = []
    try:
        _lib.tune('delta_bwd.phases', 1)
        for streams in (dev, sliced(dev)):
            x = [t.detach().requires_grad_() for t in streams]
            W = W0.to(DEV)
            y = fwp.fast_weight_delta(*x, W)
            x[0].register_hook(lambda g: seen.append(_lib.last_kernel()))
            y.backward(gy.to(DEV))
            for got, ref in zip(x, leaves):
                assert util.max_abs(got.grad, ref.grad) <= 3e-6 * max(1., ref.grad.abs().max().item())
            assert util.max_abs(W, W0) <= 2e-6
    finally:
        _lib.tune('delta_bwd.phases', -1)
    assert seen == ['delta_bwd_finish_kernel'] * 2


def test_three_launch_backward_in_segments(fwp):
    """More chunks than one segment's workspace holds: G and the rewound state cross the segment borders."""
    from recurrent_fwp_b200 import _lib
    B, H, L, d = 160, 8, 100, 64
    q, k, v, b, gy = (t.to(DEV) for t in util.delta_inputs(23, B, H, L, d))
    W0 = torch.randn(B, H, d, d, generator=util.gen(24)).to(DEV) * 0.1
    res = {}
    try:
        for plan in (0, 1):
            _lib.tune('delta_bwd.phases', plan)
            x = [t.clone().requires_grad_() for t in (q, k, v, b)]
            W = W0.clone()
            fwp.fast_weight_delta(*x, W).backward(gy)
            res[plan] = [t.grad for t in x] + [W]
    finally:
        _lib.tune('delta_bwd.phases', -1)
    for a, c in zip(res[0], res[1]):
        assert util.max_abs(a, c) <= 5e-6 * max(1., a.abs().max().item())


@pytest.mark.parametrize('E,M', [(16, 16), (9, 14), (32, 32), (21, 30), (48, 48), (56, 33), (96, 64), (128, 128)])
@pytest.mark.parametrize('L', [17, 130])
def test_three_launch_backward_of_bf16_streams(fwp, E, M, L):
    """The gradients are the fp32 ones of the same bf16 values, rounded once."""
    from recurrent_fwp_b200 import _lib
    B, H = 2, 3
    x16 = [t.to(DEV).bfloat16() for t in util.delta_inputs(27, B, H, L, E, M)]
    W0 = torch.randn(B, H, E, M, generator=util.gen(28)).to(DEV) * 0.1
    res, seen = [], []
    try:
        _lib.tune('delta_bwd.phases', 1)
        for streams in (x16, sliced(x16[:4]) + x16[4:], [t.float() for t in x16]):
            x = [t.detach().requires_grad_() for t in streams[:4]]
            W = W0.clone()
            y = fwp.fast_weight_delta(*x, W)
            x[0].register_hook(lambda g: seen.append(_lib.last_kernel()))
            y.backward(streams[4])
            res.append([t.grad.float() for t in x] + [W])
    finally:
        _lib.tune('delta_bwd.phases', -1)
    assert seen == ['delta_bwd_finish_kernel'] * 3
    for got in res[:2]:
        for a, r in zip(got, res[2]):
            assert ((a - r).abs() <= 2 ** -8 * r.abs() + 1e-5 * r.abs().max()).all()


@pytest.mark.parametrize('E,M', [(16, 16), (9, 14), (32, 32), (20, 31), (48, 48), (64, 64), (50, 33)])
@pytest.mark.parametrize('B,H,L', [(2, 3, 1), (2, 3, 17), (2, 3, 130), (75, 2, 130)])
def test_sum_rule_backward_as_three_forwards(fwp, E, M, B, H, L):
    """csrc/fwp_sum_wy.cu: gradients against the sums they stand for in fp64, packed and layer-sliced streams."""
    from recurrent_fwp_b200 import _lib
    q, k, v, _, gy = util.delta_inputs(37, B, H, L, E, M)
    Q, K, V, G = (t.double().to(DEV) for t in (q, k, v, gy))
    lower = torch.tril(torch.ones(L, L, dtype=torch.float64, device=DEV))
    A = (G @ V.transpose(-1, -2)) * lower                     # gy_t . v_i
    P = (Q @ K.transpose(-1, -2)) * lower                     # q_t . k_i
    refs = [A @ K, A.transpose(-1, -2) @ Q, P.transpose(-1, -2) @ G]
    dev = [t.to(DEV) for t in (q, k, v)]
    seen = []
    try:
        _lib.tune('sum_bwd.roles', 2)
        for streams in (dev, sliced(dev)):
            for dtype in (torch.float32, torch.bfloat16):
                x = [t.detach().to(dtype).requires_grad_() for t in streams]
                y = fwp.fast_weight_sum(*x, torch.zeros(B, H, E, M, device=DEV))
                x[0].register_hook(lambda g: seen.append(_lib.last_kernel()))
                y.backward(gy.to(DEV).to(dtype))
                for got, ref in zip(x, refs):
                    tol = 3e-6 if dtype == torch.float32 else 2e-2
                    assert util.max_abs(got.grad.float(), ref) <= tol * max(1., ref.abs().max().item())
    finally:
        _lib.tune('sum_bwd.roles', -1)
    assert len(seen) == 4 and all(s.startswith('sum_bwd_wy') for s in seen)
    assert _lib.device_fault() == 0
