"""Values that are not finite reach what depends on them and nothing else: in the chunkwise split-product plans (csrc/fwp_delta_wy.cuh,
csrc/fwp_delta_phases.cuh, csrc/fwp_sum_wy.cu) outputs of earlier steps of the same chunk, other value columns, other sequences
and gradients of later steps stay as the recurrence has them.  Expected: the recurrence in fp32 (oracle/kernels.py); which
entries are finite must agree exactly, and their values to the plans' accuracy."""
import math

import pytest
import torch

from oracle import kernels as K
from tests import util

pytestmark = pytest.mark.gpu
DEV = 'cuda:0'
INF, NAN = math.inf, math.nan
SIZES = [(16, 16), (9, 14), (32, 32), (20, 31), (48, 48), (50, 33), (96, 32), (77, 12), (32, 97), (128, 128)]
B, H, L = 2, 3, 45


def agree(got, ref, rel, what):
    """Same finite entries; values within ``rel`` of the largest entry of their step (1 at least)."""
    got, ref = got.float().cpu(), ref.float()
    assert torch.equal(got.isfinite(), ref.isfinite()), what
    zero = torch.zeros(())
    g, r = torch.where(ref.isfinite(), got, zero), torch.where(ref.isfinite(), ref, zero)
    assert ((g - r).abs() <= rel * r.abs().amax(-1, keepdim=True).clamp_min(1.)).all(), what


def forward(rule, x, W, plan):
    """The C entry point: y, W, v_old, v_insert."""
    from recurrent_fwp_b200 import _lib
    D = _lib.desc
    q, v = x[0], x[2]
    N, h, l, E = q.shape
    M = v.shape[3]
    y = torch.empty(N, h, l, M, device=DEV, dtype=q.dtype)
    vo, vi = (torch.empty(N, h, l, M, device=DEV) for _ in range(2))
    W = W.clone()
    stream, dev = _lib.stream_and_device(q)
    code = _lib.io_dtype(q)
    try:
        for key, value in plan.items():
            _lib.tune(key, value)
        if rule == 'sum':
            _lib.check(_lib.lib.fwp_causal_dot_product(N, h, l, E, M, *map(D, x), D(W), D(y), code, stream, dev), 'forward')
            return y, W
        _lib.check(_lib.lib.fwp_fast_weight_forward(N, h, l, E, M, *map(D, x), D(vo), D(vi), D(W), D(y), code, stream, dev), 'forward')
        return y, W, vo, vi
    finally:
        assert _lib.last_kernel().startswith('delta_fwd_wy')
        _lib.tune('delta.wy', -1)
        _lib.tune('delta.wy.helpers', 0)


@pytest.mark.parametrize('E,M', SIZES)
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('name,value', [('v', NAN), ('v', INF), ('k', NAN), ('k', -INF), ('k', 1e25), ('q', INF), ('q', NAN), ('beta', NAN),
                                        ('W', NAN)])
def test_forward_is_causal_for_any_value(fwp, E, M, dtype, name, value):
    """One bad element at step 21 (chunk 2 of 3, row 5) of one sequence, or in its start state."""
    from recurrent_fwp_b200 import _lib
    q, k, v, b, _ = util.delta_inputs(71, B, H, L, E, M, dtype=dtype)
    W0 = torch.randn(B, H, E, M, generator=util.gen(72)) * 0.1
    clean = dict(q=q, k=k, v=v, beta=b, W=W0)
    bad = {n: t.clone() for n, t in clean.items()}
    bad[name][1, 2, 0 if name == 'W' else 21, 0 if name == 'beta' else 3] = value
    for rule in ('delta', 'sum'):
        if rule == 'sum' and name == 'beta':
            continue
        x = {'delta': ['q', 'k', 'v', 'beta'], 'sum': ['q', 'k', 'v']}[rule]
        refs = [torch.empty(B, H, L, M) for _ in range(3)]
        kv = bad['W'].clone()
        if rule == 'delta':
            K.fast_weight_forward(*[bad[n].float() for n in x], refs[1], refs[2], kv, refs[0])
            refs = [refs[0], kv] + refs[1:]
        else:
            K.causal_dot_product(*[bad[n].float() for n in x], kv, refs[0])
            refs = [refs[0], kv]
        for helpers in (2, 4, 6):
            plan = {'delta.wy': 1, 'delta.wy.helpers': helpers}
            got = forward(rule, [bad[n].to(DEV) for n in x], bad['W'].to(DEV), plan)
            assert _lib.last_kernel() == ('delta_fwd_wy_few_kernel' if util.few_form(rule, E, M, dtype, helpers) else 'delta_fwd_wy_kernel')
            ref = forward(rule, [clean[n].to(DEV) for n in x], W0.to(DEV), plan)
            for i, (a, c, r) in enumerate(zip(got, ref, refs)):
                # bf16 outputs are rounded to 8 bits; everything else is fp32 on both sides, sums in another order
                agree(a, r, 2 ** -8 if i == 0 and dtype == torch.bfloat16 else 1e-5, (rule, helpers, i))
                a, c = (t.clone() for t in (a, c))
                a[1, 2], c[1, 2] = 0, 0
                assert torch.equal(a, c), (rule, helpers, i)


@pytest.mark.parametrize('E,M', SIZES)
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('name,value', [('gy', NAN), ('gy', INF), ('v', NAN), ('beta', NAN), ('k', INF), ('q', NAN)])
def test_three_launch_backward_is_causal_for_any_value(fwp, E, M, dtype, name, value):
    from recurrent_fwp_b200 import _lib
    q, k, v, b, gy = util.delta_inputs(73, B, H, L, E, M, dtype=dtype)
    W0 = torch.randn(B, H, E, M, generator=util.gen(74)) * 0.1
    x = dict(q=q, k=k, v=v, beta=b, gy=gy)
    x[name][1, 2, 21, 0 if name == 'beta' else 3] = value
    f = [x[n].float() for n in ('q', 'k', 'v', 'beta', 'gy')]
    y, vo, vi = (torch.empty(B, H, L, M) for _ in range(3))
    kv = W0.clone()
    K.fast_weight_forward(*f[:4], vo, vi, kv, y)
    refs = [torch.empty_like(t) for t in f[:4]]
    K.fast_weight_backward(*f[:4], vo, vi, f[4], kv, *refs)
    leaves = [x[n].to(DEV).requires_grad_() for n in ('q', 'k', 'v', 'beta')]
    seen = []
    try:
        _lib.tune('delta.wy', 1)
        _lib.tune('delta_bwd.phases', 1)
        out = fwp.fast_weight_delta(*leaves, W0.to(DEV))
        leaves[0].register_hook(lambda g: seen.append(_lib.last_kernel()))
        out.backward(x['gy'].to(DEV))
    finally:
        _lib.tune('delta.wy', -1)
        _lib.tune('delta_bwd.phases', -1)
    assert seen == ['delta_bwd_finish_kernel']
    for n, leaf, ref in zip('qkvb', leaves, refs):
        agree(leaf.grad, ref, 2 ** -8 if dtype == torch.bfloat16 else 1e-5, n)


def test_three_launch_backward_in_segments_is_causal(fwp):
    """A workspace of several segments: the bad steps lie in the last, the first and no segment of their sequences."""
    from recurrent_fwp_b200 import _lib
    N, h, l, d = 160, 8, 100, 64
    q, k, v, b, gy = (t.to(DEV) for t in util.delta_inputs(75, N, h, l, d))
    gy[3, 1, 97, 5] = NAN
    gy[4, 2, 2, 6] = INF
    W0 = torch.zeros(N, h, d, d, device=DEV)
    res = {}
    try:
        _lib.tune('delta.wy', 0)
        for plan in (0, 1):
            _lib.tune('delta_bwd.phases', plan)
            x = [t.clone().requires_grad_() for t in (q, k, v, b)]
            W = W0.clone()
            fwp.fast_weight_delta(*x, W).backward(gy)
            res[plan] = [t.grad for t in x] + [W]
    finally:
        _lib.tune('delta.wy', -1)
        _lib.tune('delta_bwd.phases', -1)
    for i, (a, c) in enumerate(zip(res[1], res[0])):
        agree(a, c.cpu(), 1e-5, i)


@pytest.mark.parametrize('E,M', [(16, 16), (9, 14), (32, 32), (48, 48), (50, 33), (64, 64)])
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('l', [45, 130])
@pytest.mark.parametrize('name,value', [('gy', NAN), ('v', INF), ('k', NAN), ('q', INF)])
def test_sum_rule_backward_is_causal_for_any_value(fwp, E, M, dtype, l, name, value):
    from recurrent_fwp_b200 import _lib
    q, k, v, _, gy = util.delta_inputs(77, B, H, l, E, M, dtype=dtype)
    x = dict(q=q, k=k, v=v, gy=gy)
    x[name][1, 2, 21, 3] = value
    f = [x[n].float() for n in ('q', 'k', 'v', 'gy')]
    refs = [torch.empty_like(t) for t in f[:3]]
    K.causal_dot_backward(*f, *refs)
    leaves = [x[n].to(DEV).requires_grad_() for n in ('q', 'k', 'v')]
    seen = []
    try:
        _lib.tune('sum_bwd.roles', 2)
        out = fwp.fast_weight_sum(*leaves, torch.zeros(B, H, E, M, device=DEV))
        leaves[0].register_hook(lambda g: seen.append(_lib.last_kernel()))
        out.backward(x['gy'].to(DEV))
    finally:
        _lib.tune('sum_bwd.roles', -1)
    assert len(seen) == 1 and seen[0].startswith('sum_bwd_wy')
    for n, leaf, ref in zip('qkv', leaves, refs):
        agree(leaf.grad, ref, 2 ** -8 if dtype == torch.bfloat16 else 1e-5, n)
