"""A delta-rule forward that no backward follows stores no old values: every kernel that can serve it gives the same
bits as when it stores them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = 'cuda:0'


@pytest.mark.parametrize('dtype,B,H,L,D,tune', [
    (torch.float32, 1, 2, 37, 16, {}), (torch.float32, 2, 3, 33, 32, {}), (torch.float32, 1, 2, 40, 64, {}),
    (torch.float32, 1, 2, 19, 128, {}), (torch.float32, 1, 2, 5, 24, {}), (torch.float32, 1, 3, 37, 16, {'delta.wy': (0, -1)}),
    (torch.float32, 1, 3, 37, 32, {'delta.wy': (0, -1)}), (torch.float32, 1, 3, 37, 64, {'delta.wy': (0, -1)}),
    (torch.bfloat16, 1, 3, 70, 64, {}), (torch.bfloat16, 2, 2, 65, 32, {}), (torch.bfloat16, 1, 3, 33, 128, {}),
    (torch.bfloat16, 1, 2, 70, 64, {'delta.pipe64': (0, 1)})])
def test_same_bits(fwp, dtype, B, H, L, D, tune):
    from recurrent_fwp_b200 import _lib
    g = torch.Generator(DEV).manual_seed(3)
    q, k, v = (torch.randn(B, H, L, D, device=DEV, generator=g).to(dtype) for _ in range(3))
    k = torch.softmax(k.float(), -1).to(dtype)
    beta = torch.sigmoid(torch.randn(B, H, L, 1, device=DEV, generator=g)).to(dtype)
    W1, W2 = torch.zeros(B, H, D, D, device=DEV), torch.zeros(B, H, D, D, device=DEV)
    try:
        for key, (value, _) in tune.items():
            _lib.tune(key, value)
        with torch.no_grad():
            y1 = fwp.fast_weight_delta(q, k, v, beta, W1)
        k1 = _lib.last_kernel()
        y2 = fwp.fast_weight_delta(q.requires_grad_(), k, v, beta, W2)
        k2 = _lib.last_kernel()
    finally:
        for key, (_, default) in tune.items():
            _lib.tune(key, default)
    assert k1 == k2 and torch.equal(y1, y2.detach()) and torch.equal(W1, W2)
