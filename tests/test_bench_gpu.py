"""The benchmark's device-resident step runs the kernels that the public op runs at the same shape."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = 'cuda:0'


@pytest.mark.parametrize('B,H,L,d', [(2, 8, 256, 16), (64, 8, 256, 16), (4, 4, 100, 128)])
def test_bench_runs_the_backward_that_users_get(fwp, B, H, L, d):
    import bench
    from recurrent_fwp_b200 import _lib
    ds = bench.DeltaStep(B, H, L, d, 1, torch.float32, torch.device(DEV), seed=1)
    ds.step()
    q, k, v, b, gy = ds.inp[0]
    x = [t.clone().requires_grad_() for t in (q, k, v, b)]
    seen = []
    y = fwp.fast_weight_delta(*x, torch.zeros(B, H, d, d, device=DEV))
    seen.append(_lib.last_kernel())
    x[0].register_hook(lambda g: seen.append(_lib.last_kernel()))
    y.backward(gy)
    assert [ds.kernels['fwd'], ds.kernels['bwd']] == seen
    for a, r in zip(ds.g[0], x):
        assert torch.equal(a, r.grad)
