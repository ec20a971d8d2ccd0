"""The workspace of the three-launch backward (csrc/fwp_delta_phases.cu): bounded for every shape, and cut right where it is cut
into groups of sequences."""
import pytest
import torch

from tests import util

DEV = 'cuda:0'
BOUND = 64 << 20


@pytest.mark.parametrize('E,M', [(16, 16), (32, 32), (48, 48), (64, 64), (32, 112), (96, 16), (96, 32), (96, 64), (128, 16), (128, 32),
                                 (128, 64), (128, 128)])
@pytest.mark.parametrize('dtype', [0, 1])
def test_scratch_is_bounded(fwp, E, M, dtype):
    from recurrent_fwp_b200 import _lib
    try:
        _lib.tune('delta_bwd.phases', 1)
        for N in (1, 7, 148, 370, 371, 1024, 5000, 100000):
            for L in (1, 16, 17, 100, 4096, 1000003):
                need = _lib.lib.fwp_fast_weight_backward_scratch_floats(N, 1, L, E, M, dtype)
                assert 0 < 4 * need <= BOUND, (N, L)
    finally:
        _lib.tune('delta_bwd.phases', -1)


@pytest.mark.gpu
@pytest.mark.parametrize('B,H,L,E,M', [(76, 4, 40, 128, 128), (139, 4, 90, 96, 64), (150, 11, 17, 60, 60)])
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
def test_groups_of_sequences_meet_the_one_launch_kernels(fwp, B, H, L, E, M, dtype):
    """More sequences than one chunk's workspace holds, the last group smaller; one of them with a gradient that is not finite."""
    from recurrent_fwp_b200 import _lib
    q, k, v, b, gy = (t.to(DEV) for t in util.delta_inputs(91, B, H, L, E, M, dtype=dtype))
    gy[B - 2, 1, L // 2, 3] = float('nan')
    W0 = torch.randn(B, H, E, M, generator=util.gen(92)).to(DEV) * 0.1
    res = {}
    try:
        _lib.tune('delta.wy', 1)
        for plan in (0, 1):
            _lib.tune('delta_bwd.phases', plan)
            x = [t.clone().requires_grad_() for t in (q, k, v, b)]
            W = W0.clone()
            fwp.fast_weight_delta(*x, W).backward(gy)
            res[plan] = [t.grad.float() for t in x] + [W]
    finally:
        _lib.tune('delta.wy', -1)
        _lib.tune('delta_bwd.phases', -1)
    rel = 2 ** -7 if dtype == torch.bfloat16 else 1e-5      # both sides round bf16 gradients to 8 bits once
    for a, r in zip(res[1], res[0]):
        assert torch.equal(a.isfinite(), r.isfinite())
        a, r = a.nan_to_num(0, 0, 0), r.nan_to_num(0, 0, 0)
        assert ((a - r).abs() <= rel * r.abs().amax(-1, keepdim=True).clamp_min(1.)).all()


@pytest.mark.gpu
def test_a_device_without_room_for_the_workspace_runs_the_one_launch_kernel(fwp):
    """The allocator is held to what it has plus room for the gradients (three segments of 48 MB), not for 61 MB of workspace."""
    from recurrent_fwp_b200 import _lib
    B, H, L, E, M = 16, 8, 256, 96, 32
    q, k, v, b, gy = (t.to(DEV) for t in util.delta_inputs(95, B, H, L, E, M))
    runs = []
    for short in (False, True):
        x = [t.clone().requires_grad_() for t in (q, k, v, b)]
        y = fwp.fast_weight_delta(*x, torch.zeros(B, H, E, M, device=DEV))
        x[0].register_hook(lambda g: runs.append(_lib.last_kernel()))
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        try:
            if short:
                torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (56 << 20)) / total)
            y.backward(gy)
            torch.cuda.synchronize()
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        runs.append([t.grad for t in x])
    assert runs[0] == 'delta_bwd_finish_kernel' and runs[2] == 'delta_bwd_generic_kernel'
    for a, r in zip(runs[1], runs[3]):
        assert util.max_abs(a, r) <= 1e-5 * max(1., r.abs().max().item())
