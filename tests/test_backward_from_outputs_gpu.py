"""The d = 32 backward entry points in their two forms: over delayed tensors that the caller made, and from the outputs that the
forward left (``..._from_outputs``).  Both run the same kernels on the same numbers, so they agree bit for bit; where no
kernel takes the outputs, nothing is launched and nothing is written."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu
DEV = 'cuda:0'
D = 32
NULL, UNSUPPORTED = 1, 6


class Call:
    """One forward through the C entry points, and its backward in both forms."""

    def __init__(self, op, B, H, L, d, offset=False):
        from recurrent_fwp_b200 import _lib
        self.lib, self.desc, self.desc3, self.delayed = _lib.lib, _lib.desc, _lib.desc3, _lib.delayed
        self.op, self.dims, self.variant = op, (B, H, L, d), int(op[-1]) if op.startswith('lstm') else 0
        self.new = lambda w: torch.empty(B, H, L, w, device=DEV)
        g = util.gen(91)
        start = lambda: (torch.randn(B, H, 1, d, generator=g) * .5).to(DEV)
        memory = lambda: (torch.randn(B, H, d, d, generator=g) * .1).to(DEV)
        wide = (util.rec_inputs if op == 'rec' else util.rnn_inputs)(92, B, H, L, d)[-1].to(DEV)
        self.gy = torch.cat([wide, wide], -1)[..., 1:d + 1] if offset else wide
        self.h0, self.c0 = start(), start()
        self.stream = _lib.stream_and_device(self.gy)
        self.out, h = self.new(d), self.h0.clone()
        T, T3, new = self.desc, self.desc3, self.new
        if op == 'rec':
            *ins, _ = (t.to(DEV) for t in util.rec_inputs(92, B, H, L, d))
            self.R, self.W = ins[4:], [memory()]
            self.saved = [new(d), new(d), new(d), new(1), new(d)]
            f, a = 'fwp_rec_update_fwm_tanh_forward', [*ins, *self.saved, h, self.W[0], self.out]
            args = [T(x) for x in a]
        elif op == 'rnn1':
            z, k, v, b, _ = (t.to(DEV) for t in util.rnn_inputs(92, B, H, L, d))
            self.W, self.saved = [memory()], [k, v, b, new(d)]
            f, args = 'fwp_fast_rnn_forward', [T(x) for x in (z, k, v, b, self.saved[3], h, self.W[0], self.out)]
        else:
            gates = [[t.to(DEV) for t in gate] for gate in util.lstm_inputs(92, B, H, L, d)[0]]
            z, k, v, b = zip(*gates)
            self.W, c = [memory() for _ in range(3)], self.c0.clone()
            self.normalised, self.cell = new(d), new(d)
            self.gates, v_old = [new(d) for _ in range(3)], [new(d) for _ in range(3)]
            self.saved = [k, v, b, v_old]
            f = 'fwp_fast_lstm_forward'
            args = [T3(z), T3(k), T3(v), T3(b), T(h), T(c), T3(self.W), T(self.out), T(self.normalised), T(self.cell), T3(self.gates), T3(v_old)]
        self.call(f, args)

    def call(self, name, args):
        lead = ([self.variant] if self.variant else []) + list(self.dims)
        rc = getattr(self.lib, name)(*lead, *args, 0, *self.stream)
        assert rc == 0 or name.endswith('_from_outputs'), (name, rc)
        return rc

    def backward(self, from_outputs, start=True, c0=True):
        """(status, memories, gradients); gradients start as 7."""
        B, H, L, d = self.dims
        T, T3 = self.desc, self.desc3
        suffix = '_from_outputs' if from_outputs else ''
        W = [w.clone() for w in self.W]
        h0, c0 = self.h0 if start else None, self.c0 if c0 else None
        full = lambda *s: torch.full(s, 7., device=DEV)
        if self.op == 'rec':
            grads = [full(B, H, L, w) for w in (d, d, d, 1)] + [full(1, H, d, d) for _ in range(3)] + [full(1, H, 1, d)]
            n = self.lib.fwp_rec_update_fwm_tanh_scratch_floats(B, H, d)
            scratch = torch.empty(n, device=DEV)
            fed = [self.out, h0] if from_outputs else [self.delayed(self.out, self.h0, 1)]
            args = [T(x) for x in (*self.saved, *fed, self.gy, *self.R, W[0], *grads)]
            import ctypes
            rc = self.call('fwp_rec_update_fwm_tanh_backward' + suffix,
                           args + [ctypes.cast(scratch.data_ptr(), ctypes.POINTER(ctypes.c_float)), n])
        elif self.op == 'rnn1':
            grads = [full(B, H, L, w) for w in (d, d, d, 1)]
            fed = h0 if from_outputs else self.delayed(self.out, self.h0)
            rc = self.call('fwp_fast_rnn_backward' + suffix, [T(x) for x in (*self.saved, self.gy, self.out, fed, W[0], *grads)])
        else:
            k, v, b, v_old = self.saved
            grads = [[full(B, H, L, w) for _ in range(3)] for w in (d, d, d, 1)]
            if from_outputs:
                fed, cells = (h0 if self.variant == 1 else self.normalised if start else None), c0
            else:
                fed = self.delayed(self.out, self.h0) if self.variant == 1 else self.normalised
                cells = self.delayed(self.cell, self.c0, 0, self.gates[1])
            rc = self.call('fwp_fast_lstm_backward' + suffix,
                           [T(self.gy), T3(k), T3(v), T3(b), T3(v_old), T(self.out), T(fed), T(self.cell), T(cells), T3(self.gates), T3(W),
                            *map(T3, grads)])
            grads = [x for g in grads for x in g]
        return rc, W, grads


OPS = ['rec', 'rnn1', 'lstm1', 'lstm2', 'lstm3', 'lstm4']


@pytest.mark.parametrize('op', OPS)
@pytest.mark.parametrize('B,H,L,offset', [(1, 3, 1, False), (2, 2, 8, False), (1, 3, 21, False), (1, 2, 70, True), (111, 4, 13, False),
                                          (74, 4, 9, False)])
def test_both_forms_agree_bit_for_bit(fwp, op, B, H, L, offset):
    from recurrent_fwp_b200 import _lib
    call = Call(op, B, H, L, D, offset)
    results = []
    for from_outputs in (False, True):
        before = _lib.launch_count()
        results.append(call.backward(from_outputs))
        assert results[-1][0] == 0
        if from_outputs:        # the recurrent delta net adds its parameter gradients up in a kernel of its own
            assert _lib.launch_count() - before == (2 if op == 'rec' else 1)
    (_, W, grads), (_, W2, grads2) = results
    for a, b in zip(W + grads, W2 + grads2):
        assert torch.equal(a, b)


@pytest.mark.parametrize('op', OPS)
@pytest.mark.parametrize('case', ['size', 'rows', 'switch', 'start', 'cell'])
def test_outputs_that_no_kernel_takes_launch_nothing(fwp, op, case):
    from recurrent_fwp_b200 import _lib
    if case == 'cell' and not op.startswith('lstm'):
        pytest.skip('the LSTM alone has a cell')
    call = Call(op, 1, 2, 20, 16 if case == 'size' else D, offset=case == 'rows')
    key = {'rec': 'rec_bwd.32.roles', 'rnn1': 'rnn_bwd.32.roles'}.get(op, 'lstm_bwd.32.roles')
    try:
        if case == 'switch':
            _lib.tune(key, 0)
        before = _lib.launch_count()
        rc, W, grads = call.backward(True, start=case != 'start', c0=case != 'cell')
    finally:
        _lib.tune(key, 1)
    assert rc == (NULL if case in ('start', 'cell') else UNSUPPORTED)
    assert _lib.launch_count() == before
    assert all(torch.equal(a, b) for a, b in zip(W, call.W)) and all((g == 7).all() for g in grads)
