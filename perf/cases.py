"""Workloads for measuring the framework: what a training step, an evaluation pass or an acting step asks of it.

A case is one call pattern of a public op.  Its keys:

  op        delta, layer (``delta_attention``: prologue, delta rule, epilogue), sum, rec (recurrent delta net),
            rnn1, rnn2, lstm1 ... lstm4
  mode      train: forward and backward through autograd; eval: forward under no_grad;
            step: forward under no_grad, the memory carried in place from call to call (acting)
  B H L E M batch, heads, steps, key size, value size (E == M for the recurrent ops)
  dtype     fp32 or bf16 streams; the memory is fp32 either way
  layout    packed: every stream a contiguous (B, H, L, d) tensor of its own;
            sliced: what the layers hand over -- transposed views of a (L, B, H, width) projection, rows of
            d elements at odd offsets where the layer passes a slice as it is
  segments  consecutive segments of one sequence, the memory handed on as a clone between them
"""
import math

import torch
import torch.nn.functional as F

from recurrent_fwp_b200.delta_layer_io import delta_attention
from recurrent_fwp_b200.fast_lstm import fast_lstm
from recurrent_fwp_b200.fast_lstm_v2 import fast_lstm_v2
from recurrent_fwp_b200.fast_lstm_v3 import fast_lstm_v3
from recurrent_fwp_b200.fast_lstm_v4 import fast_lstm_v4
from recurrent_fwp_b200.fast_transformers import fast_weight_sum
from recurrent_fwp_b200.fast_weight import fast_weight_delta
from recurrent_fwp_b200.fast_weight_rnn import fast_rnn
from recurrent_fwp_b200.fast_weight_rnn_v2 import fast_rnn_v2
from recurrent_fwp_b200.rec_update_fwm_tanh import rec_update_fwm_tanh

LSTM = {'lstm1': fast_lstm, 'lstm2': fast_lstm_v2, 'lstm3': fast_lstm_v3, 'lstm4': fast_lstm_v4}
DTYPE = {'fp32': torch.float32, 'bf16': torch.bfloat16}


def _case(op, mode, B, H, L, E, M=None, dtype='fp32', layout='packed', segments=1, **name):
    return dict(name, op=op, mode=mode, B=B, H=H, L=L, E=E, M=E if M is None else M, dtype=dtype, layout=layout,
                segments=segments)


def listed():
    return [
        # acting in an environment: one step for each of 32 environments, 4 heads of 32, memory carried in place
        _case('delta', 'step', 32, 4, 1, 32, name='act_step'),
        # the smallest training call: two sequences of the language-model recipe
        _case('delta', 'train', 2, 8, 256, 16, name='delta_small'),
        # the language-model training step: 64 sequences, four carried segments of 256 steps
        _case('delta', 'train', 64, 8, 256, 16, segments=4, name='delta_lm'),
        # one attention layer of the 16-layer language model, forward and backward from its fused projection
        _case('layer', 'train', 32, 8, 512, 32, layout='sliced', name='delta_layer'),
        # evaluation of a short last batch with a segment length and a head size that fit no tile
        _case('delta', 'eval', 5, 8, 243, 20, layout='sliced', name='delta_eval_odd'),
        # a kernel feature map three times as wide as the values (E = 2 * n_roll * d)
        _case('delta', 'train', 16, 8, 256, 96, 32, layout='sliced', name='delta_wide'),
        # scale-out training: bf16 streams, 4096 sequences of 4096 steps
        _case('delta', 'train', 256, 16, 4096, 64, dtype='bf16', name='delta_long'),
        # long sequences at a small batch: fewer sequences than the machine has SMs
        _case('delta', 'train', 8, 16, 4096, 64, dtype='bf16', name='delta_few'),
        # the additive rule at the language-model training shape
        _case('sum', 'train', 64, 8, 256, 16, name='sum_lm'),
        # recurrent delta net, its training benchmark
        _case('rec', 'train', 64, 8, 256, 32, name='rec_delta'),
        # delta RNN as its layer calls it: keys from a softmax, values a slice of the projection
        _case('rnn2', 'train', 128, 4, 512, 32, layout='sliced', name='rnn_v2'),
        # delta LSTM, its training benchmark
        _case('lstm1', 'train', 128, 4, 512, 32, name='lstm_v1'),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: an op, then sizes over the range it is used in (acting, training, evaluation)."""
    kind = rng.choice(['step', 'delta', 'delta', 'layer', 'wide', 'long', 'long', 'sum', 'rec', 'rnn', 'lstm'])
    layout = rng.choice(['packed', 'sliced'])
    mode = rng.choice(['train', 'train', 'eval'])
    H = rng.choice([4, 8, 16])
    d = rng.choice([16, 16, 32, 32, 64, rng.randrange(9, 64)])
    if kind == 'step':      # acting: a few to many environments, one step per call
        return _case(rng.choice(['delta', 'rec', 'rnn2', 'lstm1']), 'step', _log(rng, 1, 256), 4, 1,
                     rng.choice([16, 32, 64]), layout=layout)
    if kind == 'delta':     # language-model and algorithmic training recipes
        return _case('delta', mode, _log(rng, 1, 96), H, _log(rng, 16, 1024), d, layout=layout,
                     segments=rng.choice([1, 2, 4]))
    if kind == 'layer':
        return _case('layer', mode, _log(rng, 1, 96), H, _log(rng, 16, 512), rng.choice([16, 32, 64]), layout='sliced')
    if kind == 'wide':      # kernel feature maps wider than the values, delta-delta's values wider than the keys
        E, M = rng.randrange(66, 129), rng.choice([16, 32, 64])
        if rng.random() < 0.3:
            E, M = 32, 97
        return _case('delta', mode, _log(rng, 1, 64), H, _log(rng, 16, 384), E, M, layout=layout)
    if kind == 'long':      # bf16 streams over long sequences, from one sequence per head up to the scale-out batch
        return _case('delta', mode, _log(rng, 1, 256), 16, _log(rng, 64, 4096), rng.choice([32, 64, 64, 64]), dtype='bf16',
                     layout='packed')
    if kind == 'sum':
        return _case('sum', mode, _log(rng, 1, 96), H, _log(rng, 16, 512), d, dtype=rng.choice(['fp32', 'fp32', 'bf16']),
                     layout=layout)
    op = {'rec': 'rec', 'rnn': rng.choice(['rnn1', 'rnn2', 'rnn2']), 'lstm': rng.choice(sorted(LSTM))}[kind]
    return _case(op, mode, _log(rng, 1, 128), rng.choice([4, 8]), _log(rng, 16, 512), rng.choice([16, 32, 32, 64, d]),
                 layout=layout)


def _phi(x):
    x = F.elu(x) + 1.
    return x / x.sum(-1, keepdim=True)


def _streams(g, case, widths):
    """N(0,1) streams of the given widths: tensors of their own, or slices of one projection as the layers cut them."""
    B, H, L = case['B'], case['H'], case['L']
    if case['layout'] == 'packed':
        return [torch.randn(B, H, L, w, generator=g, device='cuda') for w in widths]
    x = torch.randn(L, B, H, sum(widths), generator=g, device='cuda')
    return [t.permute(1, 2, 0, 3) for t in torch.split(x, widths, -1)]


def _inputs(g, case):
    """The streams of one segment in the op's argument order, with the incoming gradient last."""
    op, B, H, L, E, M = (case[k] for k in ('op', 'B', 'H', 'L', 'E', 'M'))
    dt = DTYPE[case['dtype']]
    if op == 'layer':
        return [torch.randn(L, B, H, 3 * E + 1, generator=g, device='cuda'),
                torch.randn(L, B, H * E, generator=g, device='cuda')]
    gy = torch.randn(B, H, L, M, generator=g, device='cuda')
    if case['layout'] == 'sliced':      # the layers' output path ends in a (L, B, H * M) tensor
        gy = gy.permute(2, 0, 1, 3).contiguous().permute(1, 2, 0, 3)
    if op in ('delta', 'sum'):
        q, k, v, b = _streams(g, case, [E, E, M, 1])
        s = [_phi(q).to(dt), _phi(k).to(dt), v.to(dt)] + ([torch.sigmoid(b).to(dt)] if op == 'delta' else [])
    elif op == 'rec':
        s = _streams(g, case, [E, E, E, 1])
    else:
        n = 3 if op in LSTM else 1
        s = []
        for z, k, v, b in (_streams(g, case, [E, E, E, 1]) for _ in range(n)):
            # the layers feed z from another op's output, a contiguous tensor
            s += [z.contiguous(), torch.softmax(k, -1), v, torch.sigmoid(b)]
    return s + [gy.to(dt)]


def prepare(case, seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    op, B, H, E, M = (case[k] for k in ('op', 'B', 'H', 'E', 'M'))
    train = case['mode'] == 'train'
    segments = []
    for _ in range(case['segments']):
        *streams, gy = _inputs(g, case)
        segments.append(([t.detach().requires_grad_(train) for t in streams], gy))
    n = 3 if op in LSTM else 1
    mem = [torch.randn(B, H, E, M, generator=g, device='cuda') * 0.1 for _ in range(n)]
    if op not in ('delta', 'layer', 'sum'):     # the last output, and the cell of the LSTM
        mem += [torch.randn(B, H, 1, M, generator=g, device='cuda') * 0.1 for _ in range(2 if op in LSTM else 1)]
    weights = []
    if op == 'rec':
        weights = [(torch.randn(s, generator=g, device='cuda') / math.sqrt(E)).requires_grad_(train)
                   for s in [(1, H, E, E)] * 3 + [(1, H, 1, E)]]
    return dict(op=op, mode=case['mode'], segments=segments, mem=mem, weights=weights, scale=1. / math.sqrt(E))


def _call(s, x, mem):
    op = s['op']
    if op == 'delta':
        return fast_weight_delta(*x, mem[0])
    if op == 'layer':
        return delta_attention(x[0], mem[0], s['scale'])
    if op == 'sum':
        return fast_weight_sum(*x, mem[0])
    if op == 'rec':
        return rec_update_fwm_tanh(*x, *s['weights'], *mem)
    if op == 'rnn1':
        return fast_rnn(x[0], x[1], x[2], mem[0], x[3], mem[1])
    if op == 'rnn2':
        return fast_rnn_v2(x[0], x[1], x[2], mem[0], x[3], mem[1])
    return LSTM[op](*x[0:4], mem[0], *x[4:8], mem[1], *x[8:12], mem[2], mem[3], mem[4])


def run(state):
    """One pass: an acting step on the carried memory, or forward (and backward) of every segment of the batch."""
    if state['mode'] == 'step':
        with torch.no_grad():
            return _call(state, state['segments'][0][0], state['mem']), state['mem']
    mem = [m.clone() for m in state['mem']]
    results = []
    for x, gy in state['segments']:
        if state['mode'] == 'eval':
            with torch.no_grad():
                results.append(_call(state, x, mem))
            continue
        out = _call(state, x, mem)
        y = out[0] if isinstance(out, tuple) else out
        carried = [m.clone() for m in mem]      # the backward takes the memory back to the segment's start
        results.append((out, torch.autograd.grad(y, x + state['weights'], gy)))
        mem = carried
    return results, mem


def work(case):
    """Every input read once and every output written once over the pass, and the products of the recurrence."""
    op, B, H, L, E, M = (case[k] for k in ('op', 'B', 'H', 'L', 'E', 'M'))
    train, n, esz = case['mode'] == 'train', 3 if op in LSTM else 1, 2 if case['dtype'] == 'bf16' else 4
    ins = (2 * E + M + (0 if op == 'sum' else 1)) if op in ('delta', 'sum', 'layer', 'rec') else n * (3 * E + 1)
    outs = M * (2 if op in LSTM else 1)
    units = B * H * L * case['segments']
    elements = ins + outs + (ins + M if train else 0)
    memory = B * H * n * (E * M + (0 if op in ('delta', 'sum', 'layer') else 2 * M)) * 2 * 4
    weights = (2 if train else 1) * H * (3 * E * E + E) * 4 if op == 'rec' else 0
    forward, backward = {'sum': (4, 10), 'rec': (12, 26)}.get(op, (6, 14))
    return {'bytes': units * elements * esz + memory + weights,
            'flops': units * n * E * M * (forward + (backward if train else 0))}


def tolerance(case):
    """32-bit sums over a few hundred to a few thousand steps; bf16 streams round every output to 8 bits."""
    return {'rel': 1e-2} if case['dtype'] == 'bf16' else {'rel': 2e-5}
