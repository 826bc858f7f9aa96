"""The work that users of this package have it do, as cases that can be timed.

A case is one pass through the public entry points with everything a training program holds at that moment already
on the GPU: parameters, gradients, and an optimizer whose window is full (`m` steps have been taken).

* kind 'step':      `MicroAdam.step()` over a list of parameters;
* kind 'operators': the reference's own call sequence on the operator-level functions (what an unmodified
                    micro_adam.py does through `compat`);
* kind 'rows':      the two functions Sparse M-FAC calls on the (index, value) ring buffer.

`listed()` are fixed cases, `draw()` makes further ones of the same ranges.
"""
import os
import sys

import torch

# the package's folder lies in the repository's root, which is the working folder
sys.path.insert(0, os.path.join(os.getcwd(), 'ista-daslab-optimizers_b200'))

from ista_daslab_optimizers_b200 import CopyDirection, MicroAdam, _native, block_split, synthetic  # noqa: E402
from ista_daslab_optimizers_b200.compat import ista_daslab_cuda_micro_adam as ops  # noqa: E402
from ista_daslab_optimizers_b200.compat import ista_daslab_cuda_tools as tools  # noqa: E402

_DTYPES = {'f32': torch.float32, 'bf16': torch.bfloat16}
_BYTES = {'f32': 4, 'bf16': 2}
_LARGEST = 1 << 28        # elements of the largest drawn flat tensor (the largest listed list has eight times as many)


def _case(name, kind='step', **more):
    c = dict(name=name, kind=kind, layout='flat', numel=0, width=0, count=0, vocab=0, skip=0, param='f32', grad='f32', m=10,
             k_init=0.01, qbs=64, alpha=0.0, weight_decay=0.0)
    c.update(more)
    return c


def listed():
    return [
        # the classifier of a frozen backbone: one tiny tensor, all latency
        _case('head_fp32', numel=768 * 10 + 10),
        # one transformer block of width 768 in fp32 (12 tensors, a few of them vectors)
        _case('block_fp32', layout='block', width=768),
        # a convolutional model: many ragged tensors, fp32 master parameters with bf16 gradients
        _case('many_ragged_mixed', layout='ragged', count=120, width=512, grad='bf16', weight_decay=0.01),
        # the flat fp32 parameter of a 124 M model, one tensor (the second workload of bench.py)
        _case('flat_fp32', numel=124439808),
        # one layer of the bf16 list that bench.py steps (nine tensors of width 4096, weight decay)
        _case('layer_bf16', layout='layers', width=4096, count=1, param='bf16', grad='bf16', weight_decay=0.1),
        # a quarter of that list, which is what one of four GPUs holds: the embedding and seven layers
        _case('stack_bf16', layout='layers', width=4096, count=7, vocab=128256, param='bf16', grad='bf16', weight_decay=0.1),
        # the quantisation block of the reference's README, which ignores the borders of the top-k blocks
        _case('layer_bf16_qbs100000', layout='layers', width=4096, count=1, param='bf16', grad='bf16', weight_decay=0.1, qbs=100000),
        # the error feedback mixed into the update (alpha in (0, 1))
        _case('flat_fp32_alpha', numel=1 << 25, alpha=0.5, weight_decay=0.1),
        # the quantisation error added to the parameters (alpha == -2), a layer of half the width
        _case('layer_bf16_alpha_m2', layout='layers', width=2048, count=1, param='bf16', grad='bf16', weight_decay=0.1, alpha=-2.0),
        # a dense window: 5 % of every block in every row, an odd number of elements
        _case('flat_fp32_dense_window', numel=(1 << 26) + 3, k_init=0.05),
        # the operator-level calls in the order of the reference's update_step, with an odd number of elements
        _case('operators_fp32', kind='operators', numel=25557033, weight_decay=0.1),
        # scalar products with every row of a Sparse M-FAC ring buffer and a linear combination of its rows
        _case('sparse_rows_fp32', kind='rows', numel=25557032, m=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    u = rng.random()
    kind = 'step' if u < 0.8 else 'operators' if u < 0.9 else 'rows'
    c = _case('', kind)
    del c['name']
    c['m'] = rng.choice([5, 10, 10, 10, 20])
    c['k_init'] = rng.choice([0.005, 0.01, 0.01, 0.01, 0.02, 0.05])
    c['weight_decay'] = rng.choice([0.0, 0.01, 0.1])
    if kind == 'rows':
        c.update(numel=_log_int(rng, 4096, 1 << 26), m=rng.choice([8, 16, 32, 64]), grad=rng.choice(['f32', 'bf16']))
        return c
    c['qbs'] = rng.choice([64, 64, 64, 64, 32, 128, 100000])
    if kind == 'operators':
        dtype = rng.choice(['f32', 'bf16'])
        c.update(numel=_log_int(rng, 512, 1 << 26), param=dtype, grad=dtype)
        return c
    c['param'], c['grad'] = rng.choice([('f32', 'f32'), ('bf16', 'bf16'), ('bf16', 'bf16'), ('f32', 'bf16')])
    if c['qbs'] != 100000:
        c['alpha'] = rng.choice([0.0, 0.0, 0.0, 0.0, 0.1, 0.5] + ([-2.0] if c['param'] == c['grad'] else []))
    c['layout'] = rng.choice(['flat', 'flat', 'block', 'layers', 'ragged'])
    if c['layout'] == 'flat':
        c['numel'] = _log_int(rng, 512, _LARGEST)
        c['skip'] = rng.choice([0, 0, 0, 1, 2, 3, 5])      # a shard of a flat buffer that starts anywhere
    elif c['layout'] == 'block':
        c['width'] = 8 * _log_int(rng, 8, 250)
    elif c['layout'] == 'layers':
        c.update(width=128 * _log_int(rng, 4, 32), count=rng.choice([1, 1, 2]))
    else:
        c.update(count=rng.randrange(20, 201), width=_log_int(rng, 64, 768))
    return c


def _shapes(c):
    w = c['width']
    if c['layout'] == 'flat':
        return [(c['numel'],)]
    if c['layout'] == 'block':
        return [(w,), (w,), (3 * w, w), (3 * w,), (w, w), (w,), (w,), (w,), (4 * w, w), (4 * w,), (w, 4 * w), (w,)]
    if c['layout'] == 'layers':
        f = (7 * w // 2) // 8 * 8
        layer = [(w, w), (w // 4, w), (w // 4, w), (w, w), (f, w), (f, w), (w, f), (w,), (w,)]
        return ([(c['vocab'], w)] if c['vocab'] else []) + layer * c['count']
    return [s if i % 3 else (s[0],) for i, s in enumerate(synthetic.stress_shapes(c['count'], count=c['count'], lo=8, hi=w))]


def _numel(c):
    return sum(torch.Size(s).numel() for s in _shapes(c))


def _own_form(c):
    """Whether the pass leaves something else than the gradient in the gradient's buffer."""
    return c['kind'] == 'operators' or c['qbs'] not in (8, 16, 32, 64, 128)


def _packed(sizes, dtype):
    """One buffer and a view of it per size, every view on a 256-byte boundary."""
    step = 256 // torch.empty(0, dtype=dtype).element_size()
    at, offsets = 0, []
    for n in sizes:
        offsets.append(at)
        at += -(-n // step) * step
    buf = torch.zeros(max(at, 1), dtype=dtype, device='cuda')
    return buf, [buf[o:o + n] for o, n in zip(offsets, sizes)]


class _State:
    pass


def _prepare_step(c, s, gen):
    shapes, pd, gd = _shapes(c), _DTYPES[c['param']], _DTYPES[c['grad']]
    sigma = 1e-4 if c['param'] == 'bf16' else 1e-3
    sizes = [torch.Size(x).numel() for x in shapes]
    s.many = len(shapes) > 9        # then parameters and optimizer state live in one buffer per kind
    # parameters (and the gradient) of a flat shard may start anywhere in their buffers
    flat_p, views = _packed([sizes[0] + c['skip']] if c['layout'] == 'flat' else sizes, pd)
    flat_p.normal_(0.0, 0.02, generator=gen)
    if c['layout'] == 'flat':
        views = [views[0][c['skip']:]]
    elif not s.many:
        views = [v.clone() for v in views]
    s.params = [torch.nn.Parameter(v.view(x)) for v, x in zip(views, shapes)]
    if c['param'] != c['grad']:
        for p in s.params:
            p.grad_dtype = gd       # master parameters: torch checks the type of p.grad
    s.flat_p = flat_p if s.many else None
    s.grads = []                    # two sets, taken in turn
    for _ in range(2):
        g = [torch.empty(n + c['skip'], dtype=gd, device='cuda')[c['skip']:].view(x) for n, x in zip(sizes, shapes)]
        s.grads.append(g)
    hyper = dict(m=c['m'], lr=1e-3, quant_block_size=c['qbs'], k_init=c['k_init'], weight_decay=c['weight_decay'],
                 alpha=int(c['alpha']) if c['alpha'] in (0.0, -2.0) else c['alpha'])

    def fresh(k):
        for p, g in zip(s.params, s.grads[k]):
            g.normal_(0.0, sigma, generator=gen)
            p.grad = g

    s.opt = MicroAdam(s.params, **hyper)
    for t in range(c['m']):
        fresh(t & 1)
        s.opt.step()
    s.kept = None
    if s.many:
        # a program that keeps the optimizer's state in one buffer per kind, as one copy to and from a checkpoint
        old, s.opt = s.opt, MicroAdam(s.params, **hyper)
        s.opt.steps, s.kept = old.steps, {}
        for p in s.params:
            s.opt.state[p] = dict(old.state[p])
        for key in ('I', 'V', 'error', 'min_vals', 'max_vals') + (('quant_err',) if c['alpha'] == -2.0 else ()):
            have = [old.state[p][key] for p in s.params]
            s.kept[key], to = _packed([h.numel() for h in have], have[0].dtype)
            for p, h, v in zip(s.params, have, to):
                v.copy_(h.reshape(-1))
                s.opt.state[p][key] = v.view(h.shape)
    s.turn = 0
    fresh(1)
    fresh(0)
    if _own_form(c):
        # what the backward pass would write into the gradients before every step
        s.source = s.grads
        for p, g in zip(s.params, s.grads[0]):
            p.grad = g.clone()
        s.into = [p.grad for p in s.params]


def _prepare_operators(c, s, gen):
    d, dt = c['numel'], _DTYPES[c['param']]
    s.d, s.alpha_lr, s.qbs = d, 1e-3, c['qbs']
    most = tools.get_max_floats_for_shared_memory_per_thread_block() // 2
    s.dbs = min(d, most)
    full, s.at_tail = block_split(d, s.dbs)
    s.k_many, s.k_few = -(-int(s.dbs * c['k_init'] * 1e6) // 1000000), -(-int((d - s.at_tail) * c['k_init'] * 1e6) // 1000000)
    s.k = full * s.k_many + s.k_few
    s.m, s.steps, s.row, s.decay = c['m'], 0, 0, 1 - 1e-3 * c['weight_decay']
    s.p = torch.empty(d, dtype=dt, device='cuda').normal_(0.0, 0.02, generator=gen)
    s.I = torch.zeros(s.m, s.k, dtype=torch.int16, device='cuda')
    s.V = torch.zeros(s.m, s.k, dtype=torch.bfloat16, device='cuda')
    s.error = torch.zeros(-(-d // 2), dtype=torch.uint8, device='cuda')
    s.min_vals = torch.zeros(d // s.qbs + 1, dtype=torch.bfloat16, device='cuda')
    s.max_vals = torch.zeros(d // s.qbs + 1, dtype=torch.bfloat16, device='cuda')
    s.source = [torch.empty(d, dtype=dt, device='cuda') for _ in range(2)]
    s.grad = torch.empty(d, dtype=dt, device='cuda')
    s.blocks, s.turn = tools.get_sm_count(), 0
    for _ in range(s.m):
        s.source[s.turn].normal_(0.0, 1e-3, generator=gen)
        _run_operators(s)


def _prepare_rows(c, s, gen):
    d, gd = c['numel'], _DTYPES[c['grad']]
    s.d, s.m = d, c['m']
    s.dbs = min(d, tools.get_max_floats_for_shared_memory_per_thread_block() // 2)
    full, at = block_split(d, s.dbs)
    s.k_many, k_few = -(-int(s.dbs * c['k_init'] * 1e6) // 1000000), -(-int((d - at) * c['k_init'] * 1e6) // 1000000)
    s.k = full * s.k_many + k_few
    s.I = torch.zeros(s.m, s.k, dtype=torch.int16, device='cuda')
    s.V = torch.zeros(s.m, s.k, dtype=torch.bfloat16, device='cuda')
    x = torch.empty(d, dtype=torch.float32, device='cuda')
    for r in range(s.m):
        x.normal_(0.0, 1e-3, generator=gen)
        _native.block_topk(d, s.dbs, s.k_many, k_few, x, s.I[r])
        tools.copy_values(d, s.k, s.dbs, s.k_many, s.I[r], x, s.V[r], CopyDirection.d2k.value)
    s.g = torch.empty(d, dtype=gd, device='cuda').normal_(0.0, 1e-3, generator=gen)
    s.M = torch.empty(s.m, device='cuda').normal_(0.0, 1e-3, generator=gen)
    s.dots = torch.zeros(s.m, device='cuda')
    s.out = torch.zeros(d, dtype=gd, device='cuda')


def prepare(case, seed):
    gen = torch.Generator(device='cuda')
    gen.manual_seed(int(seed))
    s = _State()
    s.case = case
    {'step': _prepare_step, 'operators': _prepare_operators, 'rows': _prepare_rows}[case['kind']](case, s, gen)
    return s


def _run_step(s):
    s.turn ^= 1
    if _own_form(s.case):
        torch._foreach_copy_(s.into, s.source[s.turn])
    else:
        for p, g in zip(s.params, s.grads[s.turn]):
            p.grad = g
    s.opt.step()
    if s.many:
        return [s.flat_p, s.kept]
    return [[p, s.opt.state[p]['I'], s.opt.state[p]['V'], s.opt.state[p]['error'], s.opt.state[p]['min_vals'],
             s.opt.state[p]['max_vals'], s.opt.state[p].get('quant_err')] for p in s.params]


def _run_operators(s):
    """micro_adam.py:190-304 with alpha == 0."""
    s.turn ^= 1
    s.steps += 1
    g = s.grad
    g.copy_(s.source[s.turn])                                # the backward pass: the step uses the gradient as scratch
    I, V = s.I[s.row], s.V[s.row]
    ops.asymm_block_quant_inv(s.d, s.qbs, s.error, s.min_vals, s.max_vals, g, 1.0)
    _native.block_topk(s.d, s.dbs, s.k_many, s.k_few, g, I)
    tools.copy_values(s.d, s.k, s.dbs, s.k_many, I, g, V, CopyDirection.d2k.value)
    s.row = (s.row + 1) % s.m
    tools.zerorize_block_components(g, I, s.d, s.k, s.dbs, s.k_many)
    _native.quant_stats(s.d, s.qbs, s.min_vals, s.max_vals, g)
    ops.asymm_block_quant(s.d, s.qbs, s.error, s.min_vals, s.max_vals, g)
    if s.decay != 1.0:
        s.p.mul_(s.decay)
    ops.compute_microadam_update(s.blocks, 512, 100, s.steps, 0.9, 0.999, 1e-8, s.dbs, s.k_many, s.d, s.m, s.k, s.I, s.V, g)
    s.p.add_(g, alpha=-s.alpha_lr)
    return [s.p, g, s.I, s.V, s.error, s.min_vals, s.max_vals]


def _run_rows(s):
    _native.sparse_rows_dot(s.d, s.m, s.k, s.dbs, s.k_many, s.g, s.I, s.V, s.dots)
    _native.sparse_rows_combine(s.d, s.m, s.k, s.dbs, s.k_many, s.M, s.I, s.V, s.out)
    return [s.dots, s.out]


def run(state):
    return {'step': _run_step, 'operators': _run_operators, 'rows': _run_rows}[state.case['kind']](state)


def work(case):
    c, n = case, _numel(case)
    p, g, k = _BYTES[c['param']], _BYTES[c['grad']], c['k_init']
    if c['kind'] == 'rows':
        # a full row set for the products and once more for the combination, the dense vectors once each
        return {'bytes': n * (4.0 * c['m'] * k + 3 * g), 'flops': 4.0 * c['m'] * k * n}
    # gradient in, codes and statistics in and out, one window row out, the window in, the parameter in and out
    per = g + 1.0 + 8.0 / c['qbs'] + 4.0 * k + 4.0 * c['m'] * k + 2.0 * p
    if c['alpha'] == -2.0:
        per += p                                            # the quantisation error out
    if _own_form(c):
        per += 2.0 * g                                      # the gradient is written anew before the step
    return {'bytes': per * n, 'flops': 30.0 * n}


def tolerance(case):
    # indices, codes: equal. Values: a sum of m products and an approximate quotient in fp32, stored as the parameter's type.
    if case['kind'] == 'rows':
        return {'rel': 1e-2 if case['grad'] == 'bf16' else 1e-5}
    return {'rel': 1e-2 if 'bf16' in (case['param'], case['grad']) else 1e-5}
