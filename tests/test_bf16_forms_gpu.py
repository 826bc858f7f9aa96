"""The bf16 kernel A whose warps own their part of the tile: against the CPU oracle where it can go wrong (tiles that end around a
unit, a slot or a quantisation block, gradients off alignment, every block size, tensors whose bound cannot come from the one
before), and against the other form, which takes small launches with blocks of 64."""
import pytest
import torch

import cases
from ista_daslab_optimizers_b200 import synthetic as S

pytestmark = pytest.mark.gpu

DBS = 29056
SIZES = (1, 15, 16, 17, 511, 512, 513, 4095, 4104, DBS - 1, DBS, DBS + 520, 2 * DBS + 7)


def _gradient(kind, i, n, step):
    g = S.normal_tensor(51 + step, i, n, 1e-3)
    if kind == 'scales':                                 # no tensor's bound fits the next one
        g *= 2.0 ** ((i * 5) % 13 - 6)
    elif kind == 'ties':
        g[::3] = 2e-3 * torch.sign(g[::3])
    elif kind == 'cluster':                              # all that is selected lies in one warp's part, far above the rest
        g[: max(1, n // 16)] *= 300.0
    elif kind == 'few':
        g.zero_()
        g[:: max(1, n // 5)] = -1.5
    return g.bfloat16()


@pytest.mark.parametrize('kind,qbs,k_init,skip', [
    ('normal', 8, 0.01, 0), ('normal', 16, 0.02, 0), ('normal', 32, 0.01, 3), ('normal', 128, 0.05, 8), ('normal', 72, 0.01, 0),
    ('normal', 100000, 0.05, 0), ('scales', 32, 0.01, 0), ('scales', 1000, 0.01, 1), ('ties', 128, 0.05, 0), ('cluster', 32, 0.05, 0),
    ('cluster', 100000, 0.01, 0), ('few', 32, 0.01, 0), ('normal', 32, 0.2, 0)])
def test_warp_owned_tiles_match_oracle(kind, qbs, k_init, skip):
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    from oracle.microadam_oracle import MicroAdamOracle
    hyper = dict(m=4, lr=1e-3, quant_block_size=qbs, k_init=k_init, weight_decay=0.1)
    params = [torch.nn.Parameter(S.normal_tensor(50, i, n, 0.02).bfloat16().cuda()) for i, n in enumerate(SIZES)]
    cpu = [p.detach().cpu().clone() for p in params]
    opt = MicroAdam(params, **hyper)
    ref = MicroAdamOracle(cpu, d_block_size=opt.d_block_size, **hyper)
    assert opt.d_block_size == DBS
    for step in range(3):
        grads = [_gradient(kind, i, n, step) for i, n in enumerate(SIZES)]
        for p, g in zip(params, grads):
            p.grad = torch.empty(g.numel() + skip, device='cuda', dtype=torch.bfloat16)[skip:].copy_(g)
        opt.step()
        ref.step([g.clone() for g in grads])
        for i, (p, n) in enumerate(zip(params, SIZES)):
            a, b, used, row = opt.state[p], ref.state[i], -(-n // qbs), step % hyper['m']
            assert torch.equal(a['I'][row].cpu(), b['I'][row]), (n, step)
            for key, cut in (('error', None), ('min_vals', used), ('max_vals', used)):
                assert torch.equal(a[key][:cut].cpu().view(torch.uint8), b[key][:cut].view(torch.uint8)), (n, step, key)
            assert torch.equal(a['V'][row].cpu().view(torch.int16), b['V'][row].view(torch.int16)), (n, step)
            rtol, atol = cases.param_tolerances(torch.bfloat16, hyper['lr'])
            torch.testing.assert_close(p.detach().cpu(), cpu[i], rtol=rtol, atol=atol)
    assert _native.device_error() == 0


def _kernels_of(step):
    """Names of the kernels a call launches."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        step()
        torch.cuda.synchronize()
    return [e.name for e in prof.events() if e.device_type.name == 'CUDA']


def _same(a, b):
    """Equal bits; a NaN equals every other NaN."""
    if a.dtype == torch.uint8:
        return torch.equal(a, b)
    nan = torch.isnan(a.float()) & torch.isnan(b.float())
    return torch.equal(a.view(torch.int16)[~nan], b.view(torch.int16)[~nan])


# full tiles (the last one: more than 20 a SM together), and between them lengths that end around a unit, a slot or a block and
# make the warps' parts of the tile change hands
MANY = (1400 * DBS, 7, DBS - 1, 513, 600 * DBS + 4104, 64, 65 * 64 + 15, 2 * DBS + 8191, 16, 1400 * DBS + 33)


@pytest.mark.parametrize('kind,k_init,alpha', [('mixed', 0.005, 0), ('mixed', 0.01, 0), ('mixed', 0.02, 0), ('mixed', 0.01, -2),
                                               ('nan', 0.01, 0), ('inf', 0.01, 0)])
def test_large_launch_equals_small_ones(kind, k_init, alpha):
    """Blocks of 64: a step of more than ten tiles per SM takes one form of the kernel, its tensors by themselves the other one."""
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    hyper = dict(m=2, lr=1e-3, quant_block_size=64, k_init=k_init, alpha=alpha)
    gen = torch.Generator(device='cuda').manual_seed(7)
    whole = [torch.nn.Parameter(torch.zeros(n, dtype=torch.bfloat16, device='cuda')) for n in MANY]
    alone = [torch.nn.Parameter(p.detach().clone()) for p in whole]
    opt = MicroAdam(whole, **hyper)
    opts = [MicroAdam([p], **hyper) for p in alone]
    for step in range(3):
        for p, q in zip(whole, alone):
            n = p.numel()
            g = torch.empty(n, dtype=torch.bfloat16, device='cuda').normal_(0.0, 1e-3, generator=gen)
            blocks = g[:n // DBS * DBS].view(-1, DBS)
            blocks[5::97] *= 64.0                        # bounds that do not carry over
            blocks[6::97] = 0.0
            blocks[7::97, ::2] = 1e-2 * torch.sign(blocks[7::97, ::2])
            if kind == 'nan' and step < 2:
                g[3::4099] = float('nan')
                blocks[8::97, 4096:8192] = float('nan')
                blocks[9::97, :DBS - 1600] = float('nan')
            if kind == 'inf' and step < 2:
                g[3::5003] = float('inf')
                g[9::7001] = float('-inf')
                blocks[8::97, ::64] = float('inf')       # more than k of them: the residual's statistics are infinite
            p.grad = g
            q.grad = g.clone()
        if step == 0:
            names = _kernels_of(opt.step)
            assert any('ef_topk_quant_bf16_warps_kernel<6>' in x.replace('(int)', '') for x in names), names
        else:
            opt.step()
        for i, o in enumerate(opts):
            if step == 0 and i == 0:
                names = _kernels_of(o.step)
                assert any('ef_topk_quant_bf16_kernel' in x for x in names), names
            else:
                o.step()
        for p, q, o in zip(whole, alone, opts):
            a, b = opt.state[p], o.state[q]
            used = -(-p.numel() // 64)
            for key in ('I', 'V', 'error', 'min_vals', 'max_vals') + (('quant_err',) if alpha == -2 else ()):
                x, y = (t[key][step % 2] if key in ('I', 'V') else t[key][:used] if 'vals' in key else t[key] for t in (a, b))
                assert _same(x.contiguous(), y.contiguous()), (p.numel(), step, key)
            assert _same(p.detach(), q.detach()), (p.numel(), step)
    assert _native.device_error() == 0


@pytest.mark.parametrize('k_init,skip', [(0.05, 0), (0.01, 3), (0.05, 1), (0.2, 8), (0.01, 8), (0.01, -3)])
def test_line_between_the_forms(k_init, skip):
    """Blocks of 64: from ten tiles per SM on a launch takes the warp-owned form whatever k and alignment (skip < 0:
    the short tensor's gradient only), below it the other one; equal results on both sides."""
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    from ista_daslab_optimizers_b200.compat import ista_daslab_cuda_tools as tools
    tiles = 10 * tools.get_sm_count()
    sizes = ((tiles - 3) * DBS, 2 * DBS + 4104)          # tiles - 3 and three tiles
    hyper = dict(m=2, lr=1e-3, quant_block_size=64, k_init=k_init)
    gen = torch.Generator(device='cuda').manual_seed(11)
    whole = [torch.nn.Parameter(torch.zeros(n, dtype=torch.bfloat16, device='cuda')) for n in sizes]
    alone = [torch.nn.Parameter(p.detach().clone()) for p in whole]
    opt, opts = MicroAdam(whole, **hyper), [MicroAdam([p], **hyper) for p in alone]
    for step in range(2):
        for p, q in zip(whole, alone):
            off = skip if skip >= 0 else -skip if p is whole[1] else 0
            p.grad = torch.empty(p.numel() + off, dtype=torch.bfloat16, device='cuda')[off:].normal_(0.0, 1e-3, generator=gen)
            q.grad = p.grad.clone()
        for form, o in (('ef_topk_quant_bf16_warps_kernel', opt), ('ef_topk_quant_bf16_kernel', opts[0])):
            if step == 0:
                names = _kernels_of(o.step)
                assert any(form in x for x in names), names
            else:
                o.step()
        opts[1].step()
        for p, q, o in zip(whole, alone, opts):
            a, b, used = opt.state[p], o.state[q], -(-p.numel() // 64)
            for key in ('I', 'V', 'error', 'min_vals', 'max_vals'):
                x, y = (t[key][step] if key in ('I', 'V') else t[key][:used] if 'vals' in key else t[key] for t in (a, b))
                assert torch.equal(x.contiguous().view(torch.uint8), y.contiguous().view(torch.uint8)), (p.numel(), step, key)
            assert torch.equal(p.detach().view(torch.int16), q.detach().view(torch.int16)), (p.numel(), step)
    assert _native.device_error() == 0


@pytest.mark.parametrize('qbs', [8, 16, 32, 128, 64, 1000, 100000])
def test_infinities_match_the_operator_level_kernels(qbs):
    """Infinite gradients, fewer than k of a tile: selected like any large value, and nothing of them stays in the residual."""
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    hyper = dict(m=4, lr=1e-3, quant_block_size=qbs, k_init=0.01)
    pairs = []
    for use_fused in (True, False):
        params = [torch.nn.Parameter(S.normal_tensor(60, i, n, 0.02).bfloat16().cuda()) for i, n in enumerate(SIZES)]
        pairs.append((params, MicroAdam(params, use_fused=use_fused, **hyper)))
    for step in range(3):
        for i, n in enumerate(SIZES):
            g = _gradient('normal', i, n, step)
            if step < 2 and n >= 4095:
                g[11::1500] = float('inf')
                g[700::3000] = float('-inf')
            for params, _ in pairs:
                params[i].grad = g.cuda()
        for _, opt in pairs:
            opt.step()
        for p, q, n in zip(*(params for params, _ in pairs), SIZES):
            a, b, used = pairs[0][1].state[p], pairs[1][1].state[q], -(-n // qbs)
            for key in ('I', 'V', 'error', 'min_vals', 'max_vals'):
                x, y = (t[key][step] if key in ('I', 'V') else t[key][:used] if 'vals' in key else t[key] for t in (a, b))
                assert torch.equal(x.view(torch.uint8), y.view(torch.uint8)), (n, step, key)
            assert torch.isfinite(a['max_vals'][:used].float()).all()
    assert all(e.fused for e in pairs[0][1]._entries) and not any(e.fused for e in pairs[1][1]._entries)
    assert _native.device_error() == 0
