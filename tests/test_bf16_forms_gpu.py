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


@pytest.mark.parametrize('k_init', [0.005, 0.01, 0.02])
def test_large_launch_equals_small_ones(k_init):
    """Blocks of 64: one tensor of 3300 tiles takes one form of the kernel, its thirds the other one."""
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    n, parts = 3300 * DBS, 3
    hyper = dict(m=2, lr=1e-3, quant_block_size=64, k_init=k_init)
    gen = torch.Generator(device='cuda').manual_seed(7)
    whole = torch.nn.Parameter(torch.zeros(n, dtype=torch.bfloat16, device='cuda'))
    thirds = [torch.nn.Parameter(whole.detach()[i * (n // parts):(i + 1) * (n // parts)].clone()) for i in range(parts)]
    opt = MicroAdam([whole], **hyper)
    opts = [MicroAdam([p], **hyper) for p in thirds]
    for step in range(2):
        g = torch.empty(n, dtype=torch.bfloat16, device='cuda').normal_(0.0, 1e-3, generator=gen)
        blocks = g.view(-1, DBS)
        blocks[5::97] *= 64.0                            # bounds that do not carry over
        blocks[6::97] = 0.0
        blocks[7::97, ::2] = 1e-2 * torch.sign(blocks[7::97, ::2])
        whole.grad = g
        opt.step()
        for i, (p, o) in enumerate(zip(thirds, opts)):
            p.grad = g[i * (n // parts):(i + 1) * (n // parts)]
            o.step()
        a = opt.state[whole]
        for key in ('I', 'V', 'error', 'min_vals', 'max_vals'):
            have = a[key][step] if key in 'IV' else a[key]
            want = torch.cat([o.state[p][key][step] if key in 'IV' else o.state[p][key][:p.numel() // 64 if 'vals' in key else None]
                              for p, o in zip(thirds, opts)])
            assert torch.equal(have[:want.numel()].view(torch.uint8), want.view(torch.uint8)), (key, step)
    assert _native.device_error() == 0
