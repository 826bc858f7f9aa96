"""Kernel A on tiles that end anywhere (short octets, short rows, a handful of elements), for both gradient types, with
selections that take the fast route, its first bound from a histogram, and the general route: against the CPU oracle."""
import pytest
import torch

import cases
from ista_daslab_optimizers_b200 import synthetic as S

pytestmark = pytest.mark.gpu

DBS = 29056
SIZES = (1, 7, 8, 9, 63, 64, 65, 71, 130, 513, 2047, 2048, 2049, 28664, 28671, 28672, 28673, DBS - 1, DBS + 1, DBS + 57, 2 * DBS + 4093)


def _gradient(kind, n, step, dtype):
    g = S.normal_tensor(61 + step, n, n, 1e-3)
    if kind == 'wide':                                   # magnitudes over many octaves: the k-th lies far below the largest
        g = torch.sign(g) * torch.exp2(-60.0 * S.normal_tensor(71 + step, n, n, 0.3).abs().clamp(max=1.5))
        g[0] = 1e6
    elif kind == 'tiny':                                 # below the range of the histogram, and subnormal
        g *= 1e-36
    elif kind == 'equal':
        g = torch.full((n,), 0.5)
    elif kind == 'sparse':
        g[torch.arange(n) % 97 != 0] = 0.0
    return g.to(dtype)


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('kind,k_init,skip,alpha', [
    ('normal', 0.01, 0, 0), ('normal', 0.05, 8, 0), ('normal', 0.01, 1, 0), ('normal', 0.02, 2, 0), ('normal', 0.01, 5, 0),
    ('normal', 0.01, 0, -2), ('normal', 0.01, 3, -2), ('decay', 0.01, 0, 0), ('decay', 0.01, 3, 0),
    ('wide', 0.01, 0, 0), ('tiny', 0.02, 0, 0), ('equal', 0.01, 0, 0), ('sparse', 0.02, 0, 0)])
def test_short_tiles_match_oracle(kind, k_init, skip, alpha, dtype):
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    from oracle.microadam_oracle import MicroAdamOracle
    hyper = dict(m=4, lr=1e-3, quant_block_size=64, k_init=k_init, weight_decay=0.1, alpha=alpha)
    if kind == 'decay':                                  # a decay that changes bf16 parameters
        hyper.update(lr=1e-2, weight_decay=0.5)
    params = [torch.nn.Parameter(S.normal_tensor(60, i, n + skip, 0.02).to(dtype).cuda()[skip:]) for i, n in enumerate(SIZES)]
    cpu = [p.detach().cpu().clone() for p in params]
    opt = MicroAdam(params, **hyper)
    ref = MicroAdamOracle(cpu, d_block_size=opt.d_block_size, **hyper)
    for step in range(3):
        grads = [_gradient(kind, n, step, dtype) for n in SIZES]
        for p, g in zip(params, grads):
            p.grad = torch.empty(g.numel() + skip, dtype=dtype, device='cuda')[skip:].copy_(g)
        opt.step()
        ref.step([g.clone() for g in grads])
        for i, (p, n) in enumerate(zip(params, SIZES)):
            a, b, used = opt.state[p], ref.state[i], -(-n // 64)
            assert torch.equal(a['I'][step].cpu(), b['I'][step]), (n, step)
            assert torch.equal(a['V'][step].cpu().view(torch.int16), b['V'][step].view(torch.int16)), (n, step)
            for key, cut in (('error', None), ('min_vals', used), ('max_vals', used)):
                assert torch.equal(a[key][:cut].cpu().view(torch.uint8), b[key][:cut].view(torch.uint8)), (n, step, key)
            if kind != 'tiny':                           # (moments of subnormal gradients: not what this test is about)
                rtol, atol = cases.param_tolerances(dtype, hyper['lr'])
                torch.testing.assert_close(p.detach().cpu().float(), cpu[i].float(), rtol=rtol, atol=atol)
    assert _native.device_error() == 0


@pytest.mark.parametrize('qbs', [64, 32])
def test_full_tiles_that_end_inside_a_row(qbs):
    """bf16 tiles long enough for the branch-free decode whose last row of eight octets is short: the rows are permuted in
    place, the last octets of a thread among partly idle warps."""
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    from oracle.microadam_oracle import MicroAdamOracle
    sizes = (28672 + 8, 28672 + 56, 28672 + 256 - 8, 28672 + 264, DBS - 8, 2 * DBS - 40)
    hyper = dict(m=3, lr=1e-3, quant_block_size=qbs, k_init=0.01)
    params = [torch.nn.Parameter(S.normal_tensor(62, i, n, 0.02).bfloat16().cuda()) for i, n in enumerate(sizes)]
    opt = MicroAdam(params, **hyper)
    ref = MicroAdamOracle([p.detach().cpu().clone() for p in params], d_block_size=opt.d_block_size, **hyper)
    for step in range(3):
        grads = [S.normal_tensor(63 + step, n, n, 1e-3).bfloat16() for n in sizes]
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        opt.step()
        ref.step([g.clone() for g in grads])
        for i, (p, n) in enumerate(zip(params, sizes)):
            a, b, used = opt.state[p], ref.state[i], -(-n // qbs)
            assert torch.equal(a['I'][step].cpu(), b['I'][step]), (n, step)
            for key, cut in (('V', None), ('error', None), ('min_vals', used), ('max_vals', used)):
                assert torch.equal(a[key][:cut].cpu().view(torch.uint8), b[key][:cut].view(torch.uint8)), (n, step, key)
    assert _native.device_error() == 0
