"""Gradients that hold NaN: never selected (so that a row of the window holds exactly k entries of every block), whichever
route a tile takes through kernel A."""
import pytest
import torch

from ista_daslab_optimizers_b200 import synthetic as S

pytestmark = pytest.mark.gpu

DBS = 29056
SIZES = (2 * DBS, 3 * DBS + 4096, DBS + 1003, 9000, 300)


def _gradient(kind, n, step, dtype):
    g = S.normal_tensor(81 + step, n, n, 1e-3)
    if kind == 'scattered':                              # one NaN in every second octet, next to values that are selected
        g[3::16] = float('nan')
        g[4::64] *= 20.0
    return g.to(dtype)


def _expected_row(g, geo):
    """Indices and values of the window row for a zero error feedback: the k largest magnitudes of every block, NaN last."""
    key = g.float().abs()
    key[key.isnan()] = -1.0
    idx, at = [], 0
    while at < g.numel():
        n = min(geo['d_block_size'], g.numel() - at)
        k = geo['k_block_size_many'] if n == geo['d_block_size'] else geo['k_block_size_few']
        order = torch.sort(key[at:at + n], descending=True, stable=True).indices[:k].sort().values
        idx.append((order, order + at))
        at += n
    return torch.cat([i for i, _ in idx]).to(torch.int16), g[torch.cat([p for _, p in idx])].bfloat16()


@pytest.mark.parametrize('dtype,kind', [(torch.bfloat16, 'scattered'), (torch.float32, 'scattered')])
@pytest.mark.parametrize('skip,qbs', [(0, 64), (1, 64), (0, 32), (0, 1000)])
def test_nan_is_never_selected(dtype, kind, skip, qbs):
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    params = [torch.nn.Parameter(S.normal_tensor(80, i, n, 0.02).to(dtype).cuda()) for i, n in enumerate(SIZES)]
    opt = MicroAdam(params, m=3, lr=1e-3, quant_block_size=qbs, k_init=0.01)
    grads = [_gradient(kind, n, 0, dtype) for n in SIZES]
    for p, g in zip(params, grads):
        p.grad = torch.empty(g.numel() + skip, dtype=dtype, device='cuda')[skip:].copy_(g)
    opt.step()
    for p, g in zip(params, grads):
        st = opt.state[p]
        I, V = _expected_row(g, st)
        assert torch.equal(st['I'][0].cpu(), I), g.numel()
        assert torch.equal(st['V'][0].cpu().view(torch.int16), V.view(torch.int16)), g.numel()
        assert not st['I'][1:].any() and not st['V'][1:].any()          # nothing past the end of the row
    assert _native.device_error() == 0


@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
@pytest.mark.parametrize('qbs', [64, 32, 1000])
def test_nan_octets_do_not_move_the_bound(dtype, qbs):
    """Tiles with more octets of nothing but NaN than the k that are selected, met by CTAs that come with the bound of a tile
    before (more tiles than CTAs), and tiles where they leave fewer octets than k."""
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    tiles = 148 * 3 + 40
    g = S.normal_tensor(82, 1, tiles * DBS, 1e-3)
    t = g.view(tiles, DBS)
    t[300::3, 4096:8192] = float('nan')                  # 512 octets, k = 291
    t[301::6, :DBS - 1600] = float('nan')                # 200 octets are left
    t[302::7, 8:16] = float('nan')
    g = g.to(dtype)
    p = torch.nn.Parameter(torch.zeros(g.numel(), dtype=dtype, device='cuda'))
    opt = MicroAdam([p], m=2, lr=1e-3, quant_block_size=qbs, k_init=0.01)
    p.grad = g.cuda()
    opt.step()
    st = opt.state[p]
    I, V = _expected_row(g, st)
    assert torch.equal(st['I'][0].cpu(), I)
    assert torch.equal(st['V'][0].cpu().view(torch.int16), V.view(torch.int16))
    assert not st['I'][1].any() and not st['V'][1].any()
    assert _native.device_error() == 0
