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
    elif kind == 'zeros':                                # nothing but zeros next to them
        g.zero_()
        g[3::16] = float('nan')
        g[64:128] = float('nan')
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


@pytest.mark.parametrize('dtype,kind', [(torch.bfloat16, 'scattered'), (torch.float32, 'scattered'), (torch.float32, 'zeros')])
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


@pytest.mark.parametrize('dtype,qbs', [(torch.bfloat16, 64), (torch.bfloat16, 32), (torch.bfloat16, 128),
                                       (torch.float32, 64), (torch.float32, 32), (torch.float32, 1000)])
@pytest.mark.parametrize('offset', [0.0, 0.02])
def test_nan_spoils_no_neighbour(dtype, qbs, offset):
    """A NaN gets code 0 and is in no statistics: error feedback and window are, bit for bit, those of the operator-level
    kernels, whose codec is the scalar definition, and no parameter becomes NaN.  (With an offset the statistics are coarse
    against a quantisation step, and the fp32 kernel clamps.)"""
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    sizes = SIZES + (29056 + 64 * 3 + 5, 64, 71)
    hyper = dict(m=3, lr=1e-3, quant_block_size=qbs, k_init=0.01)
    pairs = []
    for use_fused in (True, False):
        params = [torch.nn.Parameter(S.normal_tensor(83, i, n, 0.02).to(dtype).cuda()) for i, n in enumerate(sizes)]
        pairs.append((params, MicroAdam(params, use_fused=use_fused, **hyper)))
    for step in range(4):
        for i, n in enumerate(sizes):
            g = S.normal_tensor(84 + step, n, n, 1e-3) + (offset if step == 0 else 0.0)
            if step < 3:
                g[3::16 + step] = float('nan')
                g[n // 2:n // 2 + 10] = float('nan')
                if n > 4096:
                    g[1280:1280 + 64 * 5] = float('nan')        # whole quantisation blocks
            for params, _ in pairs:
                params[i].grad = g.to(dtype).cuda()
        for _, opt in pairs:
            opt.step()
        for p, q in zip(*(params for params, _ in pairs)):
            a, b = pairs[0][1].state[p], pairs[1][1].state[q]
            for key in ('I', 'V', 'error', 'min_vals', 'max_vals'):
                x, y = a[key], b[key]
                if key in ('min_vals', 'max_vals'):      # (a block of nothing else: any statistics that decode to NaN)
                    x, y = x.nan_to_num(0.0, 0.0, 0.0), y.nan_to_num(0.0, 0.0, 0.0)
                assert torch.equal(x.view(torch.uint8), y.view(torch.uint8)), (step, p.numel(), key)
            assert torch.isfinite(p).all() and torch.isfinite(q).all()
    assert any(e.fused for e in pairs[0][1]._entries) and not any(e.fused for e in pairs[1][1]._entries)
    assert _native.device_error() == 0
