"""block_topk by itself, where its routes change: blocks and one more than there are SMs, blocks around an octet, k around the acceptance window's
change and beyond the octets, more equal magnitudes than the candidate list or the direct ranking holds, infinities and NaN, fewer than k numbers in a
block (NaN fill the row up, at the lowest positions), x off alignment."""
import pytest
import torch

from ista_daslab_optimizers_b200 import synthetic as S

pytestmark = pytest.mark.gpu

DBS = 29056


def _expected(x, k_many, k_few):
    key = x.float().abs()
    key[key.isnan()] = -1.0
    rows = []
    for at in range(0, x.numel(), DBS):
        n = min(DBS, x.numel() - at)
        k = k_many if n == DBS else k_few
        rows.append(torch.sort(key[at:at + n], descending=True, stable=True).indices[:k].sort().values)
    return torch.cat(rows).to(torch.int16)


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('kind,k,tail,skip', [
    ('normal', 291, 0, 0), ('normal', 291, 1, 0), ('normal', 1024, 8191, 1), ('normal', 1025, 8192, 2), ('normal', 3632, 15, 0), ('normal', 3633, 16, 3),
    ('ties', 1453, 17, 0), ('ties', 33, 4099, 0), ('scales', 291, 777, 4), ('inf', 291, 4096, 0), ('inf', 1, 9, 0), ('nan', 291, 4097, 0),
    ('zeros', 291, 100, 0), ('cluster', 600, 64, 0), ('all_nan', 291, 33, 0), ('short', 291, 300, 1), ('short', 7264, 9, 0),
    ('equal', 291, 100, 0), ('equal', 14000, 7, 1), ('three', 291, 9, 0), ('normal', 29056, 50, 0), ('zeros', 29056, 1, 0), ('zeros', 9000, 13, 2)])
def test_block_topk_routes(dtype, kind, k, tail, skip):
    from ista_daslab_optimizers_b200 import _native as N
    for full in (2, N.get_sm_count(), N.get_sm_count() + 1):
        d, k_few = full * DBS + tail, max(1, tail // 7) if tail else 0
        x = S.normal_tensor(13, full, d, 1e-3)
        if kind == 'ties':
            x = (x * 2000.0).round() / 2000.0
        elif kind == 'scales':                           # no block's bound fits the next one
            x *= 2.0 ** ((torch.arange(d) // DBS * 5) % 13 - 6)
        elif kind == 'inf':
            x[5::977] = float('inf')
            x[9::1203] = float('-inf')
        elif kind == 'nan':
            x[3::16] = float('nan')
            x[DBS:DBS + 512] = float('nan')
        elif kind == 'zeros':
            x[:DBS] = 0.0
            x[DBS:2 * DBS] = 0.0
            x[DBS + 11:2 * DBS:4001] = 1e-3
        elif kind == 'equal':                            # one magnitude, either sign
            x = torch.sign(x) * 1e-3
        elif kind == 'three':                            # zeros and two magnitudes, the larger one rare
            x = torch.where(x.abs() > 2.9e-3, 2e-3, torch.where(x.abs() > 1e-3, 1e-3, 0.0)) * torch.sign(x)
        elif kind == 'all_nan':                          # nothing else in the blocks, and in the short one behind them
            x[DBS:] = float('nan')
        elif kind == 'short':                            # one number fewer than k, zeros among them, and none
            x[:DBS][torch.arange(DBS) % (DBS // (k - 1)) != 2] = float('nan')
            x[:DBS][2 + DBS // (k - 1) * (k - 1):] = float('nan')
            x[2:DBS // 2:DBS // (k - 1)] *= 0.0
            x[DBS:2 * DBS] = float('nan')
        elif kind == 'cluster':
            x[1000:1000 + k] *= 300.0
        x = x.to(dtype)
        g = torch.empty(d + skip, dtype=dtype, device='cuda')[skip:].copy_(x)
        out = torch.full((full * k + k_few + 8,), -7, dtype=torch.int16, device='cuda')      # (what a row held before must not stay in it)
        N.block_topk(d, DBS, k, k_few, g, out[:full * k + k_few])
        assert torch.equal(out[:full * k + k_few].cpu(), _expected(x, k, k_few)), full
        assert (out[full * k + k_few:] == -7).all()
