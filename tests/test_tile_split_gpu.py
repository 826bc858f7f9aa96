"""The fp32 kernel A that keeps a tile's first 8192 elements in registers and the rest in shared memory, against the
CPU oracle where it can go wrong: tiles that end around that border, short octets, buffers that start anywhere, every
quantisation block size, and selections that leave the fast route."""
import pytest
import torch

import cases
from ista_daslab_optimizers_b200 import synthetic as S

pytestmark = pytest.mark.gpu

DBS = 29056
SIZES = (8184, 8191, 8192, 8193, 8200, DBS - 1, DBS, DBS + 8192 + 8, 2 * DBS + 8195)


def _gradient(kind, n, step):
    g = S.normal_tensor(31 + step, n, n, 1e-3)
    if kind == 'ties':                                   # more equal magnitudes than the candidate list holds
        g[::3] = 2e-3 * torch.sign(g[::3])
    elif kind == 'border':                               # everything that is selected sits around the border
        g[8000:8400] *= 100.0
    elif kind == 'few':
        g.zero_()
        g[:: max(1, n // 5)] = -1.5
    elif kind == 'inf':
        g[n // 2] = float('inf')
    return g


@pytest.mark.parametrize('kind,qbs,k_init,alpha,skip', [
    ('normal', 64, 0.01, 0.0, 0), ('normal', 64, 0.01, 0.0, 3), ('normal', 8, 0.02, 0.0, 0), ('normal', 16, 0.005, 0.0, 4),
    ('normal', 128, 0.05, 0.0, 0), ('normal', 64, 0.0647, 0.0, 0),       # k = 1880, the largest this kernel takes
    ('normal', 32, 0.01, -2.0, 0), ('ties', 64, 0.02, 0.0, 0), ('ties', 64, 0.05, -2.0, 1), ('border', 64, 0.01, 0.0, 0),
    ('few', 64, 0.01, 0.0, 0), ('inf', 64, 0.01, 0.0, 0)])
def test_split_tile_matches_oracle(kind, qbs, k_init, alpha, skip):
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    from oracle.microadam_oracle import MicroAdamOracle
    hyper = dict(m=4, lr=1e-3, quant_block_size=qbs, k_init=k_init, weight_decay=0.1, alpha=int(alpha))
    buffers = [S.normal_tensor(30, i, n + skip, 0.02).cuda() for i, n in enumerate(SIZES)]
    params = [torch.nn.Parameter(b[skip:]) for b in buffers]
    cpu = [p.detach().cpu().clone() for p in params]
    opt = MicroAdam(params, **hyper)
    ref = MicroAdamOracle(cpu, d_block_size=opt.d_block_size, **hyper)
    assert opt.d_block_size == DBS
    for step in range(1 if kind == 'inf' else 3):
        grads = [_gradient(kind, n, step) for n in SIZES]
        for p, g in zip(params, grads):
            p.grad = torch.empty(g.numel() + skip, device='cuda')[skip:].copy_(g)
        opt.step()
        ref.step([g.clone() for g in grads])
        assert all(e.fused for e in opt._entries)
        for i, (p, n) in enumerate(zip(params, SIZES)):
            a, b, used = opt.state[p], ref.state[i], -(-n // qbs)
            row = step % hyper['m']
            assert torch.equal(a['I'][row].cpu(), b['I'][row]), (n, step)
            for key, cut in (('error', None), ('min_vals', used), ('max_vals', used)):
                assert torch.equal(a[key][:cut].cpu().view(torch.uint8), b[key][:cut].view(torch.uint8)), (n, step, key)
            assert torch.equal(a['V'][row].cpu().view(torch.int16), b['V'][row].view(torch.int16)), (n, step)
            if kind != 'inf':                            # the update itself: the tolerance the parameters have everywhere
                rtol, atol = cases.param_tolerances(torch.float32, hyper['lr'])
                torch.testing.assert_close(p.detach().cpu(), cpu[i], rtol=rtol, atol=atol)
    assert _native.device_error() == 0


@pytest.mark.parametrize('rows', [8, 9, 17])
def test_sparse_rows_many_blocks(rows):
    """More top-k blocks than a cluster has warps, rows around the number fetched ahead."""
    from ista_daslab_optimizers_b200 import _native as N
    from oracle import microadam_oracle as O
    d, k_init = 131 * DBS + 777, 0.003
    geo = O.Geometry.make(d, DBS, k_init, 64)
    gen = torch.Generator().manual_seed(rows)
    few = geo.k - geo.topk_full_blocks_count * geo.k_block_size_many
    I = torch.empty(rows, geo.k, dtype=torch.int16)
    for r in range(rows):
        full = torch.rand(geo.topk_full_blocks_count, DBS, generator=gen).topk(geo.k_block_size_many, dim=1).indices.sort(dim=1).values
        tail = torch.rand(777, generator=gen).topk(few).indices.sort().values
        I[r] = torch.cat([full.reshape(-1), tail]).to(torch.int16)
    V = torch.randn(rows, geo.k, generator=gen).bfloat16()
    g, M, out = torch.randn(d, generator=gen), torch.randn(rows, generator=gen), torch.randn(d, generator=gen)
    dots, dots_g, out_g = torch.zeros(rows), torch.zeros(rows, device='cuda'), out.cuda()
    args = (d, rows, geo.k, geo.d_block_size, geo.k_block_size_many)
    O.sparse_rows_dot(*args, g, I, V, dots)
    N.sparse_rows_dot(*args, g.cuda(), I.cuda(), V.cuda(), dots_g)
    # a sum of k products of unit size in fp32: |error| <= k * 2^-24 * sum |v g| ~ 1e-4 * sqrt(k) for either order
    torch.testing.assert_close(dots_g.cpu(), dots, rtol=1e-4, atol=1e-4 * geo.k ** 0.5)
    O.sparse_rows_combine(*args, M, I, V, out)
    N.sparse_rows_combine(*args, M.cuda(), I.cuda(), V.cuda(), out_g)
    assert torch.equal(out.view(torch.int32), out_g.cpu().view(torch.int32))


def _rows(d, k_init, rows, seed):
    """A ring buffer of `rows` rows with random positions, ascending inside every block."""
    from oracle import microadam_oracle as O
    geo = O.Geometry.make(d, DBS, k_init, 64)
    gen = torch.Generator().manual_seed(seed)
    n_full = geo.topk_full_blocks_count if geo.d_index_topk > 0 else 0
    parts, at = [], 0
    while at < d:
        n = min(geo.d_block_size, d - at)
        k = geo.k_block_size_many if len(parts) < n_full else geo.k - n_full * geo.k_block_size_many
        parts.append(torch.rand(rows, n, generator=gen).topk(k, dim=1).indices.sort(dim=1).values)
        at += n
    return geo, torch.cat(parts, dim=1).to(torch.int16), torch.randn(rows, geo.k, generator=gen).bfloat16(), gen


@pytest.mark.parametrize('g_dtype,v_dtype', [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize('d,k', [(40, 1), (33, 33), (DBS, 2048), (DBS, 2049), (2 * DBS + 500, 683), (3 * DBS, 31), (20 * DBS + 777, 300),
                                 (127 * DBS, 33), (127 * DBS + 64, 33)])
def test_sparse_rows_dot_of_few_blocks(d, k, g_dtype, v_dtype):
    """Rows that one CTA takes, rows whose blocks are shared among a cluster's warps in parts, and where the two rules end."""
    from ista_daslab_optimizers_b200 import _native as N
    from oracle import microadam_oracle as O
    rows = 5
    geo, I, V, gen = _rows(d, (k - 0.5) / min(d, DBS), rows, d)
    assert geo.k_block_size_many == k
    g, V, dots = torch.randn(d, generator=gen).to(g_dtype), V.to(v_dtype), torch.zeros(rows, device='cuda')
    args = (d, rows, geo.k, geo.d_block_size, geo.k_block_size_many)
    N.sparse_rows_dot(*args, g.cuda(), I.cuda(), V.cuda(), dots)
    block = torch.arange(geo.k) // geo.k_block_size_many
    terms = V.double() * g.double()[block * geo.d_block_size + I.long()]
    # fp32 products and sums: at most k + 1 roundings of 2^-24, each of no more than the sum of the terms' magnitudes
    bound = (geo.k + 1) * 2.0 ** -24 * terms.abs().sum(dim=1)
    assert ((dots.cpu().double() - terms.sum(dim=1)).abs() <= bound).all()


def test_sparse_rows_of_a_last_block_with_the_most_entries():
    """The last, short block may have more entries than the others."""
    from ista_daslab_optimizers_b200 import _native as N
    d, rows, k_many, k_few = DBS + 5000, 3, 40, 4100
    gen = torch.Generator().manual_seed(7)
    I = torch.cat([torch.rand(rows, n, generator=gen).topk(k, dim=1).indices.sort(dim=1).values for n, k in ((DBS, k_many), (5000, k_few))], dim=1)
    V, g, M = torch.randn(rows, k_many + k_few, generator=gen).bfloat16(), torch.randn(d, generator=gen), torch.randn(rows, generator=gen)
    at = I + torch.tensor([0] * k_many + [DBS] * k_few)
    dots, out = torch.zeros(rows, device='cuda'), torch.zeros(d, device='cuda')
    args = (d, rows, k_many + k_few, DBS, k_many)
    N.sparse_rows_dot(*args, g.cuda(), I.to(torch.int16).cuda(), V.cuda(), dots)
    N.sparse_rows_combine(*args, M.cuda(), I.to(torch.int16).cuda(), V.cuda(), out)
    terms = V.double() * g.double()[at]
    assert ((dots.cpu().double() - terms.sum(dim=1)).abs() <= (k_many + k_few + 1) * 2.0 ** -24 * terms.abs().sum(dim=1)).all()
    want = torch.zeros(d, dtype=torch.float64)
    for r in range(rows):
        want[at[r]] += M[r].double() * V[r].double()
    torch.testing.assert_close(out.cpu().double(), want, rtol=1e-5, atol=1e-5)     # three fp32 products and sums of unit size


@pytest.mark.parametrize('out_dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('rows', [1, 3, 8])
@pytest.mark.parametrize('k', [383, 384, 385, 768, 769, 3000, DBS])
def test_sparse_rows_combine_of_long_rows(k, rows, out_dtype):
    """Blocks with more entries than a CTA has threads (several per thread and row), and a short last block beside them."""
    from ista_daslab_optimizers_b200 import _native as N
    from oracle import microadam_oracle as O
    d = DBS + 4001
    geo, I, V, gen = _rows(d, (k - 0.5) / DBS, rows, k)
    M, out = torch.randn(rows, generator=gen), torch.randn(d, generator=gen).to(out_dtype)
    out_g, args = out.cuda(), (d, rows, geo.k, geo.d_block_size, geo.k_block_size_many)
    O.sparse_rows_combine(*args, M, I, V, out)
    N.sparse_rows_combine(*args, M.cuda(), I.cuda(), V.cuda(), out_g)
    assert torch.equal(out.view(torch.uint8), out_g.cpu().view(torch.uint8))


@pytest.mark.parametrize('dtype,alpha', [(torch.float32, 0.5), (torch.bfloat16, 0.1), (torch.bfloat16, -2)])
@pytest.mark.parametrize('skip,qbs,offset', [(1, 64, 0.0), (3, 128, 0.0), (4, 8, 0.0), (0, 64, 0.0), (0, 64, 0.2), (2, 32, -1.0)])
def test_alpha_forms_on_slices_that_start_anywhere(dtype, alpha, skip, qbs, offset):
    """The octet-wide alpha forms of the update with unaligned parameters, whole and short last quantisation blocks, and
    residuals far from zero, whose statistics are coarse against a quantisation step (codes then change when they shrink)."""
    from ista_daslab_optimizers_b200 import MicroAdam
    from oracle.microadam_oracle import MicroAdamOracle
    sizes = (7, 200, 4096, DBS + 8 * 5, DBS + 1003)
    hyper = dict(m=3, lr=1e-3, quant_block_size=qbs, k_init=0.02, weight_decay=0.1, alpha=alpha)
    params = [torch.nn.Parameter(S.normal_tensor(40, i, n + skip, 0.02).to(dtype).cuda()[skip:]) for i, n in enumerate(sizes)]
    cpu = [p.detach().cpu().clone() for p in params]
    opt = MicroAdam(params, **hyper)
    ref = MicroAdamOracle(cpu, d_block_size=opt.d_block_size, **hyper)
    for step in range(4):
        grads = [(S.normal_tensor(41 + step, n, n, 1e-3) + (offset if step == 0 else 0.0)).to(dtype) for n in sizes]
        for p, g in zip(params, grads):
            p.grad = torch.empty(g.numel() + skip, dtype=dtype, device='cuda')[skip:].copy_(g)
        opt.step()
        ref.step([g.clone() for g in grads])
        for i, (p, n) in enumerate(zip(params, sizes)):
            a, b, used = opt.state[p], ref.state[i], -(-n // qbs)
            for key, cut in (('error', None), ('min_vals', used), ('max_vals', used)):
                assert torch.equal(a[key][:cut].cpu().view(torch.uint8), b[key][:cut].view(torch.uint8)), (n, step, key)
            rtol, atol = cases.param_tolerances(dtype, hyper['lr'])
            torch.testing.assert_close(p.detach().cpu().float(), cpu[i].float(), rtol=rtol, atol=atol)


@pytest.mark.parametrize('dtype,alpha', [(torch.float32, 0.5), (torch.bfloat16, 0.25), (torch.bfloat16, -2), (torch.float32, -2)])
@pytest.mark.parametrize('k,dense', [(3800, True), (3900, False)])
def test_alpha_forms_with_and_without_room_for_dense_arrays(k, dense, dtype, alpha):
    """The alpha forms scatter updates into dense arrays of the warps where the window's arrays leave room for them in shared
    memory, and look them up through the bitmap where they do not: both sides of that line, with a full window of 4 rows."""
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    from oracle.microadam_oracle import MicroAdamOracle
    rows = 4
    stride = (2 * k + 30 + 15) & ~15                     # window_adam.cu, wt_smem_bytes
    window = 8 * rows * k + rows * 2 * stride + 6 * 1024 + 2 * rows * k
    room = 4 * _native.get_max_floats_for_shared_memory_per_thread_block() - 4096
    assert window <= room and (window + 15 + 8192 <= room) == dense
    hyper = dict(m=rows, lr=1e-3, quant_block_size=64, k_init=(k - 0.5) / DBS, weight_decay=0.1, alpha=alpha)
    sizes = (DBS, DBS + 1003)
    params = [torch.nn.Parameter(S.normal_tensor(90, i, n, 0.02).to(dtype).cuda()) for i, n in enumerate(sizes)]
    cpu = [p.detach().cpu().clone() for p in params]
    opt = MicroAdam(params, **hyper)
    ref = MicroAdamOracle(cpu, d_block_size=opt.d_block_size, **hyper)
    for step in range(rows + 2):
        grads = [S.normal_tensor(91 + step, n, n, 1e-3).to(dtype) for n in sizes]
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        opt.step()
        ref.step([g.clone() for g in grads])
        for i, (p, n) in enumerate(zip(params, sizes)):
            a, b, used = opt.state[p], ref.state[i], -(-n // 64)
            assert a['k_block_size_many'] == k
            for key, cut in (('error', None), ('min_vals', used), ('max_vals', used)):
                assert torch.equal(a[key][:cut].cpu().view(torch.uint8), b[key][:cut].view(torch.uint8)), (n, step, key)
            rtol, atol = cases.param_tolerances(dtype, hyper['lr'])
            torch.testing.assert_close(p.detach().cpu().float(), cpu[i].float(), rtol=rtol, atol=atol)
    assert all(e.fused for e in opt._entries) and _native.device_error() == 0
