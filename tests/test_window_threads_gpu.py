"""The update kernel's threads per CTA follow the number of tiles and the window (window_adam.cu, threads_of): a launch of many tiles and
launches of one tile each sum every position's window in the same order, so they give the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DBS = 29056


@pytest.mark.parametrize('alpha,weight_decay,dtype', [(0, 0.0, torch.float32), (0, 0.1, torch.float32), (0.5, 0.1, torch.float32), (-2, 0.0, torch.bfloat16), (0.5, 0.0, torch.bfloat16)])
@pytest.mark.parametrize('rows,k,per_sm', [(3, 256, 1), (3, 257, 2), (3, 384, 3), (3, 385, 3), (10, 256, 3), (10, 291, 10), (10, 385, 1), (20, 291, 3), (3, 2500, 2)])
def test_many_tiles_equal_single_tiles(rows, k, per_sm, alpha, weight_decay, dtype):
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    from ista_daslab_optimizers_b200.compat import ista_daslab_cuda_tools as tools
    # as many tiles as the rule's lines lie at, and one more: full ones, and a short one with an element more than whole octets
    sizes = ((per_sm * tools.get_sm_count() - 1) * DBS, DBS, DBS // 2 + 9)
    hyper = dict(m=rows, lr=1e-3, quant_block_size=64, k_init=(k - 0.5) / DBS, alpha=alpha, weight_decay=weight_decay)
    gen = torch.Generator(device='cuda').manual_seed(k)
    whole = [torch.nn.Parameter(torch.empty(n, dtype=dtype, device='cuda').normal_(0.0, 0.02, generator=gen)) for n in sizes]
    alone = [torch.nn.Parameter(p.detach()[at:at + DBS].clone()) for p in whole[:2] for at in (0, (p.numel() // DBS - 1) * DBS)]
    alone.append(torch.nn.Parameter(whole[2].detach().clone()))
    views = [(0, 0), (0, (sizes[0] // DBS - 1) * DBS), (1, 0), (1, 0), (2, 0)]
    opt, opts = MicroAdam(whole, **hyper), [MicroAdam([p], **hyper) for p in alone]
    for step in range(rows + 1):
        for p in whole:
            p.grad = torch.empty(p.numel(), dtype=dtype, device='cuda').normal_(0.0, 1e-3, generator=gen)
        opt.step()
        for q, o, (i, at) in zip(alone, opts, views):
            q.grad = whole[i].grad[at:at + q.numel()].clone()
            o.step()
            assert opt.state[whole[0]]['k_block_size_many'] == k
            assert torch.equal(whole[i].detach()[at:at + q.numel()].view(torch.uint8), q.detach().view(torch.uint8)), (step, i, at)
    assert _native.device_error() == 0


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('skip', [0, 1, 2, 3, 5, 7])
def test_decay_of_slices_that_start_anywhere(dtype, skip):
    """The weight decay alone (zero gradients): parameters that start anywhere in a buffer, shorter than the elements before the first vector and longer
    than a block.  Exact: one rounded product per step, and what lies around the slices stays.  (bf16 windows of more than a few rows of 5 %
    leave the form that keeps the block in shared memory.)"""
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    sizes = (1, 2, 3, 7, 8, 9, 15, 16, 17, 250, DBS - 1, DBS, DBS + 1, 3 * DBS + 21)
    gen = torch.Generator(device='cuda').manual_seed(skip)
    buffers = [torch.empty(n + skip + 9, dtype=dtype, device='cuda').normal_(0.0, 0.02, generator=gen) for n in sizes]
    params = [torch.nn.Parameter(b[skip:skip + n]) for b, n in zip(buffers, sizes)]
    expected = [b.clone() for b in buffers]
    opt = MicroAdam(params, m=10, lr=1e-2, quant_block_size=64, k_init=0.05, weight_decay=1.0)
    decay = torch.tensor(1.0 - 1e-2, dtype=torch.float32, device='cuda')
    for step in range(11):
        for p in params:
            p.grad = torch.zeros_like(p)
        opt.step()
        for e, n in zip(expected, sizes):
            e[skip:skip + n] = (e[skip:skip + n].float() * decay).to(dtype)
        for b, e in zip(buffers, expected):
            assert torch.equal(b.view(torch.uint8), e.view(torch.uint8)), (step, b.numel())
    assert _native.device_error() == 0
