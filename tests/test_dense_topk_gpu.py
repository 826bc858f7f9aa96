"""The bf16 kernel A where its candidate selection meets its limits: k around the change of the acceptance window, around
the largest k the candidate list is used for, and tiles whose large values crowd into few octets."""
import pytest
import torch

from ista_daslab_optimizers_b200 import synthetic as S

pytestmark = pytest.mark.gpu

DBS = 29056
SIZES = (DBS, 2 * DBS + 4096, 9000)


@pytest.mark.parametrize('kind', ['normal', 'clustered'])
@pytest.mark.parametrize('k', [582, 1024, 1025, 1453, 1536, 1537])
def test_dense_selection_matches_oracle(k, kind):
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    from oracle.microadam_oracle import MicroAdamOracle
    hyper = dict(m=3, lr=1e-3, quant_block_size=64, k_init=(k - 0.5) / DBS)
    params = [torch.nn.Parameter(S.normal_tensor(50, i, n, 0.02).bfloat16().cuda()) for i, n in enumerate(SIZES)]
    opt = MicroAdam(params, **hyper)
    ref = MicroAdamOracle([p.detach().cpu().clone() for p in params], d_block_size=opt.d_block_size, **hyper)
    for step in range(3):
        grads = [S.normal_tensor(51 + step, n, n, 1e-4) for n in SIZES]
        if kind == 'clustered':
            for g in grads:
                g[1000:1000 + 4 * k // 3] *= 50.0
        grads = [g.bfloat16() for g in grads]
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        opt.step()
        ref.step([g.clone() for g in grads])
        assert opt.state[params[0]]['k_block_size_many'] == k
        for i, (p, n) in enumerate(zip(params, SIZES)):
            a, b = opt.state[p], ref.state[i]
            assert torch.equal(a['I'][step].cpu(), b['I'][step]), (n, step)
            assert torch.equal(a['V'][step].cpu().view(torch.int16), b['V'][step].view(torch.int16)), (n, step)
            assert torch.equal(a['error'].cpu(), b['error']), (n, step)
    assert _native.device_error() == 0
