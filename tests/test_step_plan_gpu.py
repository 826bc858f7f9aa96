"""The native host side of the step (csrc_host/step_plan.cpp) against the Python side it stands in for: the same bits,
and the Python side again whenever something about the parameters changes between steps."""
import ctypes
import subprocess
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _optimizer(dtype, **hyper):
    from ista_daslab_optimizers_b200 import MicroAdam
    gen = torch.Generator(device='cuda').manual_seed(3)
    params = [torch.nn.Parameter(torch.empty(n, device='cuda').normal_(0, 0.02, generator=gen).to(dtype)) for n in (7, 4096, 29056 + 72, 300)]
    opt = MicroAdam([{'params': params[:3]}, {'params': params[3:], 'lr': 5e-4}], m=4, lr=1e-3, quant_block_size=64, weight_decay=0.1, **hyper)
    return opt, params


def _same(a, b, pa, pb):
    for p, q in zip(pa, pb):
        assert torch.equal(p.detach(), q.detach())
        assert a.state[p].get('index') == b.state[q].get('index')
        for key in ('I', 'V', 'error', 'min_vals', 'max_vals'):
            if key in a.state[p]:
                assert torch.equal(a.state[p][key], b.state[q][key]), key
    assert a.steps == b.steps


@pytest.mark.parametrize('dtype,hyper', [(torch.float32, {}), (torch.bfloat16, {}), (torch.float32, {'alpha': 0.5})])
def test_native_step_follows_every_change(dtype, hyper):
    """Gradients that come, go and move, a learning rate that becomes a tensor, a parameter added, state loaded back."""
    (a, pa), (b, pb) = _optimizer(dtype, **hyper), _optimizer(dtype, **hyper)
    gen = torch.Generator(device='cuda').manual_seed(4)
    native = 0
    for t in range(9):
        for i, (p, q) in enumerate(zip(pa, pb)):
            g = torch.empty(p.shape, device='cuda').normal_(0, 1e-3, generator=gen).to(dtype)
            skip = t in (3, 4) and i == 1
            p.grad, q.grad = (None, None) if skip else (g, g.clone())
        if t == 2:
            a.param_groups[1]['lr'] = b.param_groups[1]['lr'] = torch.tensor(2e-4)
        if t == 6:
            extra = torch.empty(1000, device='cuda').normal_(0, 0.02, generator=gen).to(dtype)
            for opt, ps in ((a, pa), (b, pb)):
                ps.append(torch.nn.Parameter(extra.clone()))
                ps[-1].grad = extra.clone()
                opt.add_param_group({'params': [ps[-1]]})
        if t == 8:
            a.load_state_dict(a.state_dict())
        plan = a._plan
        a.step()
        native += plan is not None and a._plan is plan
        b._plan = None                   # the Python side every time
        b.step()
        torch.cuda.synchronize()
        _same(a, b, pa, pb)
    assert native >= 3                   # steps 1, 2, 4 and 7 find the parameters as the step before left them


def test_step_hooks_and_non_contiguous_gradients():
    """Hooks registered on the optimizer run around the native step as well; what the Python side refuses stays refused."""
    from ista_daslab_optimizers_b200 import _native as N
    opt, params = _optimizer(torch.float32)
    seen = []
    for p in params:
        p.grad = torch.ones_like(p)
    opt.step()
    assert opt._plan is not None
    handle = opt.register_step_post_hook(lambda *a: seen.append(opt.steps))
    opt.step()
    handle.remove()
    opt.step()
    assert seen == [2] and opt.steps == 3
    params[1].grad = torch.ones(2 * params[1].numel(), device='cuda')[::2]
    with pytest.raises(N.NativeError, match='contiguous'):
        opt.step()


def test_other_threads_run_while_the_library_is_called(tmp_path):
    """The call into the library may wait for the GPU (a full launch queue, a large descriptor table): Python's global lock is
    not held meanwhile.  A host function that sleeps stands in for the library."""
    from ista_daslab_optimizers_b200 import _native
    _step_plan = _native.load_step_plan()
    src, lib = tmp_path / 'slow.c', tmp_path / 'slow.so'
    src.write_text('#include <unistd.h>\nint slow(void* t, int n, const void* a, void* w, long long b, void* s) { usleep(400000); return n; }\n')
    subprocess.run(['gcc', '-shared', '-fPIC', '-o', str(lib), str(src)], check=True)
    slow = ctypes.CDLL(str(lib)).slow
    torch.zeros(1, device='cuda')
    group = {'params': [], 'lr': 0.1, 'weight_decay': 0.0}
    plan = _step_plan.plan_new([(group, [])], 0, 0, 4, 0, ctypes.cast(slow, ctypes.c_void_p).value, 0, 0)
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.005)

    thread = threading.Thread(target=tick)
    thread.start()
    time.sleep(0.05)
    begin = time.perf_counter()
    assert _step_plan.plan_step(plan, [group], 1, 64, 0, 0.9, 0.999, 1e-8) == 0
    end = time.perf_counter()
    stop.set()
    thread.join()
    assert end - begin >= 0.4
    assert sum(begin + 0.05 < t < end - 0.05 for t in ticks) >= 10      # of about 60; none with the lock held


def test_after_update_hook_runs_without_gradients():
    """A subclass may write parameters in `_after_update`, on native steps as on the others; so may a hook set on the object."""
    from ista_daslab_optimizers_b200 import MicroAdam

    class Halving(MicroAdam):
        def _after_update(self):
            assert not torch.is_grad_enabled()
            for group in self.param_groups:
                for p in group['params']:
                    p.mul_(0.5)

    p = torch.nn.Parameter(torch.ones(5000, device='cuda'))
    opt = Halving([p], m=4, lr=0.0, quant_block_size=64)
    p.grad = torch.ones_like(p)
    for _ in range(3):
        opt.step()
    assert opt._plan is not None and torch.is_grad_enabled()
    assert torch.equal(p.detach(), torch.full_like(p, 0.125))
    q = torch.nn.Parameter(torch.ones(5000, device='cuda'))
    opt = MicroAdam([q], m=4, lr=0.0, quant_block_size=64)
    seen = []
    opt._after_update = lambda: seen.append(torch.is_grad_enabled())
    q.grad = torch.ones_like(q)
    for _ in range(3):
        opt.step()
    assert seen == [False] * 3
