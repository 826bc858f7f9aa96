"""Step hooks around MicroAdam.step(), whose usual wrapper is left out while nothing would see it.  (No parameter has a
gradient here, so that a step needs no GPU.)"""
import functools
import inspect

import pytest
import torch


@pytest.fixture
def make(monkeypatch):
    from ista_daslab_optimizers_b200 import MicroAdam, _native
    monkeypatch.setattr(_native, 'get_sm_count', lambda: 148)

    def build(cls=MicroAdam):
        return cls([torch.nn.Parameter(torch.zeros(4))], m=2, lr=1e-3, quant_block_size=64, d_block_size=64)
    return build


def _calls(opt):
    """What hooks see of the three ways to call step(), the optimizer itself left out."""
    seen = []
    closure = lambda: torch.tensor(3.0)                  # noqa: E731
    opt.register_step_pre_hook(lambda o, args, kwargs: seen.append(('before', args[1:], dict(kwargs))))
    opt.register_step_post_hook(lambda o, args, kwargs: seen.append(('after', args[1:], dict(kwargs))))
    results = [opt.step(), opt.step(closure), opt.step(closure=closure)]
    return [(when, [a is closure for a in args], list(kwargs)) for when, args, kwargs in seen], results


def test_hooks_see_the_call_as_it_was_made(make):
    opt = make()
    assert _calls(opt) == _calls(torch.optim.SGD([torch.nn.Parameter(torch.zeros(4))], lr=0.1))
    assert opt.steps == 3
    assert list(inspect.signature(opt.step).parameters) == ['closure']


def test_a_pre_hook_may_change_the_call(make):
    opt = make()
    opt.register_step_pre_hook(lambda o, args, kwargs: (args, {'closure': lambda: 7}))
    assert opt.step() == 7


@pytest.mark.parametrize('marked', [False, True], ids=['plain', 'functools.wraps'])
@pytest.mark.parametrize('made', ['before', 'after'])
def test_hooks_run_once_behind_a_wrapper_around_the_class(make, monkeypatch, made, marked):
    """A program may wrap `MicroAdam.step` for all optimizers, whether they exist already or not."""
    from ista_daslab_optimizers_b200 import MicroAdam
    if made == 'before':
        opt = make()
    own, wrapped = MicroAdam.step, []

    def wrapper(self, *args, **kwargs):
        wrapped.append(self)
        return own(self, *args, **kwargs)
    monkeypatch.setattr(MicroAdam, 'step', functools.wraps(own)(wrapper) if marked else wrapper)
    if made == 'after':
        opt = make()
    seen = []
    opt.register_step_post_hook(lambda *a: seen.append(opt.steps))
    opt.step()
    opt.step()
    assert seen == [1, 2] and len(wrapped) == 2


@pytest.mark.parametrize('times', [1, 2])
def test_hooks_run_once_around_a_step_of_a_subclass(make, times):
    from ista_daslab_optimizers_b200 import MicroAdam

    class Twice(MicroAdam):
        def step(self, closure=None):
            for _ in range(times):
                super().step(closure)

    opt, seen = make(Twice), []
    opt.register_step_post_hook(lambda *a: seen.append(opt.steps))
    opt.step()
    assert seen == [times] and not opt._hooks_run
