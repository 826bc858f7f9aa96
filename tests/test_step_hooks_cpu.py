"""Step hooks around MicroAdam.step(), whose usual wrapper is left out while nothing would see it.  (No parameter has a
gradient here, so that a step needs no GPU.)"""
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
