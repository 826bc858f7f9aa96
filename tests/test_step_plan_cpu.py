"""The native host side of the step (csrc_host/step_plan.cpp) where no GPU is needed: what it does when torch throws."""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest
import torch

from conftest import ROOT

_PRELUDE = textwrap.dedent(f"""
    import ctypes, sys, warnings
    sys.path.insert(0, {ROOT + '/ista-daslab-optimizers_b200'!r})
    import torch
    from ista_daslab_optimizers_b200 import _native as N
    plan = N.load_step_plan()

    def step(p, groups):
        return plan.plan_step(p, groups, 1, 64, 0, 0.9, 0.999, 1e-8)
""")


def _run(body):
    return subprocess.run([sys.executable, '-c', _PRELUDE + textwrap.dedent(body)], capture_output=True, text=True, timeout=300)


@pytest.mark.skipif(torch.cuda.is_available(), reason='needs a machine where torch finds no CUDA device')
def test_an_error_of_torch_is_an_exception_and_changes_nothing():
    """Asking torch for the current device fails here.  The process lives, and the ring position has not moved."""
    out = _run("""
        group = {'params': [], 'lr': 0.1, 'weight_decay': 0.0}
        empty = plan.plan_new([(group, [])], 0, 0, 4, 0, 0, 0, 0)
        try:
            step(empty, [group])
        except RuntimeError as e:
            print('raised', 'CUDA' in str(e))
        # a parameter that says it lies on a CUDA device
        from torch._subclasses.fake_tensor import FakeTensorMode
        warnings.simplefilter('ignore')
        with FakeTensorMode(allow_non_fake_inputs=True):
            p = torch.nn.Parameter(torch.empty(64, device='cuda'))
            p.grad = torch.empty(64, device='cuda')
        group, state, desc = {'params': [p], 'lr': 0.1, 'weight_decay': 0.0}, {'index': 2}, (N.MabTensor * 1)()
        full = plan.plan_new([(group, [(p, 2, state, 0)])], ctypes.addressof(desc), 1, 4, 0, 0, 0, 0)
        try:
            step(full, [group])
        except RuntimeError:
            print('raised', state)
    """)
    assert out.returncode == 0, out.stderr[-2000:]
    assert out.stdout.split('\n')[:2] == ['raised True', "raised {'index': 2}"]


def test_a_plan_keeps_no_cycle_alive():
    """A group or a parameter may refer to the optimizer that holds the plan: Python's collector sees through the plan, as it
    sees through the optimizer's own dictionaries."""
    out = _run("""
        import gc, weakref

        class Holder:
            pass

        def make(where):
            h, p, desc = Holder(), torch.nn.Parameter(torch.zeros(8)), (N.MabTensor * 1)()
            p.grad = torch.zeros(8)
            group, state = {'params': [p], 'lr': 0.1, 'weight_decay': 0.0}, {'index': 0}
            h.plan = plan.plan_new([(group, [(p, 2, state, 0)])], ctypes.addressof(desc), 1, 4, 0, 0, 0, 0)
            h.group = group
            if where == 'group':
                group['owner'] = h
            elif where == 'parameter':
                p.owner = h
            elif where == 'state':
                state['owner'] = h
            return weakref.ref(h), weakref.ref(p)

        for where in ('nowhere', 'group', 'parameter', 'state'):
            refs = make(where)
            gc.collect()
            print(where, [r() is None for r in refs])
    """)
    assert out.returncode == 0, out.stderr[-2000:]
    assert out.stdout.split('\n')[:4] == [f'{w} [True, True]' for w in ('nowhere', 'group', 'parameter', 'state')]


def test_package_without_the_built_files(tmp_path):
    """A clean checkout: the package imports, what needs no built file works, and an optimizer says how to build."""
    src = os.path.join(ROOT, 'ista-daslab-optimizers_b200', 'ista_daslab_optimizers_b200')
    dst = os.path.join(tmp_path, 'ista_daslab_optimizers_b200')
    shutil.copytree(src, dst, ignore=shutil.ignore_patterns('*.so', '__pycache__'))
    body = """
        import sys
        sys.path.insert(0, {0!r})
        import torch
        from ista_daslab_optimizers_b200 import MicroAdam, _native, block_split, sharding, synthetic
        assert _native.__file__.startswith({0!r})
        assert block_split(10, 4) == (2, 8) and len(sharding.plan_shards([29056 * 4], 29056, 64, 2)) == 2
        if {1}:
            _native.load = lambda *a: None           # the library alone is there
        try:
            MicroAdam([torch.nn.Parameter(torch.zeros(4))], m=1, lr=1.0, quant_block_size=64)
        except _native.NativeError as e:
            print('build.py' in str(e))
    """
    for library_there in (False, True):
        out = subprocess.run([sys.executable, '-c', textwrap.dedent(body.format(str(tmp_path), library_there))],
                             capture_output=True, text=True, timeout=300)
        assert out.stdout == 'True\n', out.stderr[-2000:]


def test_extension_of_another_torch_is_not_taken(monkeypatch):
    """The file name carries the versions of torch and Python: for others the build is not up to date, and nothing is loaded."""
    import build
    from ista_daslab_optimizers_b200 import _native
    assert build.host_path() == _native.step_plan_path() and os.path.exists(build.host_path())
    monkeypatch.setattr(_native, '_step_plan', None)
    monkeypatch.setattr(torch, '__version__', '0.0.1')
    assert not build.up_to_date()
    with pytest.raises(_native.NativeError, match='build.py'):
        _native.load_step_plan()
    monkeypatch.undo()
    monkeypatch.setattr(sys.implementation, 'cache_tag', 'cpython-300')
    assert not build.up_to_date()
