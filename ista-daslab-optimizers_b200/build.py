"""Builds libmicroadam_b200.so (sm_100a) in-tree with nvcc, and the native host side of the step with g++.

    python build.py [--verbose] [--force]

The CUDA runtime is linked statically, so loading the library needs no CUDA libraries; the
first call into it needs an NVIDIA driver.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, 'csrc')
OUT_DIR = os.path.join(HERE, 'ista_daslab_optimizers_b200', 'lib')
LIB_PATH = os.path.join(OUT_DIR, 'libmicroadam_b200.so')
HOST_SRC = os.path.join(HERE, 'csrc_host', 'step_plan.cpp')
INCLUDE = os.path.join(os.path.dirname(HERE), 'include')


def host_path() -> str:
    """The extension, next to its users.  It is compiled against the layout of torch's and Python's objects, so its file
    name carries their versions: for others it does not exist."""
    sys.path.insert(0, HERE)
    try:
        from ista_daslab_optimizers_b200._native import step_plan_path
    finally:
        sys.path.remove(HERE)
    return step_plan_path()


def _nvcc() -> str:
    for cand in (os.environ.get('NVCC'), shutil.which('nvcc'), '/usr/local/cuda/bin/nvcc'):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError('nvcc not found (set NVCC or put it on PATH)')


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith('.cu'))


def _inputs():
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [HOST_SRC]
    deps += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return deps


def up_to_date() -> bool:
    built = (LIB_PATH, host_path())
    if not all(os.path.exists(p) for p in built):
        return False
    t = min(os.path.getmtime(p) for p in built)
    return all(os.path.getmtime(p) <= t for p in _inputs())


def host_command():
    """The g++ line of the extension that walks the optimizer's tensors (it reads torch's tensors directly)."""
    import sysconfig
    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    return [os.environ.get('CXX', 'g++'), '-O2', '-std=c++17', '-fPIC', '-shared', '-I', INCLUDE, '-I', os.path.join(base, 'include'),
            '-I', os.path.join(base, 'include', 'torch', 'csrc', 'api', 'include'), '-I', os.path.join(cuda, 'include'),
            '-I', sysconfig.get_paths()['include'], HOST_SRC, '-o', host_path(), '-L', os.path.join(base, 'lib'),
            '-ltorch_python', '-lc10_cuda', '-lc10', '-ltorch_cpu']


def build(verbose: bool = False, force: bool = False) -> str:
    if not force and up_to_date():
        return LIB_PATH
    os.makedirs(OUT_DIR, exist_ok=True)
    objs = []
    obj_dir = os.path.join(HERE, 'build')
    os.makedirs(obj_dir, exist_ok=True)
    common = [_nvcc(), '-O3', '-std=c++17', '-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo',
              '-Xcompiler', '-fPIC', '-I', INCLUDE]
    if verbose:
        common += ['-Xptxas', '-v']
    if os.environ.get('MAB_STATS'):
        common += ['-DMAB_STATS']       # development-only tile statistics
    procs = [(HOST_SRC, subprocess.Popen(host_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True))]
    for src in sources():
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + '.o')
        objs.append(obj)
        procs.append((src, subprocess.Popen(common + ['-c', src, '-o', obj], stdout=subprocess.PIPE,
                                            stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f'--- {os.path.basename(src)}\n{out}\n')
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError('a compiler failed')
    link = [_nvcc(), '-shared', '-cudart', 'static', '-gencode', 'arch=compute_100a,code=sm_100a', '-o', LIB_PATH] + objs
    subprocess.run(link, check=True)
    return LIB_PATH


if __name__ == '__main__':
    ap = argparse.ArgumentParser()
    ap.add_argument('--verbose', action='store_true', help='print ptxas register / shared-memory usage')
    ap.add_argument('--force', action='store_true')
    args = ap.parse_args()
    print(build(verbose=args.verbose, force=args.force))
