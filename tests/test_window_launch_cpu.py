"""How the update kernel's tile form is launched (csrc/window_launch.cuh): the form that starts before kernel A ends only where every CTA has one
tile, also on a part of a GPU (it went by the tiles alone once: 100 tiles on 74 SMs would have updated wrong parameters), and kernel A with a CTA on
every SM lets only that form start early (the wide form took 10 us more so)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, '..', 'ista-daslab-optimizers_b200', 'csrc')


@pytest.mark.skipif(shutil.which('nvcc') is None, reason='needs nvcc')
def test_launch_plan(tmp_path):
    exe = str(tmp_path / 'window_launch_check')
    subprocess.run(['nvcc', '-std=c++17', '-gencode', 'arch=compute_100a,code=sm_100a', '-I', CSRC, '-o', exe,
                    os.path.join(HERE, 'window_launch_check.cu')], check=True)
    out = subprocess.run([exe], check=False, capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
