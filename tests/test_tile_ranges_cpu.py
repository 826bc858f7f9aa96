"""The tiles of a persistent CTA: every tile once, and no SM with two more than another (they were spread evenly over the CTAs' numbers
once, which gave some SMs two of the longer ranges)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, '..', 'ista-daslab-optimizers_b200', 'csrc')


@pytest.mark.skipif(shutil.which('nvcc') is None, reason='needs nvcc')
def test_tiles_are_shared_out_evenly(tmp_path):
    exe = str(tmp_path / 'tile_range_check')
    subprocess.run(['nvcc', '-std=c++17', '-gencode', 'arch=compute_100a,code=sm_100a', '-I', CSRC, '-o', exe,
                    os.path.join(HERE, 'tile_range_check.cu')], check=True)
    out = subprocess.run([exe], check=False, capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
    assert 'violations 0' in out.stdout
