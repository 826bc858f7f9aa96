"""The number of loose quantisation blocks a tile touches, for blocks of up to 2^30 elements: the function the kernels call, on the
host (a tile near the end of a block of 2^30 once made 32-bit arithmetic overflow)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, '..', 'ista-daslab-optimizers_b200', 'csrc')


@pytest.mark.skipif(shutil.which('nvcc') is None, reason='needs nvcc')
def test_blocks_touched_by_a_tile(tmp_path):
    exe = str(tmp_path / 'loose_blocks_check')
    subprocess.run(['nvcc', '-std=c++17', '-gencode', 'arch=compute_100a,code=sm_100a', '-I', CSRC, '-o', exe,
                    os.path.join(HERE, 'loose_blocks_check.cu')], check=True)
    out = subprocess.run([exe], check=False, capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
    assert 'mismatches 0' in out.stdout
