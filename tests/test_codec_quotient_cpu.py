"""The encoder's two-product quotient gives the codes of the defining division: a small C program goes through every 61st
mantissa of the step (all 2^23 take it about half a minute: argument 1), all code thresholds and their neighbourhood."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which('gcc') is None, reason='needs gcc')
def test_two_product_quotient_gives_the_codes_of_the_division(tmp_path):
    exe = str(tmp_path / 'codec_quotient_check')
    subprocess.run(['gcc', '-O2', '-march=native', '-ffp-contract=off', '-o', exe, os.path.join(HERE, 'codec_quotient_check.c'), '-lm'], check=True)
    out = subprocess.run([exe, '61'], check=False, capture_output=True, text=True, timeout=900)
    assert out.returncode == 0, out.stdout + out.stderr
    assert 'quotient mismatches 0' in out.stdout
