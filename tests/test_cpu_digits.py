"""The complex128 tensor stage emulated on the CPU in the kernel's own integer
arithmetic from launch plans (tests/cpp/digit_check.cpp): against the plans'
gates in FP64, within the worst-case bound of the digits left out, for states
and matrices of every kind the stage accepts; level sums stay exact in FP32, no
digit overflows its field, every slot table is a bijection and both ways of
storing a tile occur."""
import os
import shutil
import subprocess

import pytest

from tests.test_cpu_planner import CSRC, ROOT, _cuda_include

KINDS = ['gaussian', 'basis', 'uniform', 'orders', 'hadamard', 'tiny', 'single', 'shrink', 'grow',
         'projector',
         'qft', 'phases']


@pytest.fixture(scope='module')
def digits(tmp_path_factory):
    cxx, inc = shutil.which('g++'), _cuda_include()
    if not cxx or not inc:
        pytest.skip('needs g++ and the CUDA headers')
    exe = str(tmp_path_factory.mktemp('digits') / 'digit_check')
    subprocess.run([cxx, '-O2', '-std=c++17', '-ffp-contract=off', '-fopenmp', '-I', CSRC, '-I',
                    os.path.join(ROOT, 'include'), '-I', inc,
                    os.path.join(ROOT, 'tests', 'cpp', 'digit_check.cpp'), '-o', exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {line.split()[0]: line.split()[1:] for line in out.strip().splitlines()}


@pytest.mark.parametrize('kind', KINDS)
def test_emulated_digit_stage(digits, kind):
    ratio, rel, level = digits[kind]
    assert float(ratio) < 1.
    assert int(level) < 1 << 24
    # unitary circuits on states of any kind: far below the complex128 bar
    if kind not in ('shrink', 'grow', 'projector'):
        assert float(rel) < 1e-13


def test_digit_stage_structure(digits):
    assert int(digits['bad_digit'][0]) == 0 and int(digits['bad_table'][0]) == 0
    assert int(digits['direct'][0]) > 0 and int(digits['natural'][0]) > 0
    assert int(digits['phase_ops'][0]) > 0
