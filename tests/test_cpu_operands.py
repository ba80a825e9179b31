"""The complex128 blocks' operands, formed on the host threads (tests/cpp/
operands_check.cpp): the same bytes on one thread and on many, and matrices equal to
their gates' products (a few roundings of entries of at most 1: 1e-14)."""
import os
import shutil
import subprocess

import pytest

from tests.test_cpu_planner import CSRC, ROOT, _cuda_include


def test_operands_on_any_number_of_threads(tmp_path):
    cxx, inc = shutil.which('g++'), _cuda_include()
    if not cxx or not inc:
        pytest.skip('needs g++ and the CUDA headers')
    exe = str(tmp_path / 'operands_check')
    subprocess.run([cxx, '-O2', '-std=c++17', '-fopenmp', '-I', CSRC, '-I',
                    os.path.join(ROOT, 'include'), '-I', inc,
                    os.path.join(ROOT, 'tests', 'cpp', 'operands_check.cpp'), '-o', exe],
                   check=True, capture_output=True)
    got = []
    for threads in ('1', '3', '16'):
        out = subprocess.run([exe], check=True, capture_output=True, text=True,
                             env=dict(os.environ, OMP_NUM_THREADS=threads)).stdout
        got.append(dict(line.split() for line in out.strip().splitlines()))
    assert got[0]['hash'] == got[1]['hash'] == got[2]['hash']
    assert float(got[0]['worst']) < 1e-14
