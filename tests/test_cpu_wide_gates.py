"""Gates on more lanes than a fused block (tests/cpp/wide_check.cpp): the stage
planner leaves them to passes of their own.  (A tensor stage holding one never
ended its block grouping.)"""
import os
import shutil
import subprocess

import pytest

from tests.test_cpu_planner import CSRC, ROOT, _cuda_include


def test_wide_gates_are_planned_outside_the_blocks(tmp_path):
    cxx, inc = shutil.which('g++'), _cuda_include()
    if not cxx or not inc:
        pytest.skip('needs g++ and the CUDA headers')
    exe = str(tmp_path / 'wide_check')
    subprocess.run([cxx, '-O1', '-std=c++17', '-fopenmp', '-I', CSRC, '-I',
                    os.path.join(ROOT, 'include'), '-I', inc,
                    os.path.join(ROOT, 'tests', 'cpp', 'wide_check.cpp'), '-o', exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout
    got = dict(line.split() for line in out.strip().splitlines())
    assert int(got['bad']) == 0
    assert int(got['wide']) > 100 and int(got['stages']) > 100
