"""The complex128 tensor stage's fixed-point phases (tests/cpp/phase_check.cpp):
a phase whose part lies on the tie of the table's first rounding keeps its sign
when the kernel negates the table's low word.  Bound, in units of the tile's
integers: half a unit of rounding, at most one (2^31 2^31 2^-62) for each of the
two dropped products of low words, and 2^52 times the table's 2^-62 for each of
the two parts (2^-9), below 2.51 in all."""
import os
import shutil
import subprocess

import pytest

from tests.test_cpu_planner import CSRC, ROOT, _cuda_include


def test_phase_products_are_rounded_once(tmp_path):
    cxx, inc = shutil.which('g++'), _cuda_include()
    if not cxx or not inc:
        pytest.skip('needs g++ and the CUDA headers')
    exe = str(tmp_path / 'phase_check')
    subprocess.run([cxx, '-O1', '-std=c++17', '-ffp-contract=off', '-fopenmp', '-I', CSRC, '-I',
                    os.path.join(ROOT, 'include'), '-I', inc,
                    os.path.join(ROOT, 'tests', 'cpp', 'phase_check.cpp'), '-o', exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    got = dict(line.split() for line in out.strip().splitlines())
    assert float(got['worst']) <= 2.51
    assert 2147483000. < float(got['most']) <= 2147483647.
