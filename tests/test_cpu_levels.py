"""The accumulators of the complex128 tensor stage hold their sums exactly
(tests/cpp/level_check.cpp): over Hadamard blocks with a phase, on tiles whose
digits all add up, the sums that have to be exact stay within 2^24 for any tile,
and the emulated result is off by at most what level 5 may round (16 accumulations
of two units of 2^-51 of the row's norm) and the digits cut off (as much again):
2^-45.  Some of the blocks need smaller inputs for that, and some do not.  With one set of accumulators per level the same inputs are off by more
than the complex128 bar of 1e-12."""
import os
import shutil
import subprocess

import pytest

from tests.test_cpu_planner import CSRC, ROOT, _cuda_include


def test_accumulators_are_exact(tmp_path):
    cxx, inc = shutil.which('g++'), _cuda_include()
    if not cxx or not inc:
        pytest.skip('needs g++ and the CUDA headers')
    exe = str(tmp_path / 'level_check')
    subprocess.run([cxx, '-O2', '-std=c++17', '-ffp-contract=off', '-fopenmp', '-I', CSRC, '-I',
                    os.path.join(ROOT, 'include'), '-I', inc,
                    os.path.join(ROOT, 'tests', 'cpp', 'level_check.cpp'), '-o', exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    got = {line.split()[0]: [float(x) for x in line.split()[1:]] for line in out.strip().splitlines()}
    assert got['bound'][0] <= 2 ** 24 and got['kernel'][1] <= 2 ** 24
    assert got['kernel'][0] < 2. ** -45
    assert got['per_level'][0] > 1e-12 and got['per_level'][1] > 2 ** 24  # the inputs are sharp
    assert 100 < got['lows'][0] < 2900
    src = open(os.path.join(CSRC, 'dstage.cu')).read()
    # the kernel's form is the emulated one
    assert 'kHalfCols = 7u * kLevelCols' in src and 'mma_f16_lane(dcol + 192u, da + kNext' in src
    assert '+ (int)d.op_low[b]' in src and 'emax + (int)d.op_low[0]' in src
