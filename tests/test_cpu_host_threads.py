"""Host loops use the whole OpenMP team, or helpers of their own (host_team.h).  An
OpenMP region with fewer threads than the last makes the runtime end the others,
and the next one that wants them all pays for new threads (150 to 230 us on
Grace): a 1 MB copy on four threads so slowed every larger copy after it."""
import glob
import os
import re
import shutil
import subprocess

import pytest

from tests.test_cpu_planner import CSRC, ROOT


def test_no_region_asks_for_part_of_the_team():
    for path in glob.glob(os.path.join(CSRC, '*.[ch]*')):
        for line in re.findall(r'#pragma omp[^\n]*', open(path).read()):
            assert 'num_threads' not in line, (os.path.basename(path), line)


def test_every_part_runs_once(tmp_path):
    cxx = shutil.which('g++')
    if not cxx:
        pytest.skip('needs g++')
    exe = str(tmp_path / 'team_check')
    subprocess.run([cxx, '-O2', '-std=c++17', '-fopenmp', '-I', CSRC,
                    os.path.join(ROOT, 'tests', 'cpp', 'team_check.cpp'), '-o', exe],
                   check=True, capture_output=True)
    for threads in ('1', '4', '16'):
        out = subprocess.run([exe], check=False, capture_output=True, text=True, timeout=60,
                             env=dict(os.environ, OMP_NUM_THREADS=threads)).stdout
        assert out.strip() == 'ok', (threads, out)
