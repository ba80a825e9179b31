"""Every kernel that initialises mbarriers publishes them to the async proxy: the
thread that initialises also executes fence.mbarrier_init (mbar_fence_init) before
the block synchronises.  Bulk copies and tcgen05.commit arrive on the barriers
through that proxy; without the fence they may meet one that is not there yet.
Read from the sources, as the fault cannot be provoked safely on a GPU."""
import glob
import os
import re

import pytest

from tests.test_cpu_planner import CSRC


def _block(text, at):
    """The braces of the innermost `if (tid ...) {` around position `at`."""
    start = max(m.start() for m in re.finditer(r'if \(tid[^\n]*\{', text[:at]))
    depth, i = 0, text.index('{', start)
    for j in range(i, len(text)):
        depth += {'{': 1, '}': -1}.get(text[j], 0)
        if depth == 0:
            return i, j
    raise AssertionError('unbalanced braces')


def _inits():
    for path in sorted(glob.glob(os.path.join(CSRC, '*.cu'))):
        text = open(path).read()
        for m in re.finditer(r'\bmbar_init\(', text):
            yield pytest.param(text, m.start(),
                               id='%s:%d' % (os.path.basename(path), text.count('\n', 0, m.start()) + 1))


@pytest.mark.parametrize('text,at', list(_inits()))
def test_barriers_are_published_by_their_thread(text, at):
    i, j = _block(text, at)
    assert i < at < j
    assert re.search(r'mbar_fence_init\(\)|fence\.mbarrier_init', text[at:j])
