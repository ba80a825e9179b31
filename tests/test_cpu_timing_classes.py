"""Every class of launches that the engine times is one that timing_all reads and the
header names."""
import os
import re

from tests.test_cpu_planner import CSRC, ROOT


def test_classes_are_complete():
    timed = set(re.findall(r'timed\(d, "(\w+)"', open(os.path.join(CSRC, 'api.cpp')).read()))
    text = open(os.path.join(ROOT, 'qgate_gb300', '_native.py')).read()
    known = set(re.findall(r"'(\w+)'", text.split('KERNEL_CLASSES = (')[1].split(')')[0]))
    header = open(os.path.join(ROOT, 'include', 'qgate_gb300.h')).read()
    named = set(re.findall(r'\w+', header.split('(classes:')[1].split(')')[0]))
    assert timed and timed <= known and timed <= named
