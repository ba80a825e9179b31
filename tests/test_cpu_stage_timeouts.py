"""The complex128 tensor stage's way out of a wait that gives up, read from its
source (a wait is not made to run out in a kernel that holds tensor memory):
each tile group decides by its own word, written before the barrier that its
threads read it after, so that no thread of a group leaves alone and the rest wait
for it for ever; and the polls that wait for a group's work count from its last
tile, so that they bound a wait and not a whole launch."""
import os
import re

from tests.test_cpu_planner import CSRC

SRC = re.sub(r'//[^\n]*', '', open(os.path.join(CSRC, 'dstage.cu')).read())


def test_each_group_decides_by_its_own_word():
    assert re.search(r'__shared__ int abort_sh\[2\];', SRC)
    uses = re.findall(r'abort_sh(\[\w+\])?', SRC.split('__shared__ int abort_sh[2];')[1])
    assert uses and all(u == '[g]' for u in uses)
    # set, then the group's barrier, then read: in that order, once each
    wait = SRC.index('abort_sh[g] = 1')
    read = SRC.index('(volatile int *)&abort_sh[g]')
    assert 'group_sync(gbar, kGT);' in SRC[wait:read]
    assert 'mbar_wait' not in SRC[wait:read]


def test_every_group_wait_is_skipped_once_one_gave_up():
    waits = re.findall(r'if \((ok && )?!mbar_wait\(smem_u32\(&bar_d\[', SRC)
    assert waits and all(waits)


def test_polls_count_from_the_last_tile():
    # two polls (products, operands), each reset by the groups' tile counters
    assert len(re.findall(r'beat = beat_sh\[0\] \+ beat_sh\[1\];\s*idle = 0;', SRC)) == 2
    assert re.search(r'for \(; tl < tiles && ok; tl \+= tstep\) \{\s*if \(lt == 0u\) beat_sh\[g\]', SRC)


def test_the_issuing_warp_decides_as_one():
    warp = SRC[SRC.index('the issuing' if 'the issuing' in SRC else 'elect_lane()'):]
    warp = warp[:warp.index('setmaxnreg.inc')]
    for call in re.findall(r'(\S*)\(?mbar_(?:wait|test)\(smem_u32\(&bar_(?:a|b|dfree)\[', warp):
        assert call.endswith('all('), call
