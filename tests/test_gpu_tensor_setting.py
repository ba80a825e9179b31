"""The tensor-stage setting: on again is the default again, also from a complex64
tuning result, and every size of complex128 state is asked for by name.  (On meant
every size for a while, and nothing but set_fusion(0) led back.)"""
import numpy as np
import pytest

from tests.gpu_helpers import apply_ops, new_state

pytestmark = pytest.mark.gpu


def _stages(rt, nat, dtype, n):
    nat.set_trace_replay(False)  # a replayed graph's launches are not timed
    nat.timing_enable(True)
    nat.timing_read('', reset=True)
    qs = new_state(rt, n, dtype)
    for q in range(n):
        apply_ops(qs, [('g', 'U', (0.3 + q, 0.2, 0.1), False, q, ()),
                       ('g', 'X', (), False, (q + 1) % n, (q,))])
    qs.get_raw()
    qs.delete()
    out = nat.timing_read('tstage')[0] > 0
    nat.timing_enable(False)
    nat.set_trace_replay(True)
    return out


@pytest.mark.parametrize('how', ['one', 'none', 'tuned', 'fusion', 'odd'])
def test_back_to_the_default(rt, how):
    from qgate_gb300 import _native as nat, autotune
    nat.set_tensor_blocks(False)
    assert not _stages(rt, nat, np.float32, 14) and not _stages(rt, nat, np.float64, 21)
    if how == 'one':
        nat.call('qg_set_tensor_blocks', 1)
    elif how == 'none':
        nat.set_tensor_blocks(None)
    elif how == 'tuned':
        autotune.apply(dict(prec=nat.PREC_FP32, tile_lanes=12, reg_lanes=4, cost_budget=0, tensor=1))
    elif how == 'fusion':
        nat.set_fusion(0)
    else:
        nat.call('qg_set_tensor_blocks', -3)
    assert _stages(rt, nat, np.float32, 14)
    assert not _stages(rt, nat, np.float64, 14) and _stages(rt, nat, np.float64, 21)


def test_every_size_by_name(rt):
    from qgate_gb300 import _native as nat, autotune
    nat.set_tensor_blocks(True)
    assert _stages(rt, nat, np.float64, 14)
    nat.set_fusion(0)
    autotune.apply(dict(prec=nat.PREC_FP64, tile_lanes=12, reg_lanes=3, cost_budget=0, tensor=1))
    assert _stages(rt, nat, np.float64, 14)
