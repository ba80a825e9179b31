"""complex128 amplitudes far below their neighbours keep their own precision in
fused stages: under gates that only move or turn them, in products of small
rotations.  Per-amplitude relative
errors, at the default settings (21 lanes) and with every size on the tensor
stages; k_dstage's digits alone are cut below 2^-52 of a tile's largest."""
import numpy as np
import pytest

from oracle import statevec as sv
from tests.gpu_helpers import apply_ops, new_state, random_ops

pytestmark = pytest.mark.gpu

# tiles whose largest amplitude lies below 2^-45 stay on the digits: six blocks of 64
# terms of 2^-53 of it and as much for the matrix
FLOOR = 6 * 2. ** (-45 - 46)


@pytest.fixture(params=[(21, False), (16, True), (12, True)], ids=['default_21', 'forced_16', 'forced_12'])
def lanes(request):
    from qgate_gb300 import _native as nat
    n, forced = request.param
    if forced:
        nat.set_tensor_blocks(True)
    yield n
    assert nat.tensor_stage_status(reset=True) == 0
    nat.set_fusion(0)


def _wide_state(n, seed):
    r = np.random.default_rng(seed)
    v = r.normal(size=(1 << n, 2)) @ np.array([1., 1j])
    v *= 10. ** -r.uniform(0, 15, 1 << n)
    return v / np.linalg.norm(v)


def _run(rt, n, v, ops):
    qs = new_state(rt, n, np.float64)
    if v is not None:
        qs.set_raw(v)
    apply_ops(qs, ops)
    got = qs.get_raw()
    qs.delete()
    return got


def _moves(r, n, count, kinds):
    ops = []
    for k in range(count):
        q = [int(x) for x in r.permutation(n)[:3]]
        ctrl = tuple(q[1:1 + int(r.integers(0, 3))])
        if kinds[k % len(kinds)] == 'x':
            ops.append(('g', 'X' if k % 5 else 'Y', (), False, q[0], ctrl))
        else:
            ops.append(('g', 'U1', (float(r.uniform(0, 6)),), False, q[0], ctrl))
    return ops


@pytest.mark.parametrize('kinds', ['d', 'x', 'xd'])
def test_gates_that_only_move_and_turn(rt, lanes, kinds):
    """Each gate errs by 2^-46 of the amplitude at most (double-float products), and
    by 2^-97 where a part lies below 2^-74 (FP32's exponents)."""
    r = np.random.default_rng(7)
    v = _wide_state(lanes, 1)
    ops = _moves(r, lanes, 60, kinds)
    want = sv.run_ops(lanes, ops, np.complex128, psi=v.copy())
    got = _run(rt, lanes, v, ops)
    assert np.all(np.abs(got - want) <= 60 * (2. ** -46 * np.abs(want) + 2. ** -96))


def test_gates_on_some_lanes_keep_the_others_ratio(rt, lanes):
    """Mixing gates on lanes 0..3 of a product of a random state there and lanes of
    small rotations: what the other lanes scale down keeps its precision.  A stored
    amplitude lies within 2^16 of its tile's largest and errs by at most 64 terms
    of 2^-53 and as much for the matrix, 2^-46 of that, per fused block (two here)."""
    n, r = lanes, np.random.default_rng(5)
    low = r.normal(size=(16, 2)) @ np.array([1., 1j])
    low /= np.linalg.norm(low)
    v = low
    for q in range(4, n):
        a = 10. ** -r.uniform(0, 3)
        v = np.kron(np.array([1., a]) / np.hypot(1., a), v)
    ops = [('g', 'U', tuple(r.uniform(0, 6, 3)), False, q, ()) for q in range(4)]
    ops += [('g', 'X', (), False, 1, (0,)), ('g', 'RY', (0.7,), False, 0, ())]
    ops += [('g', 'U1', (0.3,), False, q, (q - 1,)) for q in range(5, n)]
    want = sv.run_ops(n, ops, np.complex128, psi=v.copy())
    got = _run(rt, n, v, ops)
    # the 16 amplitudes of a group mix with one another: against their largest
    top = np.abs(want).reshape(-1, 16).max(1)[:, None]
    err = np.abs(got - want).reshape(-1, 16)
    assert np.all(err <= 2 * 2. ** (16 - 46) * top + FLOOR)


@pytest.mark.parametrize('angle', [1e-7, 1e-3, 0.3])
def test_products_of_small_rotations(rt, lanes, angle):
    """Every amplitude of RY(a_q)|0> on all lanes, the rarest outcomes included.  A
    block's stored amplitudes as above; at most six blocks."""
    n, r = lanes, np.random.default_rng(3)
    a = angle * r.uniform(0.5, 1.5, n)
    want = np.ones(1, np.longdouble)
    for q in range(n):
        want = np.kron(np.array([np.cos(a[q] / 2), np.sin(a[q] / 2)], np.longdouble), want)
    got = _run(rt, n, None, [('g', 'RY', (float(a[q]),), False, q, ()) for q in range(n)])
    want = want.astype(np.float64)
    assert np.all(np.abs(got - want) <= 6 * 2. ** (16 - 46) * np.abs(want) + FLOOR)


@pytest.mark.parametrize('scale', [2. ** -200, 2. ** -88, 2. ** 90, 2. ** 200])
def test_scales_outside_fp32(rt, lanes, scale):
    """Tiles outside the FP32 pairs' range stay on the digits, wide or not: errors
    within 1e-12 of the norm as ever."""
    n, r = lanes, np.random.default_rng(2)
    v = _wide_state(n, 3)
    ops = random_ops(r, n, 40, max_controls=1)
    want = sv.run_ops(n, ops, np.complex128, psi=v.copy())
    got = _run(rt, n, v * scale, ops) / scale
    assert np.max(np.abs(got - want)) < 1e-12
