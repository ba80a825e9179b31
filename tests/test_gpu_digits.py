"""The complex128 tensor stage (k_dstage) on the GPU: against the oracle and the
CUDA-core stages on states of one tile to many, all gate kinds, states of every
kind, matrices that are not unitary, and from a captured graph.  Bars: 1e-12 per
amplitude (complex128 parity) for unitary circuits; for the others 2^-39 of the
norm per gate, the worst case of one block's left-out digits, times the norm's
growth."""
import numpy as np
import pytest

from oracle import statevec as sv
from tests.gpu_helpers import apply_ops, new_state, random_ops

pytestmark = pytest.mark.gpu


@pytest.fixture
def nat():
    from qgate_gb300 import _native
    _native.set_tensor_blocks(True)  # at every size
    _native.timing_enable(True)
    _native.timing_read('', reset=True)
    yield _native
    assert _native.tensor_stage_status(reset=True) == 0
    _native.set_fusion(0)
    _native.timing_enable(False)


def _u3_cx(rng, n, depth):
    ops = []
    for _ in range(depth):
        ang = rng.uniform(0, 2 * np.pi, (n, 3))
        ops += [('g', 'U', tuple(ang[q]), False, q, ()) for q in range(n)]
        perm = rng.permutation(n)
        ops += [('g', 'X', (), False, int(perm[2 * k + 1]), (int(perm[2 * k]),))
                for k in range(n // 2)]
    return ops


@pytest.mark.parametrize('n', [12, 13, 14, 17, 20])
def test_against_the_oracle_and_the_cuda_core_stages(rt, nat, n):
    rng = np.random.default_rng(n)
    ops = _u3_cx(rng, n, 3) + random_ops(rng, n, 80, max_controls=4)
    for i in range(n):  # stages of mostly diagonal gates: phase ops
        ops.append(('g', 'H', (), False, i, ()))
        ops += [('g', 'U1', (np.pi / (1 << (j - i)),), False, i, (j,)) for j in range(i + 1, n)]
    want = sv.run_ops(n, ops, np.complex128)
    got = {}
    for on in (True, False):
        nat.set_tensor_blocks(on)
        qs = new_state(rt, n, np.float64)
        apply_ops(qs, ops)
        got[on] = qs.get_raw()
        qs.delete()
        assert (nat.timing_read('tstage', reset=True)[0] > 0) == on
    nat.set_tensor_blocks(True)
    assert np.max(np.abs(got[True] - want)) < 1e-12
    assert np.max(np.abs(got[True] - got[False])) < 1e-12


@pytest.mark.parametrize('kind', ['basis', 'uniform', 'orders', 'sparse', 'small'])
def test_states_of_every_kind(rt, nat, kind):
    n = 15
    rng = np.random.default_rng(3)
    v = rng.normal(size=(1 << n, 2)) @ np.array([1., 1j])
    if kind == 'basis':
        v[:] = 0
        v[12345] = 0.6 - 0.8j
    elif kind == 'uniform':
        v[:] = 1
    elif kind == 'orders':
        v *= 10. ** -rng.integers(0, 18, 1 << n)
    elif kind == 'sparse':  # most tiles all zero, the others partly
        v[rng.random(1 << n) < 0.999] = 0
    v /= np.linalg.norm(v)
    scale = 1e-200 if kind == 'small' else 1.
    ops = _u3_cx(rng, n, 2)
    want = sv.run_ops(n, ops, np.complex128, psi=v.copy())
    qs = new_state(rt, n, np.float64)
    qs.set_raw(v * scale)
    apply_ops(qs, ops)
    got = qs.get_raw() / scale
    qs.delete()
    assert np.max(np.abs(got - want)) < 1e-12


@pytest.mark.parametrize('graph', [False, True])
def test_matrices_that_are_not_unitary(rt, nat, graph):
    from qgate_gb300.compiled import CompiledCircuit
    n = 14
    rng = np.random.default_rng(9)
    gates, growth = [], 1.
    for k in range(60):
        m = rng.normal(size=(2, 2, 2)) @ np.array([1., 1j])
        m *= (1e-5, 1., 300.)[k % 3]
        if k % 7 == 0:
            m[1] = 0  # singular
        growth *= np.linalg.norm(m, 2)
        q = [int(x) for x in rng.permutation(n)[:2]]
        gates.append((m, False, q[0], [] if k % 4 else [q[1]]))
        growth *= 1. if k % 4 else max(1., 1. / np.linalg.norm(m, 2))
    v = rng.normal(size=(1 << n, 2)) @ np.array([1., 1j])
    v /= np.linalg.norm(v)
    want = sv.run_ops(n, [('m', m, [t], c) for m, _, t, c in gates], np.complex128, psi=v.copy())
    circ = CompiledCircuit(np.float64, gates, graph=graph)
    for _ in range(2):
        qs = new_state(rt, n, np.float64)
        qs.set_raw(v)
        circ.run(qs)
        got = qs.get_raw()
        qs.delete()
        assert np.linalg.norm(got - want) < len(gates) * 2. ** -39 * growth
    circ.delete()


def test_rows_of_very_different_norm_keep_their_precision(rt, nat):
    """A damping of 1e-12 on one lane between rotations, all in one stage: the
    damped half is as exact as the other (1e-12 of its norm).  (A later stage of
    unitary gates alone runs on the tensor cores again, whose digits are cut
    below the largest component of the whole tile.)"""
    from qgate_gb300.compiled import CompiledCircuit
    n = 12
    rng = np.random.default_rng(n)
    h = np.array([[1., 1.], [1., -1.]]) / np.sqrt(2.)
    damp = np.diag([1., 1e-12])
    gates = [(h, False, q, []) for q in range(n)] + [(damp, False, 5, [])]
    gates += [(h, False, q, [(q + 1) % n]) for q in range(n) if q != 5]
    v = rng.normal(size=(1 << n, 2)) @ np.array([1., 1j])
    v /= np.linalg.norm(v)
    want = sv.run_ops(n, [('m', m, [t], c) for m, _, t, c in gates], np.complex128, psi=v.copy())
    circ = CompiledCircuit(np.float64, gates, graph=False)
    qs = new_state(rt, n, np.float64)
    qs.set_raw(v)
    circ.run(qs)
    got = qs.get_raw()
    qs.delete()
    circ.delete()
    half = (np.arange(1 << n) >> 5 & 1) == 1
    for part in (half, ~half):
        assert np.linalg.norm((got - want)[part]) < 1e-12 * np.linalg.norm(want[part])


@pytest.mark.parametrize('n', [20, 21])
def test_default_by_size(rt, nat, n):
    nat.set_fusion(0)  # the defaults
    rng = np.random.default_rng(n)
    ops = _u3_cx(rng, n, 1)
    qs = new_state(rt, n, np.float64)
    apply_ops(qs, ops)
    got = qs.get_raw()
    qs.delete()
    assert (nat.timing_read('tstage', reset=True)[0] > 0) == (n >= 21)
    assert np.max(np.abs(got - sv.run_ops(n, ops, np.complex128))) < 1e-12


def test_a_nan_stays_in_its_tile_and_ends(rt, nat):
    n = 14
    v = np.full(1 << n, 2. ** -7, np.complex128)
    v[77] = np.nan
    qs = new_state(rt, n, np.float64)
    qs.set_raw(v)
    apply_ops(qs, [('g', 'H', (), False, q, ()) for q in range(12)])
    got = qs.get_raw()
    qs.delete()
    assert np.isnan(got[:4096]).all() and np.isfinite(got[4096:]).all()
