"""Gates with four to nine controls among ordinary ones, on states of one tile
and more, against the oracle (complex128 1e-12, complex64 8e-6: the parity bars
of fused circuits)."""
import numpy as np
import pytest

from oracle import statevec as sv
from tests.gpu_helpers import apply_ops, new_state, random_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [12, 13, 16])
@pytest.mark.parametrize('dtype', [np.float64, np.float32], ids=['c128', 'c64'])
def test_many_controls_among_fused_gates(rt, n, dtype):
    rng = np.random.default_rng(n)
    ops = []
    for k in range(4, 10):
        ops += random_ops(rng, n, 12)
        lanes = [int(q) for q in rng.permutation(n)[:k + 1]]
        ops.append(('g', 'RY' if k % 2 else 'U1', (0.9,), False, lanes[0], tuple(lanes[1:])))
    qs = new_state(rt, n, dtype)
    apply_ops(qs, ops)
    got = qs.get_raw()
    qs.delete()
    tol = 1e-12 if dtype == np.float64 else 8e-6
    assert np.max(np.abs(got - sv.run_ops(n, ops, np.complex128))) < tol
