"""k_dstage on the tiles whose digits add up most: (nearly) equal amplitudes under
Hadamards with a global phase, against FP64 (complex128 bar, 1e-12 of the norm).
With one accumulator per digit level these lost up to 4.9e-10."""
import numpy as np
import pytest

from oracle import statevec as sv
from tests.gpu_helpers import new_state

pytestmark = pytest.mark.gpu


def _phases(count):
    """Angles whose block has both parts' second digits near their largest."""
    r, out = np.random.default_rng(3), []
    while len(out) < count:
        phi = r.uniform(0, 2 * np.pi, 200000)
        x = np.stack([np.cos(phi), np.sin(phi)]) * 32 * np.sqrt(32.)
        hit = np.min(np.abs(x - np.rint(x)), axis=0) > 0.495
        out += [float(p) for p in phi[hit]]
    return out[:count]


@pytest.mark.parametrize('lanes', [(0, 1, 2, 3, 4), (3, 5, 7, 9, 11)])
def test_equal_amplitudes_under_hadamards_with_a_phase(rt, lanes):
    from qgate_gb300 import _native as nat
    from qgate_gb300.compiled import CompiledCircuit
    n, h = 12, np.array([[1., 1.], [1., -1.]]) / np.sqrt(2.)
    r = np.random.default_rng(1)
    nat.set_tensor_blocks(True)
    try:
        worst = 0.
        for k, phi in enumerate(_phases(24)):
            gates = [((np.exp(1j * phi) if q == lanes[0] else 1.) * h, False, q, []) for q in lanes]
            circ = CompiledCircuit(np.float64, gates, graph=False)
            for sign in (1., -1.):
                m = r.uniform(1.9, 1.94) * (1. + (1e-4 if k % 2 else 0.) * r.uniform(-.5, .5, (2, 1 << n)))
                v = (m[0] + 1j * sign * m[1]) * 2. ** -8
                want = sv.run_ops(n, [('m', g, [t], c) for g, _, t, c in gates], np.complex128,
                                  psi=v.copy())
                qs = new_state(rt, n, np.float64)
                qs.set_raw(v)
                circ.run(qs)
                worst = max(worst, np.linalg.norm(qs.get_raw() - want) / np.linalg.norm(v))
                qs.delete()
            circ.delete()
        assert nat.tensor_stage_status() == 0
    finally:
        nat.set_fusion(0)
    assert worst < 1e-12
