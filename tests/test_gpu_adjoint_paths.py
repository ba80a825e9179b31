"""The adjoint engine's forward sweep on either side of its rule (tensor stages
from 23 qubits on and 64 gates per checkpoint segment, CUDA-core stages below)
and its checkpoints as the stages' own inputs and outputs: gradients against the
run without tensor stages or without checkpoints (complex64 1e-5, complex128
1e-10: the bars of test_gpu_adjoint.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(n, layers, batch, dtype, every, gradient=True):
    from qgate_gb300 import adjoint
    c = adjoint.hardware_efficient_ansatz(n, layers)
    p = np.random.default_rng(n).uniform(-3, 3, (batch, c.n_params))
    return adjoint.expectation_and_gradient(c, p, adjoint.PauliSum.ising_chain(n), dtype, every,
                                            gradient)


@pytest.mark.parametrize('n,layers', [(22, 2), (23, 1), (23, 2)])
def test_forward_rule_against_cuda_core_stages(rt, n, layers):
    from qgate_gb300 import _native as nat
    e, g = _run(n, layers, 2, np.float32, 0)
    nat.set_tensor_blocks(False)
    try:
        e0, g0 = _run(n, layers, 2, np.float32, 0)
    finally:
        nat.set_tensor_blocks(True)
    assert np.max(np.abs(e - e0)) < 1e-5 * n
    assert np.max(np.abs(g - g0)) < 1e-5


@pytest.mark.parametrize('dtype,bar', [(np.float32, 1e-5), (np.float64, 1e-10)], ids=['c64', 'c128'])
@pytest.mark.parametrize('n', [3, 9, 12, 14])
@pytest.mark.parametrize('every', [1, 2, 3, 7, 1000])
def test_checkpoints_change_nothing(rt, n, every, dtype, bar):
    e0, g0 = _run(n, 2, 3, dtype, 0)
    e, g = _run(n, 2, 3, dtype, every)
    ef, _ = _run(n, 2, 3, dtype, every, gradient=False)
    assert np.max(np.abs(e - e0)) < bar * n and np.max(np.abs(ef - e0)) < bar * n
    assert np.max(np.abs(g - g0)) < bar
