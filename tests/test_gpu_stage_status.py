"""A tensor stage's wait that gave up is told by the next call that returns results,
not by qg_tensor_stage_status alone: the status is set as a kernel would set it
(complex64 and complex128 stages), every kind of result raises, the cause is kept
until it is cleared, and the engine works on afterwards."""
import numpy as np
import pytest

from tests.gpu_helpers import Lane, abs2, apply_ops, new_state, null

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('status', [1, 2, 4, 1 << 8, 2 << 8, 0x101])
def test_results_raise_until_cleared(rt, status):
    from qgate_gb300 import _native as nat, adjoint
    assert nat.tensor_stage_status() == 0
    n = 14
    qs = new_state(rt, n, np.float64)
    apply_ops(qs, [('g', 'H', (), False, q, ()) for q in range(n)])
    want = qs.get_raw()
    getter = rt.create_qubits_states_getter(np.float64)
    lanes = [(qs, [Lane(q, q) for q in range(n)])]
    h = adjoint.PauliSum.ising_chain(4)
    c = adjoint.hardware_efficient_ansatz(4, 1)

    def pool():
        getter.create_sampling_pool(list(range(n)), n, 0, lanes, []).delete()
    results = [
        qs.get_raw,
        qs.processor.synchronize,
        lambda: qs.processor.calc_probability(qs, 0),
        lambda: qs.processor.calc_pauli_expectation(qs, 1, 1),
        lambda: getter.get_states(np.empty(1 << n, np.complex128), 0, null, lanes, [], 1 << n, 0, 1),
        lambda: getter.get_states(np.empty(1 << n, np.float64), 0, abs2, lanes, [], 1 << n, 0, 1),
        pool,
        lambda: adjoint.expectation_and_gradient(c, np.zeros((1, c.n_params)), h, np.float32, 0),
    ]
    nat.call('qg_tensor_stage_raise', status)
    try:
        for call in results:
            for _ in range(2):  # it stays
                with pytest.raises(RuntimeError, match='wait gave up'):
                    call()
        assert nat.tensor_stage_status() == status
    finally:
        nat.tensor_stage_status(reset=True)
    for call in results:
        call()
    assert nat.tensor_stage_status() == 0 and np.array_equal(qs.get_raw(), want)
    qs.delete()
