"""The adjoint engine's tensor forward sweep, one launch per stage over all
parameter vectors, and its checkpoints as the stages' own inputs and outputs: gradients against the
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


# batch sizes around the SM count and sizes with fewer tiles than thread groups
@pytest.mark.parametrize('n,layers,batch', [(13, 2, 1), (13, 2, 200), (14, 2, 152), (16, 2, 37),
                                            (17, 1, 153), (20, 2, 5), (22, 2, 2), (23, 1, 2)])
def test_batched_forward_against_cuda_core_stages(rt, n, layers, batch):
    from qgate_gb300 import _native as nat
    e, g = _run(n, layers, batch, np.float32, 5)
    nat.set_tensor_blocks(False)
    try:
        e0, g0 = _run(n, layers, batch, np.float32, 5)
    finally:
        nat.set_tensor_blocks(True)
    assert np.max(np.abs(e - e0)) < 1e-5 * n
    assert np.max(np.abs(g - g0)) < 1e-5


@pytest.mark.parametrize('n', [13, 18])
def test_batch_is_its_vectors(rt, n):
    """A vector's energy in a batch is the one it has alone (the forward sweep adds
    nothing across vectors and in no other order: equal to the last bit)."""
    from qgate_gb300 import adjoint
    c = adjoint.hardware_efficient_ansatz(n, 2)
    p = np.random.default_rng(n).uniform(-3, 3, (7, c.n_params))
    h = adjoint.PauliSum.ising_chain(n)
    e, _ = adjoint.expectation_and_gradient(c, p, h, np.float32, 3, False)
    for b in range(7):
        e1, _ = adjoint.expectation_and_gradient(c, p[b:b + 1], h, np.float32, 3, False)
        assert e[b] == e1[0]


@pytest.mark.parametrize('dtype,bar', [(np.float32, 1e-5), (np.float64, 1e-10)], ids=['c64', 'c128'])
@pytest.mark.parametrize('n', [3, 9, 12, 14])
@pytest.mark.parametrize('every', [1, 2, 3, 7, 1000])
def test_checkpoints_change_nothing(rt, n, every, dtype, bar):
    e0, g0 = _run(n, 2, 3, dtype, 0)
    e, g = _run(n, 2, 3, dtype, every)
    ef, _ = _run(n, 2, 3, dtype, every, gradient=False)
    assert np.max(np.abs(e - e0)) < bar * n and np.max(np.abs(ef - e0)) < bar * n
    assert np.max(np.abs(g - g0)) < bar


@pytest.mark.parametrize('dtype,bar', [(np.float32, 1e-5), (np.float64, 1e-10)], ids=['c64', 'c128'])
@pytest.mark.parametrize('n', [8, 13])
def test_a_shared_parameter_gets_the_sum(rt, n, dtype, bar):
    """One parameter in every rotation: its gradient is the sum of those of a
    circuit with a parameter each, with targets and controls on the lowest and the
    highest lanes and stages with and without rotations."""
    from qgate_gb300 import adjoint
    one, many = adjoint.ParamCircuit(n), adjoint.ParamCircuit(n)
    rng = np.random.default_rng(n)
    for k in range(30):
        q, c = (int(x) for x in rng.permutation(n)[:2])
        for circ, p in ((one, 0), (many, k)):
            (circ.rx, circ.ry, circ.rz)[k % 3](q, p, (c,) if k % 4 == 0 else ())
            if k % 5 == 0:
                circ.cx(c, q)
                circ.cx(q, (q + 1) % n)
                circ.gate('H', c)
    h = adjoint.PauliSum.ising_chain(n).add(0.3, [(0, 'Y'), (n - 1, 'Y')]).add(0.2, [(1, 'Y')])
    for every in (0, 1, 2):
        e1, g1 = adjoint.expectation_and_gradient(one, np.full((2, 1), 0.37), h, dtype, every)
        em, gm = adjoint.expectation_and_gradient(many, np.full((2, 30), 0.37), h, dtype, every)
        assert np.max(np.abs(e1 - em)) < bar * n
        assert np.max(np.abs(g1[:, 0] - gm.sum(1))) < bar * 30
