"""Reading one state in another lane order (k_permute) and summing lanes out
(k_marginal_stream) against numpy on the same amplitudes, over every form the
dispatch distinguishes: whole vectors, aligned and unaligned ranges, orders that
keep or move the low lanes, hidden lanes low, high and mixed.  Amplitudes come
back exactly; probabilities within the rounding of their own precision (complex64
3e-7 relative, complex128 4e-16) and sums within that of their largest term
count."""
import numpy as np
import pytest

from tests.gpu_helpers import CDT, Lane, abs2, new_state, null

pytestmark = pytest.mark.gpu

DTYPES = [np.float64, np.float32]
EPS = {np.float64: 4e-16, np.float32: 3e-7}


def _state(rt, n, dtype, seed):
    r = np.random.default_rng(seed)
    v = (r.normal(size=(1 << n, 2)) @ np.array([1., 1j])).astype(CDT[dtype])
    v /= np.linalg.norm(v)
    qs = new_state(rt, n, dtype)
    qs.set_raw(v)
    return qs, v.astype(CDT[dtype])


def _abs2(v):
    """|v|^2 with no rounding to speak of."""
    re, im = v.real.astype(np.longdouble), v.imag.astype(np.longdouble)
    return re * re + im * im


def _orders(n):
    r = np.random.default_rng(n)
    yield list(range(n))[::-1]
    yield [(q + 5) % n for q in range(n)]
    yield [int(q) for q in r.permutation(n)]
    yield list(range(5)) + [5 + int(q) for q in r.permutation(n - 5)]
    yield [1, 0] + list(range(2, n))


def _local(ext_of, index):
    out = np.zeros_like(index)
    for l, e in enumerate(ext_of):
        out |= ((index >> e) & 1) << l
    return out


@pytest.mark.parametrize('dtype', DTYPES, ids=['c128', 'c64'])
@pytest.mark.parametrize('n', [9, 10, 11, 14, 17])
def test_permuted_reads(rt, n, dtype):
    qs, v = _state(rt, n, dtype, n)
    getter = rt.create_qubits_states_getter(dtype)
    N = 1 << n
    for order in _orders(n):
        lanes = [(qs, [Lane(l, e) for l, e in enumerate(order)])]
        for start, count in [(0, N), (N // 2, N // 2), (N // 4, N // 4), (3, N // 2), (0, N - 5)]:
            want = v[_local(order, np.arange(start, start + count))]
            got = np.empty(count, v.dtype)
            getter.get_states(got, 0, null, lanes, [], count, start, 1)
            assert np.array_equal(got, want), (order, start, count)
            p = np.empty(count, dtype)
            getter.get_states(p, 0, abs2, lanes, [], count, start, 1)
            ref = _abs2(want)
            assert np.all(np.abs(p - ref) <= EPS[dtype] * ref)
    qs.delete()


@pytest.mark.parametrize('dtype', DTYPES, ids=['c128', 'c64'])
@pytest.mark.parametrize('n', [11, 12, 15, 19])
def test_marginals(rt, n, dtype):
    qs, v = _state(rt, n, dtype, 100 + n)
    p = _abs2(v).astype(np.float64)
    getter = rt.create_qubits_states_getter(dtype)
    r = np.random.default_rng(n)
    picks = [list(range(n)), list(range(n))[::-1], list(range(n - 1)), list(range(1, n)),
             list(range(4, n)), list(range(n - 4)), [0], [n - 1], list(range(8)),
             list(range(8, n)), [int(q) for q in r.permutation(n)[:n // 2]],
             [int(q) for q in r.permutation(n)[:n - 3]], [int(q) for q in r.permutation(n)]]
    for vis in picks:
        ext = [-1] * n
        for k, q in enumerate(vis):
            ext[q] = k
        got = getter.create_sampling_pool(
            list(range(len(vis))), len(vis), n - len(vis),
            [(qs, [Lane(q, e) for q, e in enumerate(ext)])], [],
            sampling_pool_factory=lambda prob, empty, order: prob)
        index = np.arange(1 << n)
        out = np.zeros_like(index)
        for k, q in enumerate(vis):
            out |= ((index >> q) & 1) << k
        want = np.bincount(out, weights=p, minlength=1 << len(vis))
        # each term's rounding, the result's own (returned in the state's
        # precision), and the FP64 sums'
        tol = EPS[dtype] * want + 2. ** -52 * (1 << (n - len(vis))) * want
        assert np.all(np.abs(got - want) <= 2 * tol), vis
    qs.delete()
