"""The work that users of the engine have it do, as measurable cases.

Every case goes through the public entry points as a user's program calls
them: the runtime plugin protocol (`gb300runtime`: one call per gate, as the
simulator front-end drives a runtime, then observations), the adjoint
gradients, the batched circuits and the OpenQASM front-end.

  circuit   a whole circuit from |0...0>, gate by gate, and its state or its
            probability vector read back.  `random`: layers of U3 on every
            qubit and CX on a random matching (the headline benchmark);
            `qft`: the QFT of a basis state, without the final swaps, read in
            bit-reversed lane order (the order its result is wanted in);
            `ising`: first-order Trotter steps of the transverse-field Ising
            chain (Rx on every qubit, exp(-i J dt Z Z) as CX Rz CX)
  observe   Pr(q = 0) of every qubit and Pauli strings of a given state
  sample    a sampling pool over all lanes, or over some of them in an order
            of the user's (the others are summed out), and samples from it
  adjoint   energies and gradients of the Ising chain for a batch of
            parameter vectors of a hardware-efficient ansatz
  batch     many small hardware-efficient circuits of uneven sizes
  dynamic   an OpenQASM program with mid-circuit measurement, reset and `if`

complex128 (the front-end's default precision) and complex64 both appear.
"""
import math

import numpy as np
import torch

from qgate_gb300 import adjoint, batch, qasm
from qgate_gb300 import gb300runtime as rt
from qgate_gb300.circuit import Lane, abs2, gate_type, null

CDT = {'c64': np.complex64, 'c128': np.complex128}
RDT = {'c64': np.float32, 'c128': np.float64}
CBYTES = {'c64': 8, 'c128': 16}
EXACT_QUBITS = 28  # above it the FP64 state takes plain torch too long


def listed():
    return [
        # the smallest calls: a few dozen gates on a handful of qubits
        dict(name='random_8_c128', kind='circuit', circuit='random', n=8, depth=4, dtype='c128',
             out='state'),
        # the QFT at the size the reference's users run it, read bit-reversed
        dict(name='qft_20_c64', kind='circuit', circuit='qft', n=20, depth=1, dtype='c64',
             out='prob'),
        # an ordinary circuit in the front-end's default precision, odd size
        dict(name='random_21_c128', kind='circuit', circuit='random', n=21, depth=20,
             dtype='c128', out='state'),
        # a large circuit in the default precision
        dict(name='random_26_c128', kind='circuit', circuit='random', n=26, depth=12,
             dtype='c128', out='prob'),
        # mostly diagonal gates in the default precision
        dict(name='qft_25_c128', kind='circuit', circuit='qft', n=25, depth=1, dtype='c128',
             out='prob'),
        # the headline: 30 qubits, depth 20, complex64, the whole probability vector
        dict(name='random_30_c64', kind='circuit', circuit='random', n=30, depth=20, dtype='c64',
             out='prob'),
        # what a user asks of a final state: every qubit, some Pauli strings
        dict(name='observe_28_c64', kind='observe', n=28, paulis=8, dtype='c64'),
        # samples of the whole register
        dict(name='sample_27_c64', kind='sample', n=27, lanes=27, shuffled=False,
             samples=1000000, dtype='c64'),
        # samples of some qubits in the user's own order
        dict(name='sample_15_of_25_c128', kind='sample', n=25, lanes=15, shuffled=True,
             samples=100000, dtype='c128'),
        # one step of a variational optimisation over a batch of parameter vectors
        dict(name='adjoint_20_c64', kind='adjoint', n=20, layers=6, batch=16, dtype='c64',
             every=3),
        # a batch of uneven small circuits
        dict(name='batch_512', kind='batch', count=512, lo=8, hi=20, dlo=4, dhi=12),
        # measurement, reset and feed-forward between gates
        dict(name='dynamic_18_c64', kind='dynamic', n=18, rounds=8, dtype='c64'),
    ]


def _between(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(['circuit'] * 5 + ['observe', 'sample', 'sample', 'adjoint', 'batch',
                                         'dynamic'])
    dtype = rng.choice(['c64', 'c128'])
    if kind == 'circuit':
        which = rng.choice(['random', 'random', 'qft', 'ising'])
        top = 28 if dtype == 'c64' else 25  # sizes are exponents: uniform in n is uniform in log size
        depth = 1 if which == 'qft' else _between(rng, 2, 20 if dtype == 'c64' else 12)
        return dict(kind=kind, circuit=which, n=rng.randint(8, top), depth=depth, dtype=dtype,
                    out=rng.choice(['state', 'prob']))
    if kind == 'observe':
        return dict(kind=kind, n=rng.randint(10, 28 if dtype == 'c64' else 27),
                    paulis=rng.randint(1, 16), dtype=dtype)
    if kind == 'sample':
        n = rng.randint(10, 27 if dtype == 'c64' else 26)
        part = rng.random() < 0.5
        return dict(kind=kind, n=n, lanes=rng.randint(4, n - 1) if part else n,
                    shuffled=part, samples=_between(rng, 100, 3000000), dtype=dtype)
    if kind == 'adjoint':
        return dict(kind=kind, n=rng.randint(8, 20 if dtype == 'c64' else 15),
                    layers=rng.randint(2, 8), batch=_between(rng, 1, 16), dtype=dtype,
                    every=rng.choice([0, 2, 3]))
    if kind == 'batch':
        lo = rng.randint(8, 14)
        hi = rng.randint(lo, 20)
        return dict(kind=kind, count=_between(rng, 16, 512), lo=lo, hi=hi, dlo=2,
                    dhi=rng.randint(3, 12))
    return dict(kind=kind, n=rng.randint(6, 22 if dtype == 'c64' else 20),
                rounds=rng.randint(2, 10), dtype=dtype)


# ---------------------------------------------------------------- inputs

def circuit_ops(case, seed):
    """[(gate name, arguments, target lane, control lanes)]"""
    n, r = case['n'], np.random.default_rng(seed)
    ops = []
    if case['circuit'] == 'random':
        for _ in range(case['depth']):
            ang = r.uniform(0, 2 * math.pi, (n, 3))
            ops += [('U', tuple(float(a) for a in ang[q]), q, ()) for q in range(n)]
            p = r.permutation(n)
            ops += [('X', (), int(p[2 * k + 1]), (int(p[2 * k]),)) for k in range(n // 2)]
    elif case['circuit'] == 'qft':
        # a product state (not a basis state, whose probabilities are all alike)
        for q in range(n):
            ops.append(('RY', (float(r.uniform(0.2, math.pi - 0.2)),), q, ()))
        for i in reversed(range(n)):
            ops.append(('H', (), i, ()))
            for j in reversed(range(i)):
                ops.append(('U1', (math.pi / (1 << (i - j)),), i, (j,)))
    else:
        dt = float(r.uniform(0.05, 0.15))
        field = r.uniform(0.5, 1.5, n)
        for _ in range(case['depth']):
            ops += [('RX', (float(2 * dt * field[q]),), q, ()) for q in range(n)]
            for q in range(n - 1):
                ops.append(('X', (), q + 1, (q,)))
                ops.append(('RZ', (2 * dt,), q + 1, ()))
                ops.append(('X', (), q + 1, (q,)))
    return ops


def lane_order(case):
    """External lane of each local lane in the values read back."""
    n = case['n']
    return [n - 1 - q for q in range(n)] if case['circuit'] == 'qft' else list(range(n))


def random_amplitudes(case, seed):
    """A normalised state of the Gaussian amplitudes that deep circuits give,
    on the GPU in the state's precision."""
    g = torch.Generator(device='cuda').manual_seed(seed)
    f = torch.float32 if case['dtype'] == 'c64' else torch.float64
    v = torch.randn((1 << case['n'], 2), generator=g, device='cuda', dtype=f)
    v /= torch.linalg.vector_norm(v)
    return torch.view_as_complex(v)


def host_values(case, dtype):
    """The page-locked array a program keeps for the values it reads back."""
    kind = {np.complex64: torch.complex64, np.complex128: torch.complex128,
            np.float32: torch.float32, np.float64: torch.float64}[dtype]
    return torch.empty(1 << case['n'], dtype=kind, pin_memory=True).numpy()


def new_states(case):
    qs = rt.create_qubit_states(RDT[case['dtype']])
    qs.processor.initialize_qubit_states(qs, case['n'])
    return qs


def given_state(case, seed):
    qs = new_states(case)
    qs.set_raw(random_amplitudes(case, seed).cpu().numpy())
    return qs


def pauli_strings(case, seed):
    """[(x mask, z mask)]: strings of one to four X, Y, Z factors."""
    r = np.random.default_rng(seed + 1)
    out = []
    for _ in range(case['paulis']):
        x = z = 0
        for q in r.permutation(case['n'])[:int(r.integers(1, 5))]:
            a = int(r.integers(1, 4))
            x |= (a & 1) << int(q)
            z |= (a >> 1) << int(q)
        out.append((x, z))
    return out


def pool_lanes(case, seed):
    """(lane, external lane or -1 where it is summed out) of the pool."""
    n = case['n']
    ext = [-1] * n
    lanes = list(range(n))
    if case['shuffled']:
        lanes = [int(q) for q in np.random.default_rng(seed + 2).permutation(n)[:case['lanes']]]
    for k, q in enumerate(lanes):
        ext[q] = k
    return list(enumerate(ext))


def dynamic_ops(case, seed):
    """Rounds of: rotations and entangling gates on the data qubits, a parity
    of two of them taken by an ancilla (the last qubit), its measurement, a
    correction if it reads 1, its reset."""
    n, r = case['n'], np.random.default_rng(seed)
    data, anc = n - 1, n - 1
    ops = []
    for c in range(case['rounds']):
        for q in range(data):
            ops.append(('g', 'RY', float(r.uniform(0, math.pi)), q, None))
            ops.append(('g', 'U1', float(r.uniform(0, math.pi)), q, None))
        for q in range(data - 1):
            ops.append(('g', 'X', None, q + 1, q))
        a, b = (int(q) for q in r.permutation(data)[:2])
        ops += [('g', 'X', None, anc, a), ('g', 'X', None, anc, b), ('m', anc, c),
                ('if', c, ('g', 'X', None, a, None)), ('r', anc)]
    return ops, r.random(case['rounds'])


def dynamic_text(case, ops):
    lines = ['OPENQASM 2.0;', 'include "qelib1.inc";', 'qreg q[%d];' % case['n']]
    lines += ['creg c%d[1];' % c for c in range(case['rounds'])]

    def gate(op):
        _, name, angle, t, ctrl = op
        if name == 'X':
            return 'x q[%d];' % t if ctrl is None else 'cx q[%d],q[%d];' % (ctrl, t)
        return '%s(%.17g) q[%d];' % (name.lower(), angle, t)
    for op in ops:
        if op[0] == 'g':
            lines.append(gate(op))
        elif op[0] == 'm':
            lines.append('measure q[%d] -> c%d[0];' % op[1:])
        elif op[0] == 'r':
            lines.append('reset q[%d];' % op[1])
        else:
            lines.append('if (c%d == 1) %s' % (op[1], gate(op[2])))
    return '\n'.join(lines)


def ansatz_params(case, seed):
    shape = (case['batch'], 2 * case['n'] * case['layers'])
    return np.random.default_rng(seed).uniform(-math.pi, math.pi, shape)


def prepare(case, seed):
    kind, s = case['kind'], {'case': case}
    if kind == 'circuit':
        s['qs'] = new_states(case)
        s['gates'] = [(gate_type(name, *args), t, list(c))
                      for name, args, t, c in circuit_ops(case, seed)]
        s['getter'] = rt.create_qubits_states_getter(RDT[case['dtype']])
        s['values'] = host_values(case, (CDT if case['out'] == 'state' else RDT)[case['dtype']])
    elif kind == 'observe':
        s['qs'] = given_state(case, seed)
        s['paulis'] = pauli_strings(case, seed)
    elif kind == 'sample':
        s['qs'] = given_state(case, seed)
        s['lanes'] = pool_lanes(case, seed)
        s['getter'] = rt.create_qubits_states_getter(RDT[case['dtype']])
        s['u'] = np.random.default_rng(seed + 3).random(case['samples'])
    elif kind == 'adjoint':
        s['circuit'] = adjoint.hardware_efficient_ansatz(case['n'], case['layers'])
        s['observable'] = adjoint.PauliSum.ising_chain(case['n'])
        s['params'] = ansatz_params(case, seed)
    elif kind == 'batch':
        s['packed'] = batch.pack(hea_circuits(case, seed))
    else:
        ops, u = dynamic_ops(case, seed)
        s['program'] = qasm.parse(dynamic_text(case, ops))
        s['u'] = [float(x) for x in u]
        s['qs'] = new_states(case)
        s['getter'] = rt.create_qubits_states_getter(RDT[case['dtype']])
        s['values'] = host_values(case, CDT[case['dtype']])
    return s


def hea_circuits(case, seed):
    return batch.hea_batch(case['count'], seed, case['lo'], case['hi'], case['dlo'], case['dhi'])


def read(s, mathop, order):
    """The whole state or probability vector, in `order`."""
    qs, values = s['qs'], s['values']
    s['getter'].get_states(values, 0, mathop, [(qs, [Lane(q, e) for q, e in enumerate(order)])],
                           [], len(values), 0, 1)
    return values


def run(s):
    case = s['case']
    kind = case['kind']
    if kind == 'circuit':
        qs = s['qs']
        p = qs.processor
        p.reset_qubit_states(qs)
        for g, t, c in s['gates']:
            if c:
                p.apply_controlled_gate(g, False, qs, c, t)
            else:
                p.apply_gate(g, False, qs, t)
        return read(s, null if case['out'] == 'state' else abs2, lane_order(case))
    if kind == 'observe':
        qs = s['qs']
        p = qs.processor
        return {'prob': np.array([p.calc_probability(qs, q) for q in range(case['n'])]),
                'pauli': np.array([p.calc_pauli_expectation(qs, x, z) for x, z in s['paulis']])}
    if kind == 'sample':
        k = case['lanes']
        pool = s['getter'].create_sampling_pool(list(range(k)), k, case['n'] - k,
                                                [(s['qs'], [Lane(q, e) for q, e in s['lanes']])],
                                                [])
        out = pool.sample(len(s['u']), s['u']).intarray
        pool.delete()
        return np.asarray(out)
    if kind == 'adjoint':
        e, g = adjoint.expectation_and_gradient(s['circuit'], s['params'], s['observable'],
                                                RDT[case['dtype']], case['every'])
        return {'energy': e, 'gradient': g}
    if kind == 'batch':
        return batch.sum_z(packed=s['packed'])
    qs = s['qs']
    qs.processor.reset_qubit_states(qs)
    bits = s['program'].run(qs, s['u'], graph=True)
    return {'bits': bits, 'state': read(s, null, list(range(case['n'])))}


# ---------------------------------------------------------------- work

def work(case):
    """Each amplitude that comes back or goes in is counted once; a 2x2 gate
    that is not a permutation or a phase does 14 operations per amplitude
    (real work on all of them), a phase 6 on those it touches."""
    kind = case['kind']
    if kind in ('circuit', 'dynamic'):
        n = case['n']
        size, cb = float(1 << n), CBYTES[case['dtype']]
        if kind == 'dynamic':
            return {'bytes': size * cb, 'flops': case['rounds'] * (n - 1) * 14 * size}
        flops = 0.
        for name, _, _, c in circuit_ops(case, 0):
            flops += {'X': 0., 'RZ': 6., 'U1': 6.}.get(name, 14.) * size / (1 << len(c))
        return {'bytes': size * (cb if case['out'] == 'state' else cb // 2), 'flops': flops}
    if kind == 'observe':
        size = float(1 << case['n'])
        return {'bytes': size * CBYTES[case['dtype']],
                'flops': size * 4 * (case['n'] + 2 * case['paulis'])}
    if kind == 'sample':
        size = float(1 << case['n'])
        return {'bytes': size * CBYTES[case['dtype']] + 16. * case['samples'], 'flops': 4 * size}
    if kind == 'adjoint':
        n = case['n']
        size = float(1 << n) * case['batch']
        rotations = 2 * n * case['layers']
        return {'bytes': 16. * case['batch'] * rotations,
                'flops': size * (rotations * (14 + 2 * 14 + 8) + (2 * n - 1) * 8)}
    size = 0.
    for n, ops in hea_circuits(case, 0):
        size += float(1 << n) * sum(14. if name == 'RY' else 6. for name, _, _, c in ops if not c)
    return {'bytes': 8. * case['count'], 'flops': size}


# ---------------------------------------------------------------- exact values

def matrix(name, args):
    """The gate's 2x2 matrix in 64 bits."""
    e = np.exp
    if name == 'X':
        return [[0, 1], [1, 0]]
    if name == 'H':
        return [[math.sqrt(.5), math.sqrt(.5)], [math.sqrt(.5), -math.sqrt(.5)]]
    if name == 'U1':
        return [[1, 0], [0, e(1j * args[0])]]
    if name == 'RZ':
        return [[e(-.5j * args[0]), 0], [0, e(.5j * args[0])]]
    c, s = math.cos(args[0] / 2), math.sin(args[0] / 2)
    if name == 'RY':
        return [[c, -s], [s, c]]
    if name == 'RX':
        return [[c, -1j * s], [-1j * s, c]]
    _, phi, lam = args
    return [[e(-.5j * (lam + phi)) * c, -e(.5j * (lam - phi)) * s],
            [e(.5j * (phi - lam)) * s, e(.5j * (lam + phi)) * c]]


def zero_state(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device='cuda')
    psi[0] = 1
    return psi


def halves(psi, n, target, controls=()):
    """Views of the amplitudes with the target lane 0 and 1 (controls 1)."""
    v = psi.view([2] * n)
    at = [slice(None)] * n
    for c in controls:
        at[n - 1 - c] = 1
    at[n - 1 - target] = 0
    lo = v[tuple(at)]
    at[n - 1 - target] = 1
    return lo, v[tuple(at)]


def apply(psi, n, m, target, controls=()):
    lo, hi = halves(psi, n, target, controls)
    if m[0][1] == 0 and m[1][0] == 0:
        lo *= m[0][0]
        hi *= m[1][1]
    else:
        a, b = lo.clone(), hi.clone()
        lo.copy_(a * m[0][0] + b * m[0][1])
        hi.copy_(a * m[1][0] + b * m[1][1])


def adjoint_matrix(m):
    return np.conj(np.array(m)).T.tolist()


def exact(case, seed):
    kind = case['kind']
    if kind == 'circuit':
        n = case['n']
        if n > EXACT_QUBITS:
            return None
        psi = zero_state(n)
        for name, args, t, c in circuit_ops(case, seed):
            apply(psi, n, matrix(name, args), t, c)
        order = lane_order(case)
        v = psi.view([2] * n)
        # external lane e is axis n - 1 - e of the result
        local = {e: q for q, e in enumerate(order)}
        v = v.permute([n - 1 - local[n - 1 - a] for a in range(n)]).reshape(-1)
        if case['out'] == 'prob':
            v = v.real ** 2 + v.imag ** 2
        return v.cpu().numpy()
    if kind == 'observe':
        n = case['n']
        psi = random_amplitudes(case, seed).to(torch.complex128)
        p = psi.real ** 2 + psi.imag ** 2
        prob = [float(halves(p, n, q)[0].sum()) for q in range(n)]
        index = torch.arange(1 << n, device='cuda')
        pauli = []
        for x, z in pauli_strings(case, seed):
            b = index & z
            for k in (32, 16, 8, 4, 2, 1):
                b = b ^ (b >> k)
            sign = (1 - 2 * (b & 1)).to(torch.float64)
            # P|b> = i^ny (-1)^(b.z) |b ^ x>
            overlap = (psi[index ^ x].conj() * psi * sign).sum() * 1j ** bin(x & z).count('1')
            pauli.append(float(overlap.real))
        return {'prob': np.array(prob), 'pauli': np.array(pauli)}
    if kind == 'adjoint':
        return exact_adjoint(case, seed)
    if kind == 'batch':
        return np.array([exact_sum_z(n, ops) for n, ops in hea_circuits(case, seed)])
    if kind == 'dynamic':
        return exact_dynamic(case, seed)
    return None  # samples are whole numbers


def exact_sum_z(n, ops):
    psi = zero_state(n)
    k = 0
    while k < len(ops):
        name, args, t, c = ops[k]
        if name == 'RY' and k + 1 < len(ops) and ops[k + 1][0] == 'RZ' and ops[k + 1][2] == t:
            m = np.array(matrix('RZ', ops[k + 1][1])) @ np.array(matrix('RY', args))
            apply(psi, n, m.tolist(), t)
            k += 2
            continue
        if name == 'X':
            lo, hi = halves(psi, n, t, c)
            a = lo.clone()
            lo.copy_(hi)
            hi.copy_(a)
        else:
            apply(psi, n, matrix(name, args), t, c)
        k += 1
    p = psi.real ** 2 + psi.imag ** 2
    index = torch.arange(1 << n, device='cuda')
    ones = sum((index >> q) & 1 for q in range(n))
    return float((p * (n - 2 * ones)).sum())


def exact_adjoint(case, seed):
    n, layers = case['n'], case['layers']
    params = ansatz_params(case, seed)
    index = torch.arange(1 << n, device='cuda')
    diag = torch.zeros(1 << n, dtype=torch.float64, device='cuda')
    for q in range(n - 1):
        diag -= 1 - 2 * (((index >> q) ^ (index >> (q + 1))) & 1).to(torch.float64)
    ops = []  # (name, parameter index, target, controls)
    for layer in range(layers):
        first = 2 * n * layer
        ops += [('RY', first + q, q, ()) for q in range(n)]
        ops += [('RZ', first + n + q, q, ()) for q in range(n)]
        ops += [('X', None, (q + 1) % n, (q,)) for q in range(n)]
    energy = np.zeros(case['batch'])
    gradient = torch.zeros(params.shape, dtype=torch.float64, device='cuda')
    for b in range(case['batch']):
        psi = zero_state(n)
        for name, k, t, c in ops:
            apply(psi, n, matrix(name, () if k is None else (params[b, k],)), t, c)
        lam = psi * diag
        for q in range(n):
            lo, hi = halves(psi, n, q)
            out_lo, out_hi = halves(lam, n, q)
            out_lo -= 0.7 * hi
            out_hi -= 0.7 * lo
        energy[b] = float(torch.vdot(psi, lam).real)
        for name, k, t, c in reversed(ops):
            if k is not None:
                p0, p1 = halves(psi, n, t)
                l0, l1 = halves(lam, n, t)
                if name == 'RY':  # Im <lam|Y|psi>, Y|psi> = (-i p1, i p0)
                    g = (l1.conj() * p0 - l0.conj() * p1).real.sum()
                else:
                    g = (l0.conj() * p0 - l1.conj() * p1).imag.sum()
                gradient[b, k] = g
            m = adjoint_matrix(matrix(name, () if k is None else (params[b, k],)))
            apply(psi, n, m, t, c)
            apply(lam, n, m, t, c)
    return {'energy': energy, 'gradient': gradient.cpu().numpy()}


def exact_dynamic(case, seed):
    n = case['n']
    ops, u = dynamic_ops(case, seed)
    psi, bits, taken = zero_state(n), 0, 0

    def gate(op):
        _, name, angle, t, ctrl = op
        apply(psi, n, matrix(name, () if angle is None else (angle,)), t,
              () if ctrl is None else (ctrl,))
    value = {}
    for op in ops:
        if op[0] == 'g':
            gate(op)
        elif op[0] == 'm':
            lo, hi = halves(psi, n, op[1])
            p0 = float((lo.real ** 2 + lo.imag ** 2).sum())
            v = 0 if u[taken] < p0 else 1
            taken += 1
            (hi if v == 0 else lo).zero_()
            keep = lo if v == 0 else hi
            keep *= 1 / math.sqrt(p0 if v == 0 else 1 - p0)
            bits |= v << op[2]
            value[op[1]] = value[('c', op[2])] = v
        elif op[0] == 'r':
            if value[op[1]]:
                lo, hi = halves(psi, n, op[1])
                lo.copy_(hi)
                hi.zero_()
        elif value[('c', op[1])]:
            gate(op[2])
    return {'bits': bits, 'state': psi.cpu().numpy()}
