"""The work this engine is timed on: its public entry points over the sizes they are used at.

Every case is one call (or one sequence of calls) that a user's program makes with its inputs in
hand: ``execute`` on a small circuit, a recorded circuit's device work, the single-operation C ABI,
the read-outs, batched and template sweeps, and the noise surrogate's training and inference.  The
circuits are the seeded brick layers (U3 on every qubit, then CX on neighbouring pairs) and the QFT
that the tests and the benchmark use, with the full noise model.  ``exact`` restates each case in
64 bits with plain torch and numpy.
"""
import ctypes
import itertools
import math

import numpy as np
import torch

import __graft_entry__

PI = math.pi
_AXES = ('rx', 'ry', 'rz')
_NOISE = {'depolarisation': 1e-3, 'decoherence': 0.995, 'decay': 0.998, 'rotation_sigma': 1e-3}


def _pkg():
    return __graft_entry__.load_package()


def _device():
    return torch.device('cuda' if torch.cuda.is_available() else 'cpu')


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the everyday call: a small noisy circuit through the drop-in backend, with the whole result
        # dictionary (coefficients, density matrix, 2**n probabilities)
        {'name': 'execute_n8', 'kind': 'execute', 'n': 8, 'layers': 20, 'precision': 'double'},
        # a recorded FP32 circuit small enough that launches and single-tile latencies count
        {'name': 'circuit_n10_f32', 'kind': 'circuit', 'n': 10, 'layers': 20, 'qft': False, 'precision': 'single'},
        # QFT and random layers on 14 qubits, noise after every gate: many short-range and long-range CX
        {'name': 'qft_n14_f32', 'kind': 'circuit', 'n': 14, 'layers': 2, 'qft': True, 'precision': 'single'},
        # the headline workload's layers at its size: a 17 GB FP32 state
        {'name': 'circuit_n16_f32', 'kind': 'circuit', 'n': 16, 'layers': 6, 'qft': False, 'precision': 'single'},
        # the FP64 parity form at an odd size
        {'name': 'circuit_n13_f64', 'kind': 'circuit', 'n': 13, 'layers': 6, 'qft': False, 'precision': 'double'},
        # the batched noise sweep: uneven qubit counts and depths, many instances of each structure
        {'name': 'sweep_n6_12', 'kind': 'sweep', 'structures': 24, 'per': 24, 'nlo': 6, 'nhi': 12, 'dlo': 10,
         'dhi': 50, 'precision': 'single'},
        # one circuit at many noise points: the data generation of the surrogate
        {'name': 'template_n10', 'kind': 'template', 'n': 10, 'layers': 30, 'points': 1024, 'precision': 'single'},
        # one training step of the five-member surrogate
        {'name': 'train_b1024', 'kind': 'train', 'members': 5, 'batch': 1024, 'nout': 1024},
        # inference of the ensemble with its spread, a ragged number of points
        {'name': 'predict_s10233', 'kind': 'predict', 'members': 5, 'batch': 1024, 'nout': 1024, 'points': 10233},
        # the plain form: one sweep of the state per gate, channel and read-out through the C ABI
        {'name': 'gates_n13_f64', 'kind': 'gates', 'n': 13, 'layers': 2, 'precision': 'double'},
        {'name': 'gates_n14_f32', 'kind': 'gates', 'n': 14, 'layers': 2, 'precision': 'single'},
        # everything that is read from a final state: probabilities (Z, a direction, a subset), the
        # density matrix, an overlap, the chopped coefficients
        {'name': 'readout_n12_f64', 'kind': 'readout', 'n': 12, 'precision': 'double'},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['execute', 'circuit', 'circuit', 'sweep', 'template', 'train', 'predict', 'gates', 'readout'])
    if kind == 'execute':
        n = rng.randint(3, 10)
        return {'kind': kind, 'n': n, 'layers': _log_int(rng, 3, 40),
                'precision': rng.choice(['double', 'double', 'single'])}
    if kind == 'circuit':
        precision = rng.choice(['single', 'single', 'double'])
        n = rng.randint(7, 16 if precision == 'single' else 14)
        qft = n <= 14 - 2 * (precision == 'double') and rng.random() < 0.3
        most = max(1, min(40, int(6 * 4 ** (16 - n) / (1 if precision == 'single' else 20))))
        return {'kind': kind, 'n': n, 'layers': _log_int(rng, 1, most), 'qft': qft, 'precision': precision}
    if kind == 'sweep':
        precision = rng.choice(['single', 'single', 'double'])
        nlo = rng.randint(4, 9)
        nhi = rng.randint(nlo, 11 if precision == 'single' else 9)
        dlo = rng.randint(3, 15)
        return {'kind': kind, 'structures': rng.randint(4, 20), 'per': _log_int(rng, 1, 24), 'nlo': nlo, 'nhi': nhi,
                'dlo': dlo, 'dhi': rng.randint(dlo, 40), 'precision': precision}
    if kind == 'template':
        precision = rng.choice(['single', 'single', 'double'])
        n = rng.randint(5, 11 if precision == 'single' else 8)
        layers = _log_int(rng, 3, 40)
        most = int(min(8192, max(16, 1024 * 30 * 4 ** (10 - n) / layers)))
        return {'kind': kind, 'n': n, 'layers': layers, 'points': _log_int(rng, 8, most), 'precision': precision}
    if kind == 'train':
        return {'kind': kind, 'members': rng.randint(1, 6), 'batch': 128 * rng.randint(1, 16),
                'nout': 256 * rng.randint(1, 8)}
    if kind == 'predict':
        # whole minibatches, the last one ragged within its last 128 rows
        batch = 128 * rng.randint(1, 16)
        return {'kind': kind, 'members': rng.randint(1, 6), 'batch': batch, 'nout': 256 * rng.randint(1, 8),
                'points': batch * _log_int(rng, 1, max(1, 16000 // batch)) - rng.randint(0, 127)}
    precision = rng.choice(['single', 'double'])
    if kind == 'gates':
        n = rng.randint(2, 14)
        return {'kind': kind, 'n': n, 'layers': rng.randint(1, 6 if n < 13 else 2), 'precision': precision}
    return {'kind': kind, 'n': rng.randint(2, 12), 'precision': precision}


# ---------------------------------------------------------------------------
# seeded inputs, shared with exact()
# ---------------------------------------------------------------------------

def _rng(seed, *more):
    return np.random.default_rng([seed & 0x7fffffff, *more])


def _brick(n, layers, seed):
    ang = _rng(seed, 1).uniform(0.0, 2 * PI, size=(layers, n, 3))
    gates = []
    for L in range(layers):
        gates += [('u3', q, *(float(a) for a in ang[L, q])) for q in range(n)]
        gates += [('cx', a, a + 1) for a in range(L % 2, n - 1, 2)]
    return gates


def _qft(n):
    gates = []
    for wire in range(n - 1):
        gates.append(('u3', wire, PI / 2, 0.0, PI))
        for rot in range(wire + 1):
            lam = 2 * PI / 2 ** (wire + 2 - rot)
            gates += [('u1', wire + 1, lam / 2), ('cx', wire + 1, rot), ('u1', rot, -lam / 2), ('cx', wire + 1, rot),
                      ('u1', rot, lam / 2)]
    return gates + [('u3', n - 1, PI / 2, 0.0, PI)]


def _circuit(n, gates, barriers):
    qc = _pkg().QuantumCircuit(n, n)
    for g in gates:
        if g[0] == 'u3':
            qc.u3(g[2], g[3], g[4], g[1])
        elif g[0] == 'u1':
            qc.u1(g[2], g[1])
        else:
            qc.cx(g[1], g[2])
        if barriers:
            qc.barrier()
    qc.measure(list(range(n)), list(range(n)), basis='Ensemble', add_param='Z')
    return qc


def _gates_of(case, seed):
    pre = _qft(case['n']) if case.get('qft') else []
    return pre + _brick(case['n'], case['layers'], seed)


def _noise_points(count, seed):
    """Noise points in the surrogate's ranges: losses log-uniform, thermal factor and angle spread uniform."""
    r = _rng(seed, 2)
    raw = np.exp(r.uniform(math.log(1e-4), math.log(1e-2), size=(count, 6)))
    raw[:, 3] = r.uniform(0.8, 1.0, count)
    raw[:, 4] = r.uniform(0.0, 0.05, count)
    return raw


def _sweep_specs(case, seed):
    r = _rng(seed, 3)
    shape = _rng(0, case['structures'], case['nlo'], case['nhi'], case['dlo'], case['dhi'])
    specs = []
    for _ in range(case['structures']):
        n, depth = int(shape.integers(case['nlo'], case['nhi'] + 1)), int(shape.integers(case['dlo'], case['dhi'] + 1))
        for _ in range(case['per']):
            p, f, g = (float(x) for x in np.exp(r.uniform(math.log(1e-4), math.log(1e-2), 3)))
            specs.append({'n': n, 'depth': depth, 'seed': int(r.integers(1 << 40)), 'depolarisation': p,
                          'decoherence': 1.0 - f, 'decay': 1.0 - g})
    return specs


_WIDTHS = (64, 256, 256, 256)


def _mlp_params(members, nout, seed):
    """Flat [members, P] FP32 parameters W1 b1 ... W4 b4: normal weights of unit gain, small biases."""
    g = torch.Generator(device=_device()).manual_seed(seed & 0x7fffffff)
    widths = _WIDTHS + (nout,)
    parts = []
    for li in range(4):
        fan = 6 if li == 0 else widths[li]
        w = torch.randn(members, widths[li + 1], widths[li], generator=g, device=_device())
        w *= math.sqrt((2.0 if li < 3 else 1.0) / fan)
        if li == 0:
            w[:, :, 6:] = 0
        parts += [w.reshape(members, -1), 0.05 * torch.randn(members, widths[li + 1], generator=g, device=_device())]
    return torch.cat(parts, dim=1).contiguous()


def _mlp_data(samples, nout, seed):
    """Features in [-1, 1] and smooth target distributions of them."""
    g = torch.Generator(device=_device()).manual_seed((seed & 0x7fffffff) + 1)
    x = 2 * torch.rand(samples, 6, generator=g, device=_device()) - 1
    a = torch.randn(nout, generator=g, device=_device())
    b = 0.5 * torch.randn(6, nout, generator=g, device=_device())
    return x.contiguous(), torch.softmax(a + x @ b, dim=1).contiguous()


_STEPS = 8      # minibatches a training state holds; run() takes the next one


def _mlp_index(case, samples, seed):
    r = _rng(seed, 4)
    idx = np.stack([np.stack([r.permutation(samples)[:case['batch']] for _ in range(case['members'])])
                    for _ in range(_STEPS)])
    return torch.from_numpy(idx.astype(np.int32)).to(_device())


def _mixed_state(n, seed, dtype):
    """A physical state: a mixture of four random product states, as Pauli coefficients."""
    r = _rng(seed, 5)
    w = r.dirichlet(np.ones(4))
    out = None
    for k in range(4):
        v = r.normal(size=(n, 3))
        v *= (r.uniform(0.6, 1.0, n) / np.linalg.norm(v, axis=1))[:, None]
        a = torch.tensor([w[k] * 2.0 ** -n], dtype=torch.float64, device=_device())
        for q in range(n):
            f = torch.tensor([1.0, *v[q]], dtype=torch.float64, device=_device())
            a = (a[:, None] * f[None, :]).reshape(-1)
        out = a if out is None else out.add_(a)
    return out.to(dtype)


def _direction(seed):
    v = _rng(seed, 6).normal(size=3)
    return [float(x) for x in v / np.linalg.norm(v)]


def _dtype(case):
    return torch.float32 if case['precision'] == 'single' else torch.float64


def _fp(case, x):
    """Results of an FP32 state at the state's own precision."""
    if case['precision'] == 'double':
        return x
    return x.astype(np.float32) if isinstance(x, np.ndarray) else x.to(torch.float32)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    return _PREPARE[case['kind']](case, seed)


def run(state):
    return _RUN[state['case']['kind']](state)


def _options(case):
    opts = _pkg().noise_options(**_NOISE)
    opts['precision'] = case['precision']
    return opts


def _prepare_execute(case, seed):
    pkg = _pkg()
    qc = _circuit(case['n'], _gates_of(case, seed), False)
    return {'case': case, 'qc': qc, 'backend': pkg.BasicAer.get_backend('dm_simulator'), 'opts': _options(case)}


def _run_execute(s):
    opts = dict(s['opts'], rotation_error=dict(s['opts']['rotation_error']))
    data = _pkg().execute(s['qc'], s['backend'], **opts).result()['results'][0]['data']
    rho = data['densitymatrix']
    return {'coeffmatrix': _fp(s['case'], data['coeffmatrix']),
            'densitymatrix': rho if s['case']['precision'] == 'double' else rho.astype(np.complex64),
            'probability': _fp(s['case'], np.array(list(data['ensemble_probability'].values())))}


def _prepare_circuit(case, seed):
    pkg = _pkg()
    b = pkg.DmSimulatorGPU()
    b._set_options(backend_options=dict(_options(case), compute_densitymatrix=False, coefficients_to_host=False))
    b.record_experiment(_circuit(case['n'], _gates_of(case, seed), True).to_experiment())
    return {'case': case, 'dev': b.recorded_state}


def _run_circuit(s):
    s['dev'].replay()
    return {'state': s['dev'].state, 'probability': _fp(s['case'], s['dev'].last_readout)}


def _prepare_sweep(case, seed):
    _pkg()
    from qiskit_aakash_gb300 import batch
    p = case['precision']
    # what the autotuner picks on this device: tensor cores from 9 qubits up in FP32
    kmax = {n: batch.TC for n in range(9, 13)} if p == 'single' else {}
    prog = batch.BatchProgram(batch.compile_sweep(_sweep_specs(case, seed), [p], kmax={p: kmax})[p])
    prog.capture()
    return {'case': case, 'prog': prog}


def _run_sweep(s):
    s['prog'].run()
    return {'probability': _fp(s['case'], s['prog'].probs)}


def _prepare_template(case, seed):
    _pkg()
    from qiskit_aakash_gb300 import surrogate, template
    raw = _noise_points(case['points'], seed)
    exp = _circuit(case['n'], _brick(case['n'], case['layers'], seed), False).to_experiment()
    prog = template.TemplateProgram(exp, surrogate.options_of(raw[0]), case['precision'])
    return {'case': case, 'runner': template.TemplateRunner(prog), 'params': surrogate.param_vectors(raw)}


def _run_template(s):
    return {'probability': _fp(s['case'], s['runner'].run(s['params']))}


def _ensemble(case, seed):
    _pkg()
    from qiskit_aakash_gb300 import surrogate
    ens = surrogate.MLPEnsemble(members=case['members'], batch=case['batch'], nout=case['nout'])
    ens.set_params(_mlp_params(case['members'], case['nout'], seed))
    return ens


def _prepare_train(case, seed):
    samples = 4 * case['batch']
    x, y = _mlp_data(samples, case['nout'], seed)
    return {'case': case, 'ens': _ensemble(case, seed), 'x': x, 'y': y, 'index': _mlp_index(case, samples, seed),
            'next': itertools.cycle(range(_STEPS))}


def _run_train(s):
    s['ens'].train_step(s['x'], s['y'], s['index'][next(s['next'])], 1e-3)
    return {'loss_rows': s['ens'].loss_rows, 'grads': s['ens'].grads, 'params': s['ens'].params}


def _prepare_predict(case, seed):
    x, y = _mlp_data(case['points'], case['nout'], seed)
    return {'case': case, 'ens': _ensemble(case, seed), 'x': x, 'y': y}


def _run_predict(s):
    members = s['ens'].predict(s['x'])
    mean, spread, tv = s['ens'].ensemble(members, s['y'])
    return {'members': members, 'mean': mean, 'spread': spread, 'tv': tv}


_F, _P, _G = 0.995, 0.97, 0.998       # decoherence, thermal and decay factors of the plain form's channels
_TSP = (0.999, 0.01)                  # its CX error
_ERR = 0.999                          # polarisation of its read-outs


def _rot(theta, phi, lam, c):
    """4x4 map of U3 = Rz(lam), Ry(theta), Rz(phi), each averaged over its angle error (<cos> = c)."""
    def rz(a):
        m = np.eye(4)
        m[1, 1] = m[2, 2] = c * math.cos(a)
        m[1, 2], m[2, 1] = -c * math.sin(a), c * math.sin(a)
        return m

    def ry(a):
        m = np.eye(4)
        m[1, 1] = m[3, 3] = c * math.cos(a)
        m[3, 1], m[1, 3] = -c * math.sin(a), c * math.sin(a)
        return m
    return rz(phi) @ ry(theta) @ rz(lam)


def _plain_maps(case, seed):
    return [(g[1], _rot(g[2], g[3], g[4], 0.9999)) if g[0] == 'u3' else g for g in _brick(case['n'], case['layers'], seed)]


def _lib():
    _pkg()
    from qiskit_aakash_gb300 import _native
    return _native


def _prepare_gates(case, seed):
    N = _lib()
    n = case['n']
    ops = []
    for g in _plain_maps(case, seed):
        if g[0] == 'cx':
            ops.append(('dm_apply_cx', g[1], g[2], (ctypes.c_double * 2)(*_TSP)))
        else:
            ops.append(('dm_apply_map1', g[0], (ctypes.c_double * 16)(*g[1].reshape(16))))
    return {'case': case, 'ops': ops, 'init': (ctypes.c_double * (4 * n))(*([1.0, 0.0, 0.0, 1.0] * n)),
            'state': torch.empty(4 ** n, dtype=_dtype(case), device=_device()),
            'probs': torch.empty(2 ** n, dtype=torch.float64, device=_device()), 'mode': (ctypes.c_int * n)(*([3] * n)),
            'dtype': N.DM_F32 if case['precision'] == 'single' else N.DM_F64}


def _run_gates(s):
    N = _lib()
    n, dt, vp = s['case']['n'], s['dtype'], ctypes.c_void_p
    st, stream = vp(s['state'].data_ptr()), vp(torch.cuda.current_stream().cuda_stream)

    def noise():      # one clock cycle's memory noise on every qubit
        N.call('dm_apply_memory_noise', st, n, dt, _F, _P, _G, stream)

    N.call('dm_init_product', st, n, dt, s['init'], 0.5 ** n, stream)
    last = None
    for op in s['ops']:
        if last is not None and op[0] != last:
            noise()
        last = op[0]
        N.call(op[0], st, n, dt, *op[1:], stream)
    noise()
    N.call('dm_axis_probs', st, n, dt, s['mode'], _ERR, vp(s['probs'].data_ptr()), stream)
    return {'state': s['state'], 'probability': _fp(s['case'], s['probs'])}


def _subset(n):
    """The measured qubits of the partial read-out: every third one."""
    return list(range(0, n, 3))


def _prepare_readout(case, seed):
    N = _lib()
    n, dev = case['n'], _device()
    L = N.lib()
    part = _subset(n)
    return {'case': case, 'dtype': N.DM_F32 if case['precision'] == 'single' else N.DM_F64,
            'state': _mixed_state(n, seed, _dtype(case)), 'other': _mixed_state(n, seed + 1, _dtype(case)),
            'z': torch.empty(2 ** n, dtype=torch.float64, device=dev), 'zmode': (ctypes.c_int * n)(*([3] * n)),
            'x': torch.empty(2 ** len(part), dtype=torch.float64, device=dev),
            'xmode': (ctypes.c_int * n)(*[1 if q in part else 0 for q in range(n)]),
            'nvec': (ctypes.c_double * 3)(*_direction(seed)),
            'np': torch.empty(2 ** n, dtype=torch.float64, device=dev),
            'nscratch': torch.empty(max(8, L.dm_nbasis_probs_scratch_bytes(n)), dtype=torch.uint8, device=dev),
            'rho': torch.empty((2 ** n, 2 ** n), dtype=torch.complex128, device=dev),
            'rscratch': torch.empty(L.dm_pauli_to_matrix_scratch_bytes(n), dtype=torch.uint8, device=dev),
            'ov': torch.empty(1, dtype=torch.float64, device=dev),
            'oscratch': torch.empty(L.dm_overlap_scratch_bytes(n), dtype=torch.uint8, device=dev),
            'chop': torch.empty(4 ** n, dtype=torch.float64, device=dev)}


def _run_readout(s):
    N = _lib()
    n, dt, vp = s['case']['n'], s['dtype'], ctypes.c_void_p
    st, stream = vp(s['state'].data_ptr()), vp(torch.cuda.current_stream().cuda_stream)

    def p(k):
        return vp(s[k].data_ptr())

    N.call('dm_axis_probs', st, n, dt, s['zmode'], _ERR, p('z'), stream)
    N.call('dm_axis_probs', st, n, dt, s['xmode'], _ERR, p('x'), stream)
    N.call('dm_nbasis_probs', st, n, dt, s['nvec'], _ERR, p('np'), p('nscratch'), stream)
    N.call('dm_overlap', st, p('other'), n, dt, p('ov'), p('oscratch'), stream)
    N.call('dm_pauli_to_matrix', st, n, dt, p('rho'), p('rscratch'), stream)
    N.call('dm_chop_copy', st, n, dt, 1e-15, p('chop'), stream)
    return {'z': s['z'], 'x': s['x'], 'n': s['np'], 'overlap': s['ov'], 'rho': s['rho'], 'coefficients': s['chop']}


_PREPARE = {'execute': _prepare_execute, 'circuit': _prepare_circuit, 'sweep': _prepare_sweep,
            'template': _prepare_template, 'train': _prepare_train, 'predict': _prepare_predict,
            'gates': _prepare_gates, 'readout': _prepare_readout}
_RUN = {'execute': _run_execute, 'circuit': _run_circuit, 'sweep': _run_sweep, 'template': _run_template,
        'train': _run_train, 'predict': _run_predict, 'gates': _run_gates, 'readout': _run_readout}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    k = case['kind']
    if k in ('execute', 'circuit'):
        # the final state and its probabilities written once (FP64 results of execute(): the
        # coefficients and the matrix); per gate 10 multiply-adds per four coefficients of a U3
        n, size = case['n'], 4 if case['precision'] == 'single' else 8
        gates = _gates_of(case, 0)
        flops = 4.0 ** n * 5 * sum(g[0] != 'cx' for g in gates)
        out = 24 if k == 'execute' else size
        return {'bytes': 4.0 ** n * out + 2.0 ** n * 8, 'flops': flops}
    if k == 'sweep':
        n, d = (case['nlo'] + case['nhi']) / 2, (case['dlo'] + case['dhi']) / 2
        ns = range(case['nlo'], case['nhi'] + 1)
        mean4 = sum(4.0 ** n * n for n in ns) / len(ns)
        count = case['structures'] * case['per']
        return {'bytes': count * (2.0 ** n * 8 + d * n * 128), 'flops': count * 5 * d * mean4}
    if k == 'template':
        n, pts = case['n'], case['points']
        return {'bytes': pts * (2.0 ** n * 8 + 128), 'flops': pts * 5.0 * case['layers'] * n * 4.0 ** n}
    if k in ('train', 'predict'):
        m, nout = case['members'], case['nout']
        wide = 64 * 256 + 2 * 256 * 256 + 256 * nout
        p = wide + 768 + nout
        if k == 'train':
            b = case['batch']
            # parameters, gradients and Adam moments; features and targets of the minibatch
            return {'bytes': m * (p * 4 * 7 + b * (nout + 6) * 4), 'flops': 6.0 * m * b * wide}
        pts = case['points']
        return {'bytes': pts * (24 + nout * 4 * (m + 2)) + m * p * 4, 'flops': 2.0 * m * pts * wide}
    n, size = case['n'], 4 if case['precision'] == 'single' else 8
    if k == 'gates':
        # every call updates the state in place: one read and one write of it
        cxs = sum(g[0] == 'cx' for g in _brick(n, case['layers'], 0))
        u3s = n * case['layers']
        noises = 2 * case['layers']
        return {'bytes': 4.0 ** n * size * (2 * (u3s + cxs + noises) + 1),
                'flops': 4.0 ** n * (5 * u3s + 3 * cxs + noises * n)}
    # read-outs: the state (and the second one) read once, the matrix and the coefficients written
    return {'bytes': 4.0 ** n * (2 * size + 16 + 8) + 2.0 ** n * 16, 'flops': 4.0 ** n * (3 * n + 6)}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def exact(case, seed):
    with torch.no_grad():
        return _EXACT[case['kind']](case, seed)


class _Exact:
    """Pauli coefficients of ``count`` instances, [count, 4**n] in FP64.  Single-qubit maps are
    kept per qubit, shared ([4, 4]) or per instance ([count, 4, 4]), until something needs the qubit."""

    def __init__(self, n, count=1):
        self.n, self.count = n, count
        self.x = torch.zeros(count, 4 ** n, dtype=torch.float64, device=_device())
        idx = torch.zeros(1, dtype=torch.int64)
        for q in range(n):
            idx = torch.cat([idx, idx + 3 * 4 ** (n - 1 - q)])
        self.x[:, idx.to(self.x.device)] = 0.5 ** n
        self.todo = [None] * n

    def map(self, q, m):
        self.todo[q] = m if self.todo[q] is None else m @ self.todo[q]

    def noise(self, m):
        for q in range(self.n):
            self.map(q, m)

    def settle(self, q):
        m, self.todo[q] = self.todo[q], None
        if m is None:
            return
        v = self.x.view(self.count, 4 ** q, 4, 4 ** (self.n - 1 - q))
        if m.ndim == 2:
            rows = []
            for i in range(4):
                if np.array_equal(m[i], np.eye(4)[i]):
                    rows.append(None)
                    continue
                y = None
                for j in range(4):
                    if m[i, j] != 0.0:
                        y = v[:, :, j] * float(m[i, j]) if y is None else y.add_(v[:, :, j], alpha=float(m[i, j]))
                rows.append(torch.zeros_like(v[:, :, 0]) if y is None else y)
        else:
            c = torch.from_numpy(np.ascontiguousarray(m)).to(self.x.device)[:, :, :, None, None]
            rows = [None]
            for i in range(1, 4):
                y = v[:, :, 0] * c[:, i, 0]
                for j in range(1, 4):
                    y.addcmul_(v[:, :, j], c[:, i, j])
                rows.append(y)
        for i, y in enumerate(rows):
            if y is not None:
                v[:, :, i] = y

    def cx(self, ctl, tgt, cav=1.0, mean=0.0):
        """CX under the averaged pulse error: cav and mean numbers or one per instance."""
        self.settle(ctl)
        self.settle(tgt)
        n = self.n
        lo, hi = min(ctl, tgt), max(ctl, tgt)
        v = self.x.view(self.count, 4 ** lo, 4, 4 ** (hi - lo - 1), 4, 4 ** (n - 1 - hi))
        c2 = 4 * cav - 3
        co = {'c': cav * np.cos(mean), 's': cav * np.sin(mean), 'p': 0.5 * (1 + c2 * np.cos(2 * mean)),
              'm': 0.5 * (1 - c2 * np.cos(2 * mean)), 'x': c2 * np.sin(mean) * np.cos(mean)}

        def at(k):
            pc, pt = divmod(k, 4)
            return v[:, :, pc, :, pt] if ctl < tgt else v[:, :, pt, :, pc]

        def times(w):
            k = co[w[-1]] * (-1.0 if w[0] == '-' else 1.0)
            if np.ndim(k) == 0:
                return float(k)
            return torch.from_numpy(np.asarray(k)).to(self.x.device)[:, None, None, None]

        old = {k: at(k).clone() for k in range(2, 16) if k not in (12, 13)}
        for dst, terms in _CX_ROWS.items():
            y = None
            for src, w in terms:
                k = times(w)
                if isinstance(k, float) and k == 0.0:
                    continue
                y = old[src] * k if y is None else y.add_(old[src] * k)
            at(dst).copy_(y)

    def settle_all(self):
        for q in range(self.n):
            self.settle(q)

    def probabilities(self, vec, err):
        """Outcome probabilities [count, 2**n], every qubit measured along ``vec``; err a number or one per instance."""
        self.settle_all()
        return _probabilities(self.x, self.n, [vec] * self.n, err)


# rows of the CX map that are not the identity, index 4 * control + target (I, X, Y, Z)
_CX_ROWS = {2: [(2, 'm'), (14, 'p'), (3, '-x'), (15, 'x')], 14: [(2, 'p'), (14, 'm'), (3, 'x'), (15, '-x')],
            3: [(3, 'm'), (15, 'p'), (2, 'x'), (14, '-x')], 15: [(3, 'p'), (15, 'm'), (2, '-x'), (14, 'x')],
            4: [(5, 'c'), (8, '-s')], 5: [(4, 'c'), (9, '-s')], 6: [(10, '-s'), (11, 'c')],
            7: [(10, '-c'), (11, '-s')], 8: [(4, 's'), (9, 'c')], 9: [(5, 's'), (8, 'c')],
            10: [(6, 's'), (7, '-c')], 11: [(6, 'c'), (7, 's')]}


def _probabilities(x, n, vecs, err):
    """[count, outcomes]: qubit q measured along vecs[q] (None: summed over its outcomes)."""
    count = x.shape[0]
    e = torch.as_tensor(np.asarray(err, dtype=np.float64), device=x.device).reshape(-1, 1, 1)
    t = x
    for q in range(n):              # qubit q becomes the slowest remaining axis of t's right part
        t = t.reshape(count, -1, 4, 4 ** (n - 1 - q))
        i = t[:, :, 0]
        if vecs[q] is None:
            t = 2.0 * i
        else:
            d = sum(float(vecs[q][k]) * t[:, :, k + 1] for k in range(3)) * e
            t = torch.stack([i + d, i - d], dim=2)
    return t.reshape(count, -1)


def _matrix(x, n):
    """The 2**n x 2**n matrix of coefficients x[4**n]."""
    t = x.to(torch.complex128).reshape(-1)
    for q in range(n):
        v = t.reshape(4 ** q, 4, 4 ** (n - 1 - q))
        i, a, b, z = v[:, 0], v[:, 1], v[:, 2], v[:, 3]
        t = torch.stack([i + z, a - 1j * b, a + 1j * b, i - z], dim=1).reshape(-1)
    t = t.reshape([2, 2] * n)
    return t.permute(list(range(0, 2 * n, 2)) + list(range(1, 2 * n, 2))).reshape(2 ** n, 2 ** n)


def _levels(n, gates, barriers):
    """Clock cycles: one gate each behind barriers, else each gate as early as its qubits allow."""
    if barriers:
        return [[g] for g in gates]
    free, levels = [0] * n, []
    for g in gates:
        qs = g[1:3] if g[0] == 'cx' else g[1:2]
        at = max(free[q] for q in qs)
        if at == len(levels):
            levels.append([])
        levels[at].append(g)
        for q in qs:
            free[q] = at + 1
    return levels


def _noise_map(f, p, g):
    """Memory noise of one cycle; f, p, g numbers or arrays (one map each)."""
    f, p, g = np.broadcast_arrays(f, p, g)
    m = np.zeros(f.shape + (4, 4))
    m[..., 0, 0] = 1.0
    m[..., 1, 1] = m[..., 2, 2] = np.sqrt(g) * f
    m[..., 3, 3] = g
    m[..., 3, 0] = (1 - g) * (2 * p - 1)
    return m


def _gate_map(g, c):
    """4x4 map of a u1 / u3 with <cos> = c on each rotation (c an array: one map each)."""
    c = np.asarray(c, dtype=np.float64)

    def plane(a, i, j):
        m = np.zeros(c.shape + (4, 4))
        m[...] = np.eye(4)
        m[..., i, i] = m[..., j, j] = c * math.cos(a)
        m[..., i, j], m[..., j, i] = -c * math.sin(a), c * math.sin(a)
        return m
    if g[0] == 'u1':
        return plane(g[2], 1, 2)
    return plane(g[3], 1, 2) @ plane(g[2], 3, 1) @ plane(g[4], 1, 2)


def _simulate(sim, gates, barriers, noise, c, cav=1.0):
    for level in _levels(sim.n, gates, barriers):
        for g in level:
            if g[0] == 'cx':
                sim.cx(g[1], g[2], cav)
            else:
                sim.map(g[1], _gate_map(g, c))
        sim.noise(noise)


_Z = (0.0, 0.0, 1.0)


def _exact_state(case, seed, barriers):
    sim = _Exact(case['n'])
    noise = _noise_map(_NOISE['decoherence'], 1.0, _NOISE['decay'])
    _simulate(sim, _gates_of(case, seed), barriers, noise, math.exp(-0.5 * _NOISE['rotation_sigma'] ** 2))
    probs = sim.probabilities(_Z, 1.0 - _NOISE['depolarisation'])[0]
    sim.noise(noise)          # the cycle of the measurement
    sim.settle_all()
    return sim.x[0], probs


def _exact_execute(case, seed):
    x, p = _exact_state(case, seed, False)
    rho = _matrix(x, case['n'])
    return {'coeffmatrix': x.cpu().numpy(), 'densitymatrix': rho.cpu().numpy(), 'probability': p.cpu().numpy()}


def _exact_circuit(case, seed):
    x, p = _exact_state(case, seed, True)
    return {'state': x, 'probability': p}


def _exact_sweep(case, seed):
    specs = _sweep_specs(case, seed)
    # the batch packs its instances largest first
    order = sorted(range(len(specs)), key=lambda i: -(4 ** specs[i]['n'] * specs[i]['depth']))
    out = []
    for i in order:
        s = specs[i]
        n = s['n']
        ang = np.random.default_rng(s['seed']).uniform(0.0, 2 * PI, size=(s['depth'], n, 3))
        gates = []
        for L in range(s['depth']):
            gates += [('u3', q, *(float(a) for a in ang[L, q])) for q in range(n)]
            gates += [('cx', a, a + 1) for a in range(L % 2, n - 1, 2)]
        sim = _Exact(n)
        _simulate(sim, gates, False, _noise_map(s['decoherence'], 1.0, s['decay']), 1.0)
        out.append(sim.probabilities(_Z, 1.0 - s['depolarisation'])[0])
    return {'probability': torch.cat(out)}


def _exact_template(case, seed):
    raw = _noise_points(case['points'], seed)
    out = []
    step = max(1, (1 << 30) // 4 ** case['n'])
    for s0 in range(0, len(raw), step):
        r = raw[s0:s0 + step]
        sim = _Exact(case['n'], len(r))
        _simulate(sim, _brick(case['n'], case['layers'], seed), False, _noise_map(1 - r[:, 1], r[:, 3], 1 - r[:, 2]),
                  np.exp(-0.5 * r[:, 4] ** 2), 1 - r[:, 5])
        out.append(sim.probabilities(_Z, 1 - r[:, 0]))
    return {'probability': torch.cat(out)}


def _forward(flat, x, nout):
    """Logits [members, rows, nout] of flat FP64 parameters on inputs x [members, rows, 64]."""
    widths = _WIDTHS + (nout,)
    h, o = x, 0
    for li in range(4):
        a, b = widths[li + 1], widths[li]
        w = flat[:, o:o + a * b].reshape(-1, a, b)
        h = h @ w.transpose(1, 2) + flat[:, None, o + a * b:o + a * b + a]
        o += a * b + a
        if li < 3:
            h = torch.nn.functional.gelu(h, approximate='tanh')
    return h


def _pad(x):
    return torch.nn.functional.pad(x.to(torch.float64), (0, 58))


def _exact_train(case, seed):
    samples = 4 * case['batch']
    x, y = _mlp_data(samples, case['nout'], seed)
    idx = _mlp_index(case, samples, seed)[0].long()
    with torch.enable_grad():
        flat = _mlp_params(case['members'], case['nout'], seed).to(torch.float64).requires_grad_(True)
        t = y.to(torch.float64)[idx]
        logq = torch.log_softmax(_forward(flat, _pad(x)[idx], case['nout']), dim=2)
        loss = (t * (torch.log(t) - logq)).sum(dim=2)
        grads, = torch.autograd.grad(loss.mean(dim=1).sum(), flat)
    # the first Adam step: both bias-corrected moments are the gradient's own
    params = flat.detach() - 1e-3 * grads / (grads.abs() + 1e-8)
    return {'loss_rows': loss.detach(), 'grads': grads, 'params': params}


def _exact_predict(case, seed):
    x, y = _mlp_data(case['points'], case['nout'], seed)
    flat = _mlp_params(case['members'], case['nout'], seed).to(torch.float64)
    xs = _pad(x)[None].expand(case['members'], -1, -1)
    q = torch.softmax(_forward(flat, xs, case['nout']), dim=2)
    mean = q.mean(dim=0)
    return {'members': q, 'mean': mean, 'spread': 0.5 * (q - mean).abs().sum(dim=2).mean(dim=0),
            'tv': 0.5 * (mean - y.to(torch.float64)).abs().sum(dim=1)}


def _exact_gates(case, seed):
    sim = _Exact(case['n'])
    noise = _noise_map(_F, _P, _G)
    last = None
    for g in _plain_maps(case, seed):
        is_cx = g[0] == 'cx'
        if last is not None and is_cx != last:
            sim.noise(noise)
        last = is_cx
        if is_cx:
            sim.cx(g[1], g[2], *_TSP)
        else:
            sim.map(g[0], g[1])
    sim.noise(noise)
    return {'probability': sim.probabilities(_Z, _ERR)[0], 'state': sim.x[0]}


def _exact_readout(case, seed):
    n = case['n']
    x = _mixed_state(n, seed, _dtype(case)).to(torch.float64)
    other = _mixed_state(n, seed + 1, _dtype(case)).to(torch.float64)
    part = set(_subset(n))
    return {'z': _probabilities(x[None], n, [_Z] * n, _ERR)[0],
            'x': _probabilities(x[None], n, [(1.0, 0.0, 0.0) if q in part else None for q in range(n)], _ERR)[0],
            'n': _probabilities(x[None], n, [_direction(seed)] * n, _ERR)[0],
            'overlap': (x @ other).reshape(1) * 2.0 ** n, 'rho': _matrix(x, n),
            'coefficients': torch.where(x.abs() < 1e-15, torch.zeros_like(x), x)}


_EXACT = {'execute': _exact_execute, 'circuit': _exact_circuit, 'sweep': _exact_sweep, 'template': _exact_template,
          'train': _exact_train, 'predict': _exact_predict, 'gates': _exact_gates, 'readout': _exact_readout}
