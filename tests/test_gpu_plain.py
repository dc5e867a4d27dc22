"""Single-operation sweeps and read-outs at the edges of their kernels, against the CPU oracle:
every axis and pair, maps of every zero pattern, states off 16-byte alignment, register sizes on
both sides of each split into sweeps, and decay factors on both sides of the scale-at-the-end rule.

Tolerances: eps = 2**-53 (FP64) or 2**-24 (FP32) times the operations on a coefficient's path times
the largest intermediate the operands allow."""
import ctypes

import numpy as np
import pytest

from oracle import dm_oracle as O
from qiskit_aakash_gb300 import _native as N
from qiskit_aakash_gb300 import program as P

pytestmark = pytest.mark.gpu
EPS = {N.DM_F64: 2.0 ** -53, N.DM_F32: 2.0 ** -24}


def _torch():
    import torch
    return torch


def _vp(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(_torch().cuda.current_stream().cuda_stream)


def _state(a, dtype, shift=0):
    """``a`` on the device, ``shift`` elements past a 16-byte boundary."""
    torch = _torch()
    t = torch.zeros(a.size + 16, dtype=torch.float64 if dtype == N.DM_F64 else torch.float32, device='cuda')
    v = t[shift:shift + a.size]
    v.copy_(torch.from_numpy(a))
    return v


def _rand(n, dtype, seed):
    a = np.random.default_rng(seed).normal(size=4 ** n)
    return a.astype(np.float32).astype(np.float64) if dtype == N.DM_F32 else a


@pytest.mark.parametrize('dtype', [N.DM_F64, N.DM_F32])
@pytest.mark.parametrize('shift', [0, 1])
@pytest.mark.parametrize('n', [1, 2, 3, 4, 6, 7, 9, 10, 11])
def test_memory_noise_sweeps(n, shift, dtype):
    for seed, (f, p, g) in enumerate([(0.97, 0.2, 0.93), (0.9, 1.0, 0.5), (0.8, 0.9, 0.49), (0.7, 0.3, 0.0),
                                      (0.0, 1.0, 1.0)]):
        a = _rand(n, dtype, 10 * n + seed)
        t = _state(a, dtype, shift)
        N.call('dm_apply_memory_noise', _vp(t), n, dtype, f, p, g, _stream())
        want = O.memory_noise(a.copy(), n, f, p, g)
        # each axis at most doubles a coefficient (|Z| + |I|), two roundings per axis
        bound = EPS[dtype] * (2 * n + 4) * np.abs(a).max() * (1 + abs(1 - g)) ** n * 2
        np.testing.assert_allclose(t.double().cpu().numpy(), want, rtol=0, atol=bound)


def _maps(rng):
    rot = P.rotation_ptm('ry', 0.7, (0.99, 0.01)) @ P.rotation_ptm('rz', 1.9, (0.98, 0.02))
    tp = P.noise_ptm(0.9, 0.8, 0.95) @ rot
    row0 = rng.normal(size=(4, 4))
    row0[0] = [1, 0, 0, 0]
    return [rot, tp, row0, rng.normal(size=(4, 4))]


@pytest.mark.parametrize('dtype', [N.DM_F64, N.DM_F32])
@pytest.mark.parametrize('shift', [0, 1])
@pytest.mark.parametrize('n', [1, 2, 3, 5])
def test_map1_every_axis_and_pattern(n, shift, dtype):
    rng = np.random.default_rng(n)
    for q in range(n):
        for k, m in enumerate(_maps(rng)):
            a = _rand(n, dtype, 7 * n + k)
            t = _state(a, dtype, shift)
            N.call('dm_apply_map1', _vp(t), n, dtype, q, N.f64_array(m.reshape(16)), _stream())
            want = np.einsum('ij,ajb->aib', m, a.reshape(4 ** q, 4, 4 ** (n - 1 - q))).reshape(-1)
            bound = EPS[dtype] * 8 * np.abs(a).max() * np.abs(m).sum(axis=1).max()
            np.testing.assert_allclose(t.double().cpu().numpy(), want, rtol=0, atol=bound)


@pytest.mark.parametrize('dtype', [N.DM_F64, N.DM_F32])
@pytest.mark.parametrize('shift', [0, 1])
@pytest.mark.parametrize('n', [2, 3, 5])
def test_cx_every_pair(n, shift, dtype):
    for c in range(n):
        for q in range(n):
            if c == q:
                continue
            for tsp in ([1.0, 0.0], [0.96, 0.07]):
                a = _rand(n, dtype, 16 * c + q)
                t = _state(a, dtype, shift)
                N.call('dm_apply_cx', _vp(t), n, dtype, c, q, N.f64_array(tsp), _stream())
                bound = EPS[dtype] * 16 * np.abs(a).max()
                np.testing.assert_allclose(t.double().cpu().numpy(), O.cx_apply(a.copy(), n, c, q, tsp), rtol=0,
                                           atol=bound)


@pytest.mark.parametrize('dtype', [N.DM_F64, N.DM_F32])
@pytest.mark.parametrize('n', [1, 2, 3, 5, 6, 7, 8, 9, 10, 11])
def test_matrix_sweeps(n, dtype):
    torch = _torch()
    a = _rand(n, dtype, n)
    t = _state(a, dtype, 1)
    out = torch.empty((2 ** n, 2 ** n), dtype=torch.complex128, device='cuda')
    scratch = torch.empty(N.lib().dm_pauli_to_matrix_scratch_bytes(n), dtype=torch.uint8, device='cuda')
    N.call('dm_pauli_to_matrix', _vp(t), n, dtype, _vp(out), _vp(scratch), _stream())
    got = out.cpu().numpy()
    want = O.pauli_to_matrix(a, n)
    # an entry sums 2**n coefficients through n + 2 additions
    np.testing.assert_allclose(got, want, rtol=0, atol=2 * EPS[N.DM_F64] * (n + 2) * 2 ** n * np.abs(a).max())
    assert np.array_equal(got, got.conj().T)


@pytest.mark.parametrize('dtype', [N.DM_F64, N.DM_F32])
@pytest.mark.parametrize('n', [1, 2, 5, 6, 7, 8, 9, 10])
def test_probability_sweeps(n, dtype):
    torch = _torch()
    a = _rand(n, dtype, 3 * n)
    t = _state(a, dtype, 1)
    bound = 4 * EPS[N.DM_F64] * (3 * n + 2) * 4 ** n * np.abs(a).max()
    v = np.array([0.6, -0.48, 0.64])
    out = torch.empty(2 ** n, dtype=torch.float64, device='cuda')
    scratch = torch.empty(max(8, N.lib().dm_nbasis_probs_scratch_bytes(n)), dtype=torch.uint8, device='cuda')
    N.call('dm_nbasis_probs', _vp(t), n, dtype, N.f64_array(v), 0.95, _vp(out), _vp(scratch), _stream())
    np.testing.assert_allclose(out.cpu().numpy(), O.ensemble_probabilities(a, n, 'N', v, 0.95), rtol=0, atol=bound)
    for basis, code in (('X', 1), ('Y', 2), ('Z', 3)):
        N.call('dm_axis_probs', _vp(t), n, dtype, (ctypes.c_int * n)(*([code] * n)), 0.95, _vp(out), _stream())
        np.testing.assert_allclose(out.cpu().numpy(), O.ensemble_probabilities(a, n, basis, None, 0.95), rtol=0,
                                   atol=bound)


@pytest.mark.parametrize('m', [0, 1, 7, 8, 9, 10, 11, 12, 13])
def test_partial_read_out_sweeps(m):
    """2**m outcomes of the first m of 13 qubits against a Walsh-Hadamard transform of the sub-lattice."""
    torch = _torch()
    n = 13
    t = torch.randn(4 ** n, dtype=torch.float64, device='cuda', generator=torch.Generator('cuda').manual_seed(m))
    out = torch.empty(2 ** m, dtype=torch.float64, device='cuda')
    N.call('dm_axis_probs', _vp(t), n, N.DM_F64, (ctypes.c_int * n)(*([3] * m + [0] * (n - m))), 0.9, _vp(out),
           _stream())
    idx = np.zeros(1, dtype=np.int64)
    pop = np.zeros(1, dtype=np.int64)
    for q in range(m):
        idx = (idx[:, None] + np.array([0, 3 * 4 ** (n - 1 - q)])).reshape(-1)
        pop = (pop[:, None] + np.array([0, 1])).reshape(-1)
    w = t[torch.from_numpy(idx).cuda()].cpu().numpy() * 0.9 ** pop * 2.0 ** (n - m)
    for b in range(m):
        w = w.reshape(-1, 2, 2 ** b)
        w = np.stack([w[:, 0] + w[:, 1], w[:, 0] - w[:, 1]], axis=1)
    w = w.reshape(-1)
    np.testing.assert_allclose(out.cpu().numpy(), w, rtol=0,
                               atol=4 * EPS[N.DM_F64] * (m + 4) * 2 ** n * 8)


def _matrix_parts(a, n):
    """Real and imaginary part of the matrix by additions alone (a product 0 * inf would be NaN)."""
    re, im = a.reshape([4] * n), np.zeros([4] * n)
    with np.errstate(invalid='ignore'):
        for q in range(n):
            (i, x, y, z), (ii, xi, yi, zi) = np.moveaxis(re, q, 0), np.moveaxis(im, q, 0)
            re = np.moveaxis(np.stack([i + z, x + yi, x - yi, i - z]), 0, q)
            im = np.moveaxis(np.stack([ii + zi, xi - y, xi + y, ii - zi]), 0, q)
    order = [2 * j for j in range(n)] + [2 * j + 1 for j in range(n)]
    return tuple(np.transpose(p.reshape([2] * (2 * n)), order).reshape(2 ** n, 2 ** n) for p in (re, im))


@pytest.mark.parametrize('dtype', [N.DM_F64, N.DM_F32])
@pytest.mark.parametrize('n', [1, 2, 5, 6, 7, 8, 9, 10])
def test_matrix_of_infinities_and_nan(n, dtype):
    """An entry's part is infinite or NaN only where a coefficient that it sums is."""
    torch = _torch()
    rng = np.random.default_rng(n)
    for values in ([np.inf], [-np.inf], [np.nan], [np.inf, np.inf, -np.inf, np.nan], [np.nan] * 4 ** n):
        a = _rand(n, dtype, n)
        finite = np.abs(a).max()
        a[rng.choice(4 ** n, size=min(len(values), 4 ** n), replace=False)] = values[:4 ** n]
        t = _state(a, dtype, 1)
        out = torch.empty((2 ** n, 2 ** n), dtype=torch.complex128, device='cuda')
        scratch = torch.empty(N.lib().dm_pauli_to_matrix_scratch_bytes(n), dtype=torch.uint8, device='cuda')
        N.call('dm_pauli_to_matrix', _vp(t), n, dtype, _vp(out), _vp(scratch), _stream())
        got = out.cpu().numpy()
        for g, w in zip((got.real, got.imag), _matrix_parts(a, n)):
            np.testing.assert_allclose(g, w, rtol=0, atol=2 * EPS[N.DM_F64] * (n + 2) * 2 ** n * finite)


@pytest.mark.parametrize('dtype', [N.DM_F64, N.DM_F32])
@pytest.mark.parametrize('n', [1, 2, 3])
def test_memory_noise_of_few_qubits_costs_no_more_than_its_maps(n, dtype):
    """One call against the n one-qubit maps it stands for, host time included."""
    import time
    torch = _torch()
    f, p, g = 0.97, 0.2, 0.93
    k, d = np.sqrt(g) * f, (1 - g) * (2 * p - 1)
    m = N.f64_array([1, 0, 0, 0, 0, k, 0, 0, 0, 0, k, 0, d, 0, 0, g])
    t = _state(_rand(n, dtype, n), dtype)
    s = _stream()

    def noise():
        N.call('dm_apply_memory_noise', _vp(t), n, dtype, f, p, g, s)

    def maps():
        for q in range(n):
            N.call('dm_apply_map1', _vp(t), n, dtype, q, m, s)

    best = {noise: np.inf, maps: np.inf}
    for _ in range(20):
        for call in best:
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for _ in range(100):
                call()
            torch.cuda.synchronize()
            best[call] = min(best[call], time.perf_counter() - t0)
    assert best[noise] < 1.25 * best[maps]
