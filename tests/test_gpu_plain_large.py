"""Whole-state sweeps and read-outs where they take the most of them: 12 to 17 qubits, against closed forms.

The states are sums of two products of one-qubit vectors, (I, X, Y, Z) each, so that a noise channel, a
read-out and a row of the density matrix are such sums too.  The vectors' entries are all of one order, each
its own: a coefficient in the wrong place differs by far more than the bounds.

Tolerances: eps = 2**-53 (FP64) or 2**-24 (FP32, which rounds the state itself) times the operations on a
value's path times the largest value the vectors allow."""
import ctypes

import numpy as np
import pytest

from qiskit_aakash_gb300 import _native as N

pytestmark = pytest.mark.gpu
EPS = {N.DM_F64: 2.0 ** -53, N.DM_F32: 2.0 ** -24}
SIZES = [(12, N.DM_F64), (13, N.DM_F64), (14, N.DM_F64), (12, N.DM_F32), (13, N.DM_F32), (14, N.DM_F32),
         (15, N.DM_F32), (16, N.DM_F32), (17, N.DM_F32)]
TAIL = 12      # the chunks that states are filled and compared in: 4**12 coefficients


def _torch():
    import torch
    return torch


def _vp(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(_torch().cuda.current_stream().cuda_stream)


@pytest.fixture(autouse=True)
def _give_back():
    yield
    _torch().cuda.empty_cache()


def _vectors(n, seed):
    """[2, n, 4]: I in 0.9 .. 1, X, Y, Z of either sign in 0.8 .. 1."""
    r = np.random.default_rng(seed)
    v = r.uniform(0.8, 1.0, size=(2, n, 4)) * r.choice([-1.0, 1.0], size=(2, n, 4))
    v[:, :, 0] = r.uniform(0.9, 1.0, size=(2, n))
    return v


def _product(vs):
    """The product of vectors, the first one slowest (device, FP64)."""
    torch = _torch()
    out = torch.ones(1, dtype=torch.float64, device='cuda')
    for v in vs:
        out = (out[:, None] * torch.from_numpy(np.ascontiguousarray(v)).cuda()[None, :]).reshape(-1)
    return out


def _chunks(v):
    """(offset, values) of the state of ``v``."""
    n = v.shape[1]
    h = max(0, n - TAIL)
    heads = [_product(t[:h]).cpu().tolist() for t in v]
    tails = [_product(t[h:]) for t in v]
    for i in range(4 ** h):
        yield i * 4 ** (n - h), heads[0][i] * tails[0] + heads[1][i] * tails[1]


def _state(v, dtype):
    torch = _torch()
    t = torch.empty(4 ** v.shape[1], dtype=torch.float64 if dtype == N.DM_F64 else torch.float32, device='cuda')
    for off, c in _chunks(v):
        t[off:off + c.numel()] = c
    return t


@pytest.mark.parametrize('n,dtype', SIZES)
@pytest.mark.parametrize('f,p,g', [(0.98, 0.9, 0.95), (0.98, 0.2, 0.45)])
def test_memory_noise(n, dtype, f, p, g):
    v = _vectors(n, n)
    t = _state(v, dtype)
    N.call('dm_apply_memory_noise', _vp(t), n, dtype, f, p, g, _stream())
    k, d = np.sqrt(g) * f, (1 - g) * (2 * p - 1)
    w = v * np.array([1, k, k, g])
    w[:, :, 3] += d * v[:, :, 0]
    # every axis leaves values of at most 1 (g |Z| + |d| |I| <= 1), two roundings each, in two terms
    bound = 2 * EPS[dtype] * (2 * n + 8)
    worst = max(float((t[off:off + c.numel()] - c).abs().max()) for off, c in _chunks(w))
    assert worst <= bound


@pytest.mark.parametrize('n,dtype', SIZES)
def test_probabilities(n, dtype):
    torch = _torch()
    v = _vectors(n, 50 + n)
    t = _state(v, dtype)
    err = 0.9
    for code in (1, 3):
        for free in (0, 1):               # every qubit measured, or all but the first
            m = n - free
            out = torch.empty(2 ** m, dtype=torch.float64, device='cuda')
            N.call('dm_axis_probs', _vp(t), n, dtype, (ctypes.c_int * n)(*([0] * free + [code] * m)), err, _vp(out),
                   _stream())
            i, a = v[:, :, 0], err * v[:, :, code]
            rows = np.stack([i + a, i - a], axis=2)
            want = sum(2.0 ** free * i[z, :free].prod() * _product(rows[z, free:]) for z in range(2))
            bound = 2 * 2 ** free * EPS[dtype] * (3 * n + 8) * (i + np.abs(a)).prod(axis=1).sum()
            assert float((out - want).abs().max()) <= bound
    u = np.array([0.6, -0.48, 0.64])
    out = torch.empty(2 ** n, dtype=torch.float64, device='cuda')
    scratch = torch.empty(N.lib().dm_nbasis_probs_scratch_bytes(n), dtype=torch.uint8, device='cuda')
    N.call('dm_nbasis_probs', _vp(t), n, dtype, N.f64_array(u), err, _vp(out), _vp(scratch), _stream())
    i, a = v[:, :, 0], err * (v[:, :, 1:] @ u)
    rows = np.stack([i + a, i - a], axis=2)
    want = sum(_product(rows[z]) for z in range(2))
    bound = 2 * EPS[dtype] * (5 * n + 8) * (i + err * (np.abs(v[:, :, 1:]) @ np.abs(u))).prod(axis=1).sum()
    assert float((out - want).abs().max()) <= bound


@pytest.mark.parametrize('n,dtype', [s for s in SIZES if s[0] <= 15] + [(15, N.DM_F64)])
def test_matrix_rows(n, dtype):
    torch = _torch()
    v = _vectors(n, 100 + n)
    v[:, :, 3] *= 0.5                     # I - Z of the order of I + Z
    t = _state(v, dtype)
    out = torch.empty((2 ** n, 2 ** n), dtype=torch.complex128, device='cuda')
    scratch = torch.empty(N.lib().dm_pauli_to_matrix_scratch_bytes(n), dtype=torch.uint8, device='cuda')
    N.call('dm_pauli_to_matrix', _vp(t), n, dtype, _vp(out), _vp(scratch), _stream())
    i, x, y, z = np.moveaxis(v, 2, 0)
    one = np.stack([np.stack([i + z, x - 1j * y], axis=2), np.stack([x + 1j * y, i - z], axis=2)], axis=2)
    bound = 2 * EPS[dtype] * (3 * n + 8) * (np.maximum(i + np.abs(z), np.abs(x) + np.abs(y))).prod(axis=1).sum()
    rng = np.random.default_rng(n)
    for r in [0, 2 ** n - 1] + rng.integers(0, 2 ** n, 30).tolist():
        bits = [(r >> (n - 1 - q)) & 1 for q in range(n)]
        want = sum(_product([one[k, q, bits[q]] for q in range(n)]) for k in range(2))
        assert float((out[r] - want).abs().max()) <= bound
        assert float((out[:, r] - want.conj()).abs().max()) <= bound
