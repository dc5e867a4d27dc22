"""dm_compose_passes: the round images of several passes in one launch."""
import ctypes

import numpy as np
import pytest

from qiskit_aakash_gb300 import _native as N
from qiskit_aakash_gb300 import program as P


def _passes(n, count, seed):
    """(DmBatchPass, coefficients, format) of the planned passes of random maps, CX, pair maps."""
    rng = np.random.default_rng(seed)
    ops = []
    for _ in range(count):
        k = rng.integers(4)
        a, b = (int(x) for x in rng.choice(n, 2, replace=False))
        if k == 0:
            m = rng.normal(size=(4, 4)) * 0.5
            if rng.random() < 0.5:
                m[0] = [1, 0, 0, 0]
            ops.append(P.Op('map1', (a,), m))
        elif k == 1:
            coef, ideal = P.cx_coefficients([1.0, 0.0] if rng.random() < 0.5 else [0.98, 0.03])
            ops.append(P.Op('cx', (a, b), np.array(coef), ideal))
        elif k == 2:
            ops.append(P.Op('diag2', (a, b), rng.normal(size=16)))
        else:
            ops.append(P.Op('map2', (a, b), rng.normal(size=(16, 16)) * 0.3))
    out = []
    for i, p in enumerate(P.plan_passes(ops, n, 7, 2)):
        kernel = ('tc', 'tma')[i % 2]
        coefs = []
        try:
            _, bp = P.encode_pass_tc_ops(p, n, coefs, kernel)
        except P.TcPlanError:
            coefs = []
            _, bp = P.encode_pass_tc_ops(p, n, coefs, 'tc')
            kernel = 'tc'
        out.append((bp, np.concatenate(coefs), N.DM_IMAGE_TMA if kernel == 'tma' else N.DM_IMAGE_TC))
    return out


def _tables(items):
    passes = (N.DmBatchPass * len(items))(*[bp for bp, _, _ in items])
    rounds, mats, size = [], 0, 0
    for k, (bp, coefs, fmt) in enumerate(items):
        for r in range(bp.nrounds):
            e = N.DmComposeRound()
            e.pass_, e.round, e.format, e.mats_off, e.image_off = k, r, fmt, mats, size
            rounds.append(e)
            size += 8192 if fmt == N.DM_IMAGE_TMA else 12288
        mats += coefs.size
    return passes, (N.DmComposeRound * len(rounds))(*rounds), np.concatenate([c for _, c, _ in items]), size


@pytest.mark.gpu
def test_equal_to_one_launch_per_pass():
    import torch
    items = _passes(10, 150, 5)
    assert len(items) >= 4
    passes, rounds, mats, size = _tables(items)

    def up(b):
        return torch.from_numpy(np.frombuffer(bytes(b), dtype=np.uint8).copy()).cuda()

    def vp(t, off=0):
        return ctypes.c_void_p(t.data_ptr() + off)

    pd, rd, md = up(passes), up(rounds), torch.from_numpy(mats).cuda()
    got = torch.zeros(size, dtype=torch.int16, device='cuda')
    want = torch.zeros_like(got)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    N.call('dm_compose_passes', passes, vp(pd), len(items), rounds, vp(rd), len(rounds), vp(md),
           ctypes.c_size_t(mats.size), vp(got), ctypes.c_size_t(size), s)
    for e in rounds:
        if e.round == 0:
            bp, coefs, fmt = items[e.pass_]
            N.call('dm_compose_rounds', fmt, ctypes.byref(bp), vp(md, 8 * e.mats_off), ctypes.c_size_t(coefs.size),
                   vp(want, 2 * e.image_off), ctypes.c_size_t(size - e.image_off), s)
    assert torch.equal(got, want) and int((got != 0).sum()) > 0


def test_bad_tables_are_rejected_on_host():
    """Checked before any CUDA call."""
    items = _passes(9, 30, 6)
    passes, rounds, mats, size = _tables(items)
    dev = ctypes.c_void_p(1 << 20)

    def run(passes=passes, rounds=rounds, count=mats.size, images=dev, nimg=size, npasses=len(items)):
        return N.lib().dm_compose_passes(passes, dev, npasses, rounds, dev, len(rounds), dev, ctypes.c_size_t(count),
                                         images, ctypes.c_size_t(nimg), None)

    def changed(**kw):
        bad = (N.DmComposeRound * len(rounds)).from_buffer_copy(bytes(rounds))
        for k, v in kw.items():
            setattr(bad[len(rounds) - 1], k, v)
        return bad

    last = rounds[len(rounds) - 1]
    assert run(images=ctypes.c_void_p((1 << 20) + 8)) == N.DM_ERR_ARG
    assert run(nimg=size - 1) == N.DM_ERR_ARG
    assert run(count=mats.size - 1) == N.DM_ERR_PROGRAM
    assert run(npasses=len(items) - 1) == N.DM_ERR_ARG
    assert run(rounds=changed(format=7)) == N.DM_ERR_ARG
    assert run(rounds=changed(pass_=-1)) == N.DM_ERR_ARG
    assert run(rounds=changed(mats_off=-1)) == N.DM_ERR_ARG
    assert run(rounds=changed(image_off=last.image_off + 4)) == N.DM_ERR_ARG
    assert run(rounds=changed(round=items[-1][0].nrounds)) == N.DM_ERR_PROGRAM
    bad = (N.DmBatchPass * len(items)).from_buffer_copy(bytes(passes))
    bad[0].ops[0].kind = 9
    assert run(passes=bad) == N.DM_ERR_PROGRAM
