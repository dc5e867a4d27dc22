"""The compiled planner against the same scan written over sets of axes, and its descriptors against program order."""
import ctypes
import importlib
import os
import subprocess
import sys

import numpy as np
import pytest

from test_planner import apply_op, random_ops

P = importlib.import_module('qiskit-aakash_gb300.program')
N = importlib.import_module('qiskit-aakash_gb300._native')


def scan(ops, n, kmax, low, partial):
    """(pass, slot) of each op, and the passes' resident sets."""
    kmax = min(kmax, n)
    base = set(range(n - 1, n - 1 - min(low, kmax), -1))
    where, residents, pending = [(-1, -1)] * len(ops), [], list(range(len(ops)))
    while pending:
        resident, blocked, taken, last, slots, closed = set(base), set(), [], {}, 0, False
        for i in pending:
            axes = set(ops[i].axes)
            if blocked & axes or len(resident | axes) > kmax or slots >= N.DM_MAX_PASS_OPS:
                blocked |= axes
                if (len(resident) >= kmax and blocked >= resident) or len(blocked) >= n:
                    closed = True
                    break
                continue
            resident |= axes
            if ops[i].kind == 'map1' and last.get(ops[i].axes[0]) is not None:
                slot = last[ops[i].axes[0]]
            else:
                slot, slots = slots, slots + 1
                for a in axes:
                    last[a] = slot if ops[i].kind == 'map1' else None
            taken.append((i, slot))
        assert taken
        if partial and not closed:
            break
        for i, slot in taken:
            where[i] = (len(residents), slot)
        residents.append(resident)
        gone = {i for i, _ in taken}
        pending = [i for i in pending if i not in gone]
    return where, residents


CASES = [(1, 6, 2), (2, 6, 2), (5, 4, 2), (8, 6, 2), (8, 7, 3), (9, 4, 0), (6, 2, 0), (17, 7, 2), (16, 3, 0)]


@pytest.mark.parametrize('partial', [False, True])
@pytest.mark.parametrize('n,kmax,low', CASES)
def test_same_passes_as_the_scan_over_sets(n, kmax, low, partial):
    rng = np.random.default_rng(n * 100 + kmax * 10 + low + partial)
    for count in (0, 1, 2, 40, 300, 900):
        ops = random_ops(rng, n, count)
        plan = P.Plan(ops, n, kmax, low, partial)
        where, residents = scan(ops, n, kmax, low, partial)
        assert list(zip(plan.pass_of.tolist(), plan.slot_of.tolist())) == where
        assert [{q for q in range(n) if m >> q & 1} for m in plan.resident.tolist()] == residents
        assert plan.rest() == [op for op, (p, _) in zip(ops, where) if p < 0]


@pytest.mark.parametrize('width', [2, 3, None])
@pytest.mark.parametrize('n,kmax,low', [(1, 6, 2), (3, 6, 2), (5, 4, 2), (8, 6, 2), (8, 7, 2), (7, 5, 0)])
def test_descriptors_equal_program_order(n, kmax, low, width):
    rng = np.random.default_rng(7 * n + kmax + low)
    for count in (1, 30, 250):
        ops = random_ops(rng, n, count)
        for op in ops:                  # bounded growth, so that a relative bound means something
            if op.kind in ('map1', 'map2'):
                op.data = op.data / np.abs(op.data).sum(axis=1, keepdims=True)
            elif op.kind == 'diag2':
                op.data = np.clip(op.data, -1, 1)
        want = got = rng.normal(size=4 ** n)
        for op in ops:
            want = apply_op(want, n, op)
        plan = P.Plan(ops, n, kmax, low)
        mats = np.empty(plan.coefficients())
        descs, used = P.encode_plan(plan, n, np.float64, width, mats.ctypes.data, mats.size)
        if kmax <= 6:      # the FP32 form: the same descriptors, the coefficients rounded once
            mats32 = np.empty(plan.coefficients(), np.float32)
            descs32, used32 = P.encode_plan(plan, n, np.float32, width, mats32.ctypes.data, mats32.size)
            assert used32 == used and bytes(descs32) == bytes(descs)
            assert np.array_equal(mats32[:used], mats[:used].astype(np.float32))
        at = 0
        for d in descs:
            axes = list(d.axes[:d.k])
            assert axes == sorted(axes, reverse=True)
            for i in range(d.nops):
                o = d.ops[i]
                assert o.moff == at
                kind = {v: k for k, v in P._OP_KINDS.items()}[o.kind]
                size = {'map1': 16, 'cx': 5, 'diag2': 16, 'map2': 256}[kind]
                data = mats[at:at + size]
                at += size
                local = (o.a,) if kind == 'map1' else (o.a, o.b)
                if d.nrounds:
                    r = next(r for r in range(d.nrounds) if i < d.round_end[r])
                    digits = list(d.round_axes[r])
                    assert digits[width:] == [-1] * (4 - width) and digits[:width] == sorted(set(digits[:width]))
                    assert tuple(digits[(o.flags >> (8 + 4 * j)) & 15] for j in range(len(local))) == local
                shape = {'map1': (4, 4), 'map2': (16, 16)}.get(kind, (size,))
                if kind == 'map1':
                    assert bool(o.flags & N.DM_MAP1_ROW0_IDENTITY) == bool(data[0] == 1 and not data[1:4].any())
                    assert bool(o.flags & N.DM_MAP1_XY_UNITAL) == bool(data[4] == 0 and data[8] == 0)
                got = apply_op(got, n, P.Op(kind, tuple(axes[a] for a in local), data.reshape(shape),
                                            bool(kind == 'cx' and o.flags & N.DM_CX_IDEAL)))
        assert at == used
        # every op rounds each value once per term: 250 ops x 16 terms x half an ulp, doubled
        eps = np.finfo(np.float64).eps
        np.testing.assert_allclose(got, want, rtol=0, atol=250 * 16 * eps * np.abs(want).max() + 1e-300)


def test_full_pass_of_128_ops_and_what_is_refused():
    coef, ideal = P.cx_coefficients([0.99, 0.01])
    ops = [P.Op('cx', (i % 2, 1 - i % 2), np.array(coef), ideal) for i in range(300)]
    passes = P.plan_passes(ops, 2, 2, 2)
    assert [len(p.ops) for p in passes] == [128, 128, 44]
    with pytest.raises(RuntimeError, match='no progress'):
        P.plan_passes([P.Op('cx', (0, 1), np.array(coef), ideal)], 4, 1, 0)
    with pytest.raises(N.NativeError):
        P.plan_passes([P.Op('map1', (4,), np.eye(4))], 4, 4, 2)
    with pytest.raises(ValueError):
        P.plan_passes([P.Op('swap', (0, 1), np.eye(16))], 4, 4, 2)
    # a buffer that is too small is an error, not an overrun
    plan = P.Plan([P.Op('map1', (0,), np.eye(4))], 1, 1, 0)
    mats = np.full(32, 7.0)
    with pytest.raises(N.NativeError):
        P.encode_plan(plan, 1, np.float64, None, mats.ctypes.data, 15)
    assert (mats == 7.0).all()
    with pytest.raises(ValueError):
        P.encode_plan(P.Plan([P.Op('map1', (0,), np.eye(3))], 1, 1, 0), 1, np.float64, None, mats.ctypes.data, 16)


@pytest.mark.parametrize('kinds,axes,slots,ok', [
    (('map1', 'map1', 'map1'), ((0,), (1,), (0,)), (0, 1, 0), True),
    (('cx', 'cx'), ((0, 1), (0, 1)), (0, 0), False),              # 5 coefficients each
    (('diag2', 'diag2'), ((0, 1), (0, 1)), (0, 0), False),
    (('cx', 'map1'), ((0, 1), (0,)), (0, 0), False),
    (('map1', 'cx'), ((0,), (0, 1)), (0, 0), False),
    (('map1', 'map1'), ((0,), (1,)), (0, 0), False),              # two axes
    (('map1', 'map1'), ((0,), (1,)), (0, 2), False),              # a gap
    (('map1', 'map1'), ((0,), (1,)), (1, 0), False)])
@pytest.mark.parametrize('width', [None, 2])
def test_slots_that_no_scan_gives_are_refused(kinds, axes, slots, ok, width):
    size = {'map1': (4, 4), 'cx': (5,), 'diag2': (16,)}
    ops = [P.Op(k, a, np.ones(size[k])) for k, a in zip(kinds, axes)]
    plan = P.Plan(ops, 2, 2, 2)
    assert len(plan.resident) == 1
    plan.slot_of = np.array(slots, dtype=np.int32)
    mats = np.full(64, 7.0)
    if ok:
        _, used = P.encode_plan(plan, 2, np.float64, width, mats.ctypes.data, mats.size)
        assert used == 32
        return
    with pytest.raises(N.NativeError) as e:
        P.encode_plan(plan, 2, np.float64, width, mats.ctypes.data, mats.size)
    assert e.value.code == N.DM_ERR_ARG
    assert (mats == 7.0).all()


@pytest.mark.parametrize('data', [
    [np.ones(4), np.ones(28)],                        # two maps whose lengths add up to two maps'
    [np.eye(4), np.ones(17)], [np.eye(4), np.ones(15)]])
def test_operations_of_the_wrong_length_are_refused(data):
    plan = P.Plan([P.Op('map1', (q,), d) for q, d in enumerate(data)], 2, 2, 2)
    mats = np.full(64, 7.0)
    with pytest.raises(ValueError):
        P.encode_plan(plan, 2, np.float64, None, mats.ctypes.data, mats.size)
    cx = P.Op('cx', (0, 1), np.ones(16))
    diag = P.Op('diag2', (0, 1), np.ones(5))          # 16 and 5 the wrong way round
    with pytest.raises(ValueError):
        P.encode_plan(P.Plan([cx, diag], 2, 2, 2), 2, np.float64, None, mats.ctypes.data, mats.size)
    assert (mats == 7.0).all()
    P.encode_plan(P.Plan([P.Op('map1', (0,), np.eye(4).tolist())], 2, 2, 2), 2, np.float64, None, mats.ctypes.data, 64)


_NO_MEMORY = """
import ctypes, importlib, resource
import numpy as np
N = importlib.import_module('qiskit-aakash_gb300._native')
L, count = N.lib(), 1 << 21
vp = lambda a: ctypes.c_void_p(a.ctypes.data)
table = np.zeros((count, 4), np.int16)
table[:, 0] = N.DM_OP_MAP1
pass_of, slot_of, mats = np.zeros(count, np.int32), np.zeros(count, np.int32), np.zeros(16)
resident, coefs, descs = np.ones(count, np.uint32), np.zeros((count, 16)), (N.DmPass * 1)()
npasses, used = ctypes.c_int32(), ctypes.c_size_t()
pages = int(open('/proc/self/statm').read().split()[0])
limit = pages * resource.getpagesize() + (4 << 20)          # the calls' lists take 8 and 16 MB
resource.setrlimit(resource.RLIMIT_AS, (limit, limit))
print(L.dm_plan_passes(1, 1, 0, vp(table), count, 0, vp(pass_of), vp(slot_of), vp(resident), ctypes.byref(npasses)),
      L.dm_encode_passes(1, N.DM_F64, 0, 6, vp(table), count, vp(coefs), vp(pass_of), vp(slot_of), vp(resident), 1, 0,
                         ctypes.cast(descs, ctypes.c_void_p), vp(mats), 16, ctypes.byref(used)))
"""


@pytest.mark.skipif(not sys.platform.startswith('linux'), reason='limits its own address space')
def test_no_memory_is_an_error_code():
    """An allocation that fails in the planner comes back as a status, not as an exception through the C ABI."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(P.__file__)))
    r = subprocess.run([sys.executable, '-c', _NO_MEMORY], cwd=root, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == [str(N.DM_ERR_MEMORY)] * 2
