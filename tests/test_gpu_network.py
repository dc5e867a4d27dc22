"""The surrogate network's kernels at the edges of their tiles: chunk counts around the GEMM's stages,
rows that do not fill a softmax CTA, weight shapes that do not fill an Adam tile, ragged predictions.

Tolerances: BF16 products are exact in FP32, so a GEMM of K terms is held to K * 2**-24 times the sum
of the terms' magnitudes; softmax and KL sums to (nout + 16) * 2**-24 times theirs."""
import ctypes

import numpy as np
import pytest

from oracle import mlp_oracle as MO
from qiskit_aakash_gb300 import _native as N
from qiskit_aakash_gb300 import surrogate as S

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


def _torch():
    import torch
    return torch


def _bf16(a):
    r = MO.bf16(a).astype(np.float32).view(np.uint32) >> 16
    return _torch().from_numpy(r.astype(np.uint16).view(np.int16)).cuda()


def _f(t):
    return (t.cpu().numpy().view(np.uint16).astype(np.uint32) << 16).view(np.float32)


@pytest.mark.parametrize('K', [64, 128, 192, 256, 320, 448])
@pytest.mark.parametrize('aligned', [True, False])
def test_gemm_stages_and_transposed_copy(K, aligned):
    """1 to 7 chunks through the stages; the transposed copy with and without 16-byte alignment."""
    torch = _torch()
    M, Nn, Z = 256, 128, 2
    rng = np.random.default_rng(K)
    A = MO.bf16(rng.normal(size=(Z, M, K)).astype(np.float32))
    B = MO.bf16(rng.normal(size=(Z, Nn, K)).astype(np.float32))
    pre = rng.normal(size=(Z, M, Nn)).astype(np.float32)
    a, b, pt = _bf16(A), _bf16(B), torch.from_numpy(pre).cuda()
    ld = M + (0 if aligned else 1)
    f32 = torch.zeros((Z, M, Nn), dtype=torch.float32, device='cuda')
    bf = torch.zeros((Z, M, Nn), dtype=torch.int16, device='cuda')
    t = torch.zeros((Z, Nn, ld), dtype=torch.int16, device='cuda')
    status = torch.zeros(1, dtype=torch.int32, device='cuda')
    for epi in (N.DM_MLP_EPI_F32, N.DM_MLP_EPI_GELU_BWD):
        g = N.DmMlpGemm()
        g.epi, g.M, g.N, g.K, g.members = epi, M, Nn, K, Z
        g.A, g.lda, g.a_ms, g.B, g.ldb, g.b_ms = a.data_ptr(), K, M * K, b.data_ptr(), K, Nn * K
        if epi == N.DM_MLP_EPI_F32:
            g.out_f32, g.ld_f32, g.f32_ms = f32.data_ptr(), Nn, M * Nn
        else:
            g.pre, g.ld_pre, g.pre_ms = pt.data_ptr(), Nn, M * Nn
            g.out_bf16, g.ld_bf16, g.bf16_ms = bf.data_ptr(), Nn, M * Nn
            g.out_t, g.ld_t, g.t_ms = t.data_ptr(), ld, Nn * ld
        N.call('dm_mlp_gemm_run', ctypes.byref(g), ctypes.c_void_p(status.data_ptr()), None)
    assert int(status.item()) == 0
    A64, B64 = A.astype(np.float64), B.astype(np.float64)
    want = np.einsum('zmk,znk->zmn', A64, B64)
    terms = np.einsum('zmk,znk->zmn', np.abs(A64), np.abs(B64))
    assert np.all(np.abs(f32.cpu().numpy() - want) <= K * U * terms)
    d = want * MO.gelu_grad(pre.astype(np.float64))
    # one BF16 rounding of the FP32 result (GELU' itself to a few FP32 units of 1)
    assert np.all(np.abs(_f(bf) - d) <= 2.0 ** -8 * np.abs(d) + (K + 32) * U * terms)
    assert np.array_equal(bf.cpu().numpy(), np.swapaxes(t.cpu().numpy()[:, :, :M], 1, 2))


@pytest.mark.parametrize('rows', [1, 31, 32, 40, 100])
@pytest.mark.parametrize('nout', [256, 1024, 4096])
def test_softmax_rows(rows, nout):
    torch = _torch()
    Z = 2
    rng = np.random.default_rng(rows + nout)
    x = (3 * rng.normal(size=(Z, rows, nout))).astype(np.float32)
    t = rng.dirichlet(np.ones(nout) * 0.3, size=(Z, rows)).astype(np.float32)
    lx, lt = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    probs = torch.zeros_like(lx)
    dz = torch.zeros((Z, rows, nout), dtype=torch.int16, device='cuda')
    dzt = torch.zeros((Z, nout, rows), dtype=torch.int16, device='cuda')
    loss = torch.zeros((Z, rows), dtype=torch.float32, device='cuda')
    vp = ctypes.c_void_p
    N.call('dm_mlp_softmax_xent', vp(lx.data_ptr()), vp(lt.data_ptr()), rows, Z, nout, ctypes.c_float(0.25),
           vp(probs.data_ptr()), vp(dz.data_ptr()), vp(dzt.data_ptr()), vp(loss.data_ptr()), None)
    x64 = x.astype(np.float64)
    lq = x64 - x64.max(axis=2, keepdims=True)
    lq -= np.log(np.exp(lq).sum(axis=2, keepdims=True))
    q = np.exp(lq)
    tol = (nout + 16) * U
    got = probs.cpu().numpy()
    # the exponent's own FP32 rounding (|x| < 40) beside the sum's
    assert np.all(np.abs(got - q) <= (tol + 64 * U) * q)
    t64 = t.astype(np.float64)
    terms = np.where(t64 > 0, t64 * (np.log(np.where(t64 > 0, t64, 1.0)) - lq), 0.0)
    assert np.all(np.abs(loss.cpu().numpy() - terms.sum(axis=2)) <= (tol + 64 * U) * (np.abs(terms).sum(axis=2) + 1))
    d = (q - t64) * 0.25
    assert np.all(np.abs(_f(dz) - d) <= 2.0 ** -8 * np.abs(d) + (tol + 64 * U) * q)
    assert np.array_equal(dz.cpu().numpy(), np.swapaxes(dzt.cpu().numpy(), 1, 2))


@pytest.mark.parametrize('shapes', [[(5, 7), (33, 64), (64, 33), (300, 32), (1, 1)],      # element by element
                                    [(8, 4), (36, 64), (64, 36), (300, 32)]])             # four weights at once
def test_adam_of_ragged_shapes(shapes):
    torch = _torch()
    P = sum(o * i + o for o, i in shapes)
    Z = 3
    rng = np.random.default_rng(1)
    p0 = rng.normal(size=(Z, P)).astype(np.float32)
    g = rng.normal(size=(Z, P)).astype(np.float32)
    p, gd = torch.from_numpy(p0).cuda(), torch.from_numpy(g).cuda()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    wb = torch.full((Z, P), 7, dtype=torch.int16, device='cuda')
    wtb = torch.full((Z, P), 7, dtype=torch.int16, device='cuda')
    flat = (ctypes.c_int32 * (2 * len(shapes)))(*[x for s in shapes for x in s])
    vp = ctypes.c_void_p
    N.call('dm_mlp_adam', vp(p.data_ptr()), vp(gd.data_ptr()), vp(m.data_ptr()), vp(v.data_ptr()), ctypes.c_int64(P),
           Z, flat, len(shapes), ctypes.c_float(1e-2), ctypes.c_float(0.9), ctypes.c_float(0.999), ctypes.c_float(1e-8),
           1, vp(wb.data_ptr()), vp(wtb.data_ptr()), None)
    want = p0 - 1e-2 * np.sign(g) * (np.abs(g) / (np.abs(g) + 1e-8))
    got = p.cpu().numpy()
    assert np.max(np.abs(got - want)) < 1e-6
    off = 0
    bits = (MO.bf16(got).view(np.uint32) >> 16).astype(np.uint16).view(np.int16)
    for o, i in shapes:
        for z in range(Z):
            w = bits[z, off:off + o * i]
            assert np.array_equal(wb[z, off:off + o * i].cpu().numpy(), w)
            assert np.array_equal(wtb[z, off:off + o * i].cpu().numpy().reshape(i, o), w.reshape(o, i).T)
        assert int((wb[:, off + o * i:off + o * i + o] != 7).sum()) == 0      # biases have no copies
        off += o * i + o


@pytest.mark.parametrize('points', [1, 127, 128, 129, 300, 513])
def test_predictions_do_not_depend_on_the_last_chunk(points):
    """A last chunk of any length gives each member the rows it has in whole chunks."""
    torch = _torch()
    ens = S.MLPEnsemble(members=3, batch=256, nout=256, seed=2)
    f = torch.rand(1024, 6, device='cuda', generator=torch.Generator('cuda').manual_seed(points)) * 2 - 1
    whole = ens.predict(f)
    assert torch.equal(ens.predict(f[:points].contiguous()), whole[:, :points])
    assert float((whole.sum(dim=2) - 1).abs().max()) < 1e-5
    assert not torch.equal(whole[0], whole[1])


def test_network_calls_reject_bad_arguments():
    """Checked before any launch."""
    ens = S.MLPEnsemble(members=2, batch=128, nout=256)
    for rows in (0, 129, 32):
        with pytest.raises(N.NativeError) as e:
            ens.loss_and_grads(rows)
        assert e.value.code == N.DM_ERR_ARG
    net = ens._net()
    net._obj.count -= 1
    assert N.lib().dm_mlp_forward(net, 128, 0, None) == N.DM_ERR_ARG
    net = ens._net()
    net._obj.h[1] = None
    assert N.lib().dm_mlp_forward(net, 128, 0, None) == N.DM_ERR_ARG


@pytest.mark.parametrize('workspace', [1, 3 << 20, 64 << 20])
@pytest.mark.parametrize('points', [1, 700, 1301])
def test_predictions_do_not_depend_on_the_workspace(points, workspace, monkeypatch):
    """Passes of one batch, of several tiles and of all points; member strides and ragged ends."""
    torch = _torch()
    ens = S.MLPEnsemble(members=3, batch=128, nout=512, seed=4)
    f = torch.rand(points, 6, device='cuda', generator=torch.Generator('cuda').manual_seed(points)) * 2 - 1
    want = torch.cat([ens.predict(f[i:i + 128].contiguous()) for i in range(0, points, 128)], dim=1)
    monkeypatch.setattr(S, 'PREDICT_WORKSPACE', workspace)
    assert ens._predict_rows(points) % 128 == 0
    assert torch.equal(ens.predict(f), want)


@pytest.mark.parametrize('nout', [1024, 1023, 4, 1, 258])
@pytest.mark.parametrize('members', [1, 5, 8])
def test_ensemble_statistics(nout, members):
    """Rows that are and are not multiples of four columns, against FP64 sums."""
    torch = _torch()
    rows = 5
    rng = np.random.default_rng(nout + members)
    p = rng.random((members, rows, nout)).astype(np.float32)
    ref = rng.random((rows, nout)).astype(np.float32)
    pd, rd = torch.from_numpy(p).cuda(), torch.from_numpy(ref).cuda()
    mean = torch.empty((rows, nout), dtype=torch.float32, device='cuda')
    spread, tv = (torch.empty(rows, dtype=torch.float32, device='cuda') for _ in range(2))
    vp = ctypes.c_void_p
    N.call('dm_mlp_ensemble', vp(pd.data_ptr()), rows, members, nout, vp(rd.data_ptr()), vp(mean.data_ptr()),
           vp(spread.data_ptr()), vp(tv.data_ptr()), None)
    mu = p.astype(np.float64).mean(axis=0)
    tol = (nout + 16) * U * max(nout, 1)
    assert np.abs(mean.cpu().numpy() - mu).max() <= 16 * U
    assert np.abs(spread.cpu().numpy() - 0.5 * np.abs(p - mu).sum(axis=2).mean(axis=0)).max() <= tol
    assert np.abs(tv.cpu().numpy() - 0.5 * np.abs(mu - ref).sum(axis=1)).max() <= tol


@pytest.mark.parametrize('M,N_,K,members', [(128, 64, 64, 1), (128, 64, 576, 1), (256, 192, 512, 3), (256, 192, 640, 3),
                                            (2560, 1024, 64, 1), (640, 1024, 192, 4)])
@pytest.mark.parametrize('epi', ['f32', 'fwd', 'bwd'])
def test_gemm_launch_shapes(M, N_, K, members, epi):
    """The narrow, the deep and the wide tiles: few and many of them, short and long K, each epilogue."""
    torch = _torch()
    rng = np.random.default_rng(M + K)
    A = MO.bf16(rng.normal(size=(members, M, K)).astype(np.float32))
    B = MO.bf16((rng.normal(size=(members, N_, K)) / np.sqrt(K)).astype(np.float32))
    pre = rng.normal(size=(members, M, N_)).astype(np.float32)
    bias = rng.normal(size=(members, N_)).astype(np.float32)
    a, b, pt, bt = _bf16(A), _bf16(B), torch.from_numpy(pre).cuda(), torch.from_numpy(bias).cuda()
    f32 = torch.full((members, M, N_), 7.0, device='cuda')
    bf = torch.zeros((members, M, N_), dtype=torch.int16, device='cuda')
    t = torch.zeros((members, N_, M), dtype=torch.int16, device='cuda')
    status = torch.zeros(1, dtype=torch.int32, device='cuda')
    g = N.DmMlpGemm()
    g.epi = {'f32': N.DM_MLP_EPI_F32, 'fwd': N.DM_MLP_EPI_GELU_FWD, 'bwd': N.DM_MLP_EPI_GELU_BWD}[epi]
    g.M, g.N, g.K, g.members = M, N_, K, members
    g.A, g.lda, g.a_ms, g.B, g.ldb, g.b_ms = a.data_ptr(), K, M * K, b.data_ptr(), K, N_ * K
    if epi != 'bwd':
        g.out_f32, g.ld_f32, g.f32_ms = f32.data_ptr(), N_, M * N_
    if epi != 'f32':
        g.bias, g.bias_ms = bt.data_ptr(), N_
        g.pre, g.ld_pre, g.pre_ms = pt.data_ptr(), N_, M * N_
        g.out_bf16, g.ld_bf16, g.bf16_ms = bf.data_ptr(), N_, M * N_
        g.out_t, g.ld_t, g.t_ms = t.data_ptr(), M, M * N_
    N.call('dm_mlp_gemm_run', ctypes.byref(g), ctypes.c_void_p(status.data_ptr()), None)
    assert int(status.item()) == 0
    A64, Bt = A.astype(np.float64), np.swapaxes(B.astype(np.float64), 1, 2)
    want = A64 @ Bt
    tol = (K + 2) * U * (np.abs(A64) @ np.abs(Bt) + 4)
    if epi == 'fwd':
        want = want + bias[:, None, :]
    if epi != 'bwd':
        assert np.all(np.abs(f32.cpu().numpy() - want) <= tol)
    if epi != 'f32':
        # GELU (slope below 1.13) and its derivative (below 1.13) in FP32, rounded to BF16
        x = want if epi == 'fwd' else pre.astype(np.float64)
        c, k = 0.7978845608028654, 0.044715
        y = c * (x + k * x ** 3)
        gate = 0.5 * (1 + np.tanh(y))
        d = gate + 0.5 * x * (1 - np.tanh(y) ** 2) * c * (1 + 3 * k * x * x)
        want = x * gate if epi == 'fwd' else want * d
        err = np.abs(_f(bf) - want)
        assert np.all(err <= 2.0 ** -8 * np.abs(want) + 1.13 * tol + 64 * U)
        assert np.array_equal(bf.cpu().numpy(), np.swapaxes(t.cpu().numpy(), 1, 2))


@pytest.mark.parametrize('rows', [1, 31, 32, 33, 100])
@pytest.mark.parametrize('nfeat,width', [(6, 64), (64, 64), (7, 8), (33, 40)])
def test_gather(rows, nfeat, width):
    """Blocks of 32 rows, ragged ends, widths that are no multiple of 32; indexes outside the data set read sample 0."""
    torch = _torch()
    members, nout, samples = 3, 12, 50
    rng = np.random.default_rng(rows + nfeat)
    f = rng.normal(size=(samples, nfeat)).astype(np.float32)
    t = rng.normal(size=(samples, nout)).astype(np.float32)
    idx = rng.integers(0, samples, (members, rows)).astype(np.int32)
    idx[0, 0], idx[1, rows - 1] = -1, samples
    used = np.where((idx < 0) | (idx >= samples), 0, idx)
    x = torch.full((members, rows, width), 7, dtype=torch.int16, device='cuda')
    xt = torch.full((members, width, rows), 7, dtype=torch.int16, device='cuda')
    td = torch.zeros((members, rows, nout), device='cuda')
    fd, tg, ix = (torch.from_numpy(a).cuda() for a in (f, t, idx))
    vp = ctypes.c_void_p
    N.call('dm_mlp_gather', vp(fd.data_ptr()), nfeat, vp(tg.data_ptr()), nout, ctypes.c_int64(samples), vp(ix.data_ptr()),
           rows, members, width, vp(x.data_ptr()), vp(xt.data_ptr()), vp(td.data_ptr()), None)
    want = np.zeros((members, rows, width), np.float32)
    want[:, :, :nfeat] = MO.bf16(f)[used]
    assert np.array_equal(_f(x), want)
    assert np.array_equal(_f(xt), np.swapaxes(want, 1, 2))
    assert np.array_equal(td.cpu().numpy(), t[used])


def test_train_step_equals_its_parts():
    """The step reads its targets from the data set; gathering them first gives the same parameters."""
    torch = _torch()
    g = torch.Generator('cuda').manual_seed(8)
    f = torch.rand(300, 6, device='cuda', generator=g) * 2 - 1
    t = torch.softmax(torch.randn(300, 256, device='cuda', generator=g), dim=1)
    index = torch.randint(-2, 303, (2, 128), device='cuda', generator=g, dtype=torch.int32)
    a, b = (S.MLPEnsemble(members=2, batch=128, nout=256, seed=3) for _ in range(2))
    a.train_step(f, t, index, 1e-3)
    b.gather(f, t, index, 128)
    b.loss_and_grads(128)
    b._adam(1, 1e-3)
    assert torch.equal(a.params, b.params) and torch.equal(a.loss_rows, b.loss_rows) and torch.equal(a.grads, b.grads)


@pytest.mark.parametrize('members', [1, 3])
def test_prediction_of_no_points(members):
    """An empty set, whose tensors have no address, has an empty result; more points without one are refused."""
    torch = _torch()
    ens = S.MLPEnsemble(members=members, batch=128, nout=256)
    got = ens.predict(torch.empty((0, 6), device='cuda'))
    assert got.shape == (members, 0, 256) and got.dtype == torch.float32 and got.is_cuda
    assert N.lib().dm_mlp_predict(ens._net(), None, 6, ctypes.c_int64(1), None, None) == N.DM_ERR_ARG


def test_predictions_where_no_workspace_fits():
    """With room for the result alone, the passes run in a batch's buffers."""
    torch = _torch()
    ens = S.MLPEnsemble(members=2, batch=128, nout=1024, seed=5)
    f = torch.rand(4000, 6, device='cuda', generator=torch.Generator('cuda').manual_seed(1)) * 2 - 1
    want = ens.predict(f).cpu()
    assert ens._predict_rows(4000) == 4096          # its workspace: 47 MB beside 33 MB of results
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (48 << 20)) / total)
        got = ens.predict(f)
        with pytest.raises(torch.OutOfMemoryError):   # a result that does not fit is refused as ever
            ens.predict(torch.rand(20000, 6, device='cuda'))
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize('shift', [0, 1])
@pytest.mark.parametrize('shapes', [[(5, 7), (33, 64), (64, 33), (300, 32), (1, 1)],
                                    [(8, 4), (36, 64), (64, 36), (300, 32)]])
def test_adam_steps_follow_the_rule(shapes, shift):
    """Three steps in a row, a new gradient each, from moments that are not zero, against the rule in FP64;
    with the state off 16-byte alignment (element by element) as well."""
    torch = _torch()
    P = sum(o * i + o for o, i in shapes)
    Z = 2
    rng = np.random.default_rng(3)

    def place(a):
        t = torch.zeros(a.size + 8, dtype=torch.float32, device='cuda')[shift:shift + a.size]
        t.copy_(torch.from_numpy(a.reshape(-1)))
        return t

    lr, b1, b2, eps = (float(np.float32(x)) for x in (1e-2, 0.9, 0.999, 1e-8))
    p = rng.normal(size=(Z, P)).astype(np.float32)
    m = (0.3 * rng.normal(size=(Z, P))).astype(np.float32)
    v = rng.uniform(0.01, 0.1, size=(Z, P)).astype(np.float32)
    dp, dm, dv = place(p), place(m), place(v)
    grads = [rng.normal(size=(Z, P)).astype(np.float32) for _ in range(3)]
    dg = [place(g) for g in grads]
    wb, wtb = (torch.zeros((Z, P), dtype=torch.int16, device='cuda') for _ in range(2))
    flat = (ctypes.c_int32 * (2 * len(shapes)))(*[x for s in shapes for x in s])
    vp = ctypes.c_void_p
    for step in (1, 2, 3):
        N.call('dm_mlp_adam', vp(dp.data_ptr()), vp(dg[step - 1].data_ptr()), vp(dm.data_ptr()), vp(dv.data_ptr()),
               ctypes.c_int64(P), Z, flat, len(shapes), ctypes.c_float(lr), ctypes.c_float(b1), ctypes.c_float(b2),
               ctypes.c_float(eps), step, vp(wb.data_ptr()), vp(wtb.data_ptr()), None)
    # FP64, with a running bound of the FP32 roundings: three per moment, eight in the update, one on p
    p, m, v = (a.astype(np.float64) for a in (p, m, v))
    em, ev, ep = np.zeros_like(m), np.zeros_like(v), np.zeros_like(p)
    for step, g in enumerate(grads, 1):
        g = g.astype(np.float64)
        em = b1 * em + 4 * U * (b1 * np.abs(m) + (1 - b1) * np.abs(g))
        ev = b2 * ev + 4 * U * (b2 * v + (1 - b2) * g * g)
        # 1 - beta in FP32 is exact to U of 1
        em, ev = em + U * np.abs(g), ev + U * g * g
        m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
        mh, vh = m / (1 - b1 ** step), np.sqrt(v / (1 - b2 ** step)) + eps
        ep = ep + lr / vh * (em / (1 - b1 ** step) + np.abs(mh) * (0.5 * ev / v + 8 * U)) + U * (np.abs(p) + 1)
        p = p - lr * mh / vh
    for got, want, bound in ((dp, p, ep), (dm, m, em), (dv, v, ev)):
        assert np.all(np.abs(got.cpu().numpy().reshape(Z, P) - want) <= 1.01 * bound)
    off = 0
    bits = (MO.bf16(dp.cpu().numpy().reshape(Z, P)).view(np.uint32) >> 16).astype(np.uint16).view(np.int16)
    for o, i in shapes:
        w = bits[:, off:off + o * i]
        assert np.array_equal(wb[:, off:off + o * i].cpu().numpy(), w)
        assert np.array_equal(wtb[:, off:off + o * i].cpu().numpy().reshape(Z, i, o),
                              np.swapaxes(w.reshape(Z, o, i), 1, 2))
        off += o * i + o
