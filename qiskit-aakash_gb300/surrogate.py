"""Learned noise surrogate: an MLP ensemble from noise parameters to a template's outcome distribution.

The reference has no learned part; this is the engine's own extension.  A
fixed circuit template (by default 10 qubits, 30 random brick layers, Z
ensemble measurement) is simulated for many noise-parameter points by the
template sweep (``template.TemplateRunner``); an ensemble of small MLPs
(6 -> 256 -> 256 -> 256 -> 1024, GELU, softmax) learns the map from the six
noise parameters to the 1024 outcome probabilities.  At inference the
ensemble's spread (mean total-variation distance of the members to their
mean) decides where the surrogate is trusted: points above the threshold
fall back to the plain simulation.

Every step runs in libdmgb300.so: BF16 tensor-core GEMMs with fused
bias / GELU / GELU' epilogues (FP32 master weights), softmax with the KL
loss, bias gradients, Adam, the minibatch gather and the ensemble
statistics.  torch tensors are only device buffers.

Noise dimensions (the six inputs, and how each maps to backend options):
    depolarisation p   log-uniform [1e-4, 1e-2]  -> depolarization_factor = 1 - p (at measurement)
    decoherence 1 - f  log-uniform [1e-4, 1e-2]  -> decoherence_factor = f
    decay 1 - g        log-uniform [1e-4, 1e-2]  -> decay_factor = g
    thermal p_th       uniform [0.8, 1.0]        -> thermal_factor
    rotation sigma     uniform [0, 0.05]         -> rotation_error <cos> = exp(-sigma**2 / 2), mean 0
    CX error 1 - c     log-uniform [1e-4, 1e-2]  -> tsp_model_error = [c, 0]
"""
import ctypes
import math
import time

import numpy as np

from . import _native as N
from . import template as TP
from .circuit import noise_options, random_layer_circuit
from .exceptions import BasicAerError

NOISE_DIMS = ('depolarisation', 'decoherence_loss', 'decay_loss', 'thermal', 'rotation_sigma', 'cx_loss')
LOG_DIMS = (0, 1, 2, 5)
LOG_RANGE = (1e-4, 1e-2)
LIN_RANGES = {3: (0.8, 1.0), 4: (0.0, 0.05)}
WIDTHS = (64, 256, 256, 256, 1024)
N_FEATURES = 6

# Bytes of activations of one pass of a prediction: a pass of 1,024 points leaves the chip half empty in
# every launch (10,233 points, 1,024 outcomes, 5 members: 440 us in passes of 1,024, 353 us in 64 MB, 312 us
# in 96-256 MB, 285 us in one).
PREDICT_WORKSPACE = 512 << 20


def sample_noise(count, seed):
    """Seeded noise points [count, 6] in the physical units of NOISE_DIMS."""
    rng = np.random.default_rng(seed)
    raw = np.empty((count, N_FEATURES))
    lo, hi = np.log(LOG_RANGE[0]), np.log(LOG_RANGE[1])
    for d in LOG_DIMS:
        raw[:, d] = np.exp(rng.uniform(lo, hi, count))
    for d, (a, b) in LIN_RANGES.items():
        raw[:, d] = rng.uniform(a, b, count)
    return raw


def features(raw):
    """Network inputs in [-1, 1]: log10 of the log-uniform dimensions, the others linearly."""
    raw = np.asarray(raw, dtype=np.float64)
    x = np.empty_like(raw)
    llo, lhi = np.log10(LOG_RANGE[0]), np.log10(LOG_RANGE[1])
    for d in LOG_DIMS:
        x[:, d] = 2 * (np.log10(raw[:, d]) - llo) / (lhi - llo) - 1
    for d, (a, b) in LIN_RANGES.items():
        x[:, d] = 2 * (raw[:, d] - a) / (b - a) - 1
    return x.astype(np.float32)


def options_of(row):
    """Backend options of one noise point."""
    return noise_options(depolarisation=row[0], decoherence=1 - row[1], decay=1 - row[2], thermal=row[3],
                         rotation_sigma=row[4], tsp=[1 - row[5], 0.0])


def param_vectors(raw):
    """Template-sweep parameter vectors [count, PARAM_STRIDE] of noise points (the options_of mapping)."""
    raw = np.asarray(raw, dtype=np.float64)
    v = np.zeros((raw.shape[0], TP.PARAM_STRIDE))
    v[:, 0] = 1 - raw[:, 1]
    v[:, 1] = raw[:, 3]
    v[:, 2] = 1 - raw[:, 2]
    c = np.exp(-0.5 * raw[:, 4] ** 2)
    v[:, 3] = v[:, 5] = v[:, 7] = c
    v[:, 9] = 1 - raw[:, 5]
    v[:, 11] = 1 - raw[:, 0]
    return v


class Template:
    """The fixed circuit of the surrogate and its template sweep on the device."""

    def __init__(self, n=10, layers=30, seed=0, precision='single', device=None):
        self.n, self.layers, self.seed = n, layers, seed
        self.circuit = random_layer_circuit(n, layers, seed)
        centre = sample_noise(1, 12345)[0]
        self.program = TP.TemplateProgram(self.circuit.to_experiment(), options_of(centre), precision)
        self.runner = TP.TemplateRunner(self.program, device)

    def simulate(self, raw):
        """Outcome distributions [count, 2**n] (FP64, device) of noise points, by the plain simulation."""
        return self.runner.run(param_vectors(raw))


def _layer_offsets(widths):
    offs, o = [], 0
    for li in range(4):
        out, inp = widths[li + 1], widths[li]
        offs.append((o, o + out * inp, out, inp))
        o += out * inp + out
    return offs, o


class MLPEnsemble:
    """``members`` networks trained together; every buffer is [members, ...] on the device."""

    def __init__(self, members=5, batch=1024, seed=0, nout=1024, device=None):
        import torch
        if not torch.cuda.is_available():
            raise BasicAerError('the surrogate needs a CUDA device')
        N.lib()
        if batch % 128:
            raise BasicAerError('the batch size must be a multiple of 128')
        if nout % 256 or not 256 <= nout <= 4096:
            raise BasicAerError('the output width must be a multiple of 256 up to 4096')
        self.M, self.B, self.nout = members, batch, nout
        self.widths = WIDTHS[:4] + (nout,)
        self.device = torch.device(device or 'cuda')
        self.layers, self.P = _layer_offsets(self.widths)
        self.shapes = (ctypes.c_int32 * 8)(*[v for (_, _, out, inp) in self.layers for v in (out, inp)])
        dev, f32, bf = self.device, torch.float32, torch.int16
        M, B, P = members, batch, self.P
        z = lambda *s, dt=f32: torch.zeros(*s, dtype=dt, device=dev)  # noqa: E731
        self.params, self.grads, self.m, self.v = z(M, P), z(M, P), z(M, P), z(M, P)
        self.wb, self.wtb = z(M, P, dt=bf), z(M, P, dt=bf)
        self.status = z(1, dt=torch.int32)
        self.step_count = 0
        self._alloc(B)
        self.init_params(seed)

    def _alloc(self, B):
        import torch
        dev, f32, bf = self.device, torch.float32, torch.int16
        M = self.M
        z = lambda *s, dt=f32: torch.empty(*s, dtype=dt, device=dev)  # noqa: E731
        self.bufB = B
        self.x, self.xt = z(M, B, 64, dt=bf), z(M, 64, B, dt=bf)
        self.pre = [z(M, B, 256) for _ in range(3)]
        self.h = [z(M, B, 256, dt=bf) for _ in range(3)]
        self.ht = [z(M, 256, B, dt=bf) for _ in range(3)]
        K = self.nout
        self.logits, self.t = z(M, B, K), z(M, B, K)
        self.dz, self.dzt = z(M, B, K, dt=bf), z(M, K, B, dt=bf)
        self.du = [z(M, B, 256, dt=bf) for _ in range(3)]
        self.dut = [z(M, 256, B, dt=bf) for _ in range(3)]
        self.loss_rows = z(M, B)
        self.probs = z(M, B, K)

    # -- parameters ------------------------------------------------------------
    def init_params(self, seed):
        """He-style normal initialisation (std sqrt(2 / fan_in); sqrt(1 / fan_in) for the output layer)."""
        import torch
        host = np.zeros((self.M, self.P), dtype=np.float32)
        for z in range(self.M):
            rng = np.random.default_rng([seed, z])
            for li, (w0, b0, out, inp) in enumerate(self.layers):
                real_in = N_FEATURES if li == 0 else inp
                std = math.sqrt((2.0 if li < 3 else 1.0) / real_in)
                w = np.zeros((out, inp), dtype=np.float32)
                w[:, :real_in] = rng.normal(0.0, std, size=(out, real_in))
                host[z, w0:w0 + out * inp] = w.reshape(-1)
        self.set_params(torch.from_numpy(host))

    def set_params(self, flat):
        """Load [members, P] FP32 parameters (W1 b1 ... W4 b4 per member); resets Adam."""
        import torch
        self.params.copy_(torch.as_tensor(flat, dtype=torch.float32))
        self.m.zero_()
        self.v.zero_()
        self.step_count = 0
        self._adam(0, 0.0)

    def unpack(self, flat):
        """[W1, b1, ..., W4, b4] numpy arrays of one member's flat parameter vector."""
        out = []
        for (w0, b0, o, i) in self.layers:
            out += [flat[w0:w0 + o * i].reshape(o, i), flat[b0:b0 + o]]
        return out

    # -- kernels -----------------------------------------------------------------
    def _stream(self):
        import torch
        return ctypes.c_void_p(torch.cuda.current_stream(self.device).cuda_stream)

    def _net(self):
        """The network's description for the library, from the buffers as they are now."""
        net = N.DmMlpNet()
        net.members, net.batch, net.nout, net.count = self.M, self.bufB, self.nout, self.P
        for f in ('params', 'grads', 'm', 'v', 'wb', 'wtb', 'x', 'xt', 'logits', 't', 'dz', 'dzt', 'loss_rows',
                  'probs', 'status'):
            setattr(net, f, getattr(self, f).data_ptr())
        for f in ('pre', 'h', 'ht', 'du', 'dut'):
            setattr(net, f, (ctypes.c_void_p * 3)(*[b.data_ptr() for b in getattr(self, f)]))
        return ctypes.byref(net)

    def _adam(self, step, lr, beta1=0.9, beta2=0.999, eps=1e-8):
        vp = ctypes.c_void_p
        N.call('dm_mlp_adam', vp(self.params.data_ptr()), vp(self.grads.data_ptr()), vp(self.m.data_ptr()),
               vp(self.v.data_ptr()), ctypes.c_int64(self.P), self.M, self.shapes, 4, ctypes.c_float(lr),
               ctypes.c_float(beta1), ctypes.c_float(beta2), ctypes.c_float(eps), step, vp(self.wb.data_ptr()),
               vp(self.wtb.data_ptr()), self._stream())

    def forward(self, rows, train):
        """Forward pass of the members on self.x (rows <= batch); logits in self.logits."""
        N.call('dm_mlp_forward', self._net(), rows, int(bool(train)), self._stream())

    def backward(self, rows):
        """Gradients of the mean KL loss (self.dz / self.dzt already hold dL/dz) into self.grads."""
        N.call('dm_mlp_backward', self._net(), rows, self._stream())

    def gather(self, feats, targets, index, rows):
        vp = ctypes.c_void_p
        N.call('dm_mlp_gather', vp(feats.data_ptr()), N_FEATURES, vp(targets.data_ptr()), self.nout,
               ctypes.c_int64(feats.shape[0]), vp(index.data_ptr()), rows, self.M, 64, vp(self.x.data_ptr()),
               vp(self.xt.data_ptr()), vp(self.t.data_ptr()), self._stream())

    def loss_and_grads(self, rows):
        """Forward + softmax/KL + backward on the gathered minibatch (self.x, self.t)."""
        N.call('dm_mlp_loss_and_grads', self._net(), rows, self._stream())

    def train_step(self, feats, targets, index, lr):
        vp = ctypes.c_void_p
        step = self.step_count + 1
        N.call('dm_mlp_train_step', self._net(), vp(feats.data_ptr()), N_FEATURES, vp(targets.data_ptr()),
               ctypes.c_int64(feats.shape[0]), vp(index.data_ptr()), ctypes.c_float(lr), ctypes.c_float(0.9),
               ctypes.c_float(0.999), ctypes.c_float(1e-8), step, self._stream())
        self.step_count = step

    def fit(self, feats, targets, epochs, lr=2e-3, lr_min=2e-5, seed=0, log_every=0):
        """Train every member on (feats [S, 6], targets [S, 1024]) device tensors; own shuffles per member."""
        import torch
        S = feats.shape[0]
        steps_per_epoch = S // self.B
        if steps_per_epoch < 1:
            raise BasicAerError('fewer samples than one batch')
        total = epochs * steps_per_epoch
        rng = np.random.default_rng(seed)
        history = []
        t0 = time.perf_counter()
        for ep in range(epochs):
            perm = np.stack([rng.permutation(S)[:steps_per_epoch * self.B] for _ in range(self.M)]).astype(np.int32)
            perm_d = torch.from_numpy(perm).to(self.device)
            for s in range(steps_per_epoch):
                k = ep * steps_per_epoch + s
                lr_k = lr_min + 0.5 * (lr - lr_min) * (1 + math.cos(math.pi * k / total))
                idx = perm_d[:, s * self.B:(s + 1) * self.B].contiguous()
                self.train_step(feats, targets, idx, lr_k)
                if log_every and k % log_every == 0:
                    history.append((k, float(self.loss_rows.mean())))
        torch.cuda.synchronize(self.device)
        if int(self.status.item()) != 0:
            raise BasicAerError('a tensor-core GEMM abandoned a bounded wait')
        return {'steps': total, 'seconds': time.perf_counter() - t0, 'history': history}

    def predict(self, feats):
        """Member distributions [members, S, 1024] (FP32, device) of feature rows [S, 6] (device)."""
        import torch
        S = feats.shape[0]
        out = torch.empty((self.M, S, self.nout), dtype=torch.float32, device=self.device)
        net, work = self._net(), self._predict_work(S)
        if work:
            n = net._obj
            n.batch = work[0].shape[1]
            n.x, n.logits = work[0].data_ptr(), work[4].data_ptr()
            n.h = (ctypes.c_void_p * 3)(*[b.data_ptr() for b in work[1:4]])
        vp = ctypes.c_void_p
        N.call('dm_mlp_predict', net, vp(feats.data_ptr()), N_FEATURES, ctypes.c_int64(S), vp(out.data_ptr()),
               self._stream())
        return out

    def _predict_work(self, S):
        """Activations of a prediction's passes (x, three layers, logits) where they are larger than a batch's;
        None where a batch's buffers do, also when the device has no room for more."""
        import torch
        rows = self._predict_rows(S)
        if rows <= self.bufB:
            return None
        try:
            return [torch.empty((m, rows, w), dtype=t, device=self.device)
                    for m, w, t in ((1, 64, torch.int16), (self.M, 256, torch.int16), (self.M, 256, torch.int16),
                                    (self.M, 256, torch.int16), (self.M, self.nout, torch.float32))]
        except torch.OutOfMemoryError:
            return None

    def _predict_rows(self, S):
        """Points per pass through the network: the batch, or as many as PREDICT_WORKSPACE holds activations of,
        in equal passes of whole tiles."""
        per = self.M * (2 * (64 + 3 * 256) + 4 * self.nout)
        cap = max(self.bufB, PREDICT_WORKSPACE // per // 128 * 128)
        passes = max(1, -(-S // cap))
        return -(-S // (passes * 128)) * 128

    def ensemble(self, member_probs, ref=None):
        """(mean [S, 1024], spread [S], TV(mean, ref) [S] or None), all on the device."""
        import torch
        M, S, K = member_probs.shape
        mean = torch.empty((S, K), dtype=torch.float32, device=self.device)
        spread = torch.empty(S, dtype=torch.float32, device=self.device)
        tv = torch.empty(S, dtype=torch.float32, device=self.device) if ref is not None else None
        vp = ctypes.c_void_p
        N.call('dm_mlp_ensemble', vp(member_probs.data_ptr()), S, M, K, vp(ref.data_ptr()) if ref is not None else None,
               vp(mean.data_ptr()), vp(spread.data_ptr()), vp(tv.data_ptr()) if tv is not None else None,
               self._stream())
        return mean, spread, tv
