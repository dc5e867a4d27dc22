"""Launches that set up while the kernel before them runs: what they read must be complete all the same.

Back to back, without a synchronisation, and replayed from a CUDA graph, the results are those of the
same calls with a synchronisation after each."""
import numpy as np
import pytest

from qiskit_aakash_gb300 import engine
from qiskit_aakash_gb300 import program as P
from qiskit_aakash_gb300 import surrogate as S

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    return torch


def _record(n, layers, seed):
    """A recorded FP32 circuit: CX over short and long distances, so that TMA-fed and cp.async-fed passes occur."""
    rng = np.random.default_rng(seed)
    dev = engine.DeviceState(n, precision='single')
    dev.record()
    dev.init_product([[1.0, 0.0, 0.0, 1.0]] * n, 2.0 ** -n)
    noise = P.noise_ptm(0.999, 0.99, 0.998)
    err = {'rx': [1, 0], 'ry': [1, 0], 'rz': [1, 0]}
    for _ in range(layers):
        for q in range(n):
            dev.map1(q, P.u_gate_ptm('u3', rng.uniform(0, 6, 3), err))
            dev.map1(q, noise)
        order = rng.permutation(n)
        for a, b in zip(order[::2], order[1::2]):
            dev.cx(int(a), int(b), [0.995, 0.01])
    dev.flush()
    return dev


@pytest.mark.parametrize('n', [7, 8, 10, 11, 12])      # 1 to 1,024 tiles: below, around and above the SMs
def test_circuits_back_to_back(n):
    torch = _torch()
    dev = _record(n, 8, n)
    dev.replay(on_call=lambda name, before: None if before else torch.cuda.synchronize())
    want = dev.state.clone()
    for _ in range(20):
        dev.state.fill_(float('nan'))          # a kernel that knows nothing of early starts, before the first call
        dev.replay()
        got = dev.state.clone()                # and one right after the last
        assert torch.equal(got, want)
    assert int(dev.status.item()) == 0


def test_circuit_in_a_graph():
    torch = _torch()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        dev = _record(10, 8, 3)
        want = dev.state.clone()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        dev.replay()
    for _ in range(5):
        dev.state.fill_(float('nan'))
        graph.replay()
        assert torch.equal(dev.state, want)
    assert int(dev.status.item()) == 0


def _train(sync, steps=12):
    torch = _torch()
    g = torch.Generator('cuda').manual_seed(4)
    f = torch.rand(700, 6, device='cuda', generator=g) * 2 - 1
    t = torch.softmax(torch.randn(700, 256, device='cuda', generator=g), dim=1)
    ens = S.MLPEnsemble(members=3, batch=256, nout=256, seed=5)
    for i in range(steps):
        index = torch.randint(700, (3, 256), device='cuda', generator=g, dtype=torch.int32)
        ens.train_step(f, t, index, 1e-3)
        if sync:
            torch.cuda.synchronize()
    return ens, ens.params.clone(), ens.predict(f)


def test_training_back_to_back():
    torch = _torch()
    _, params, probs = _train(True)
    for _ in range(3):
        ens, p, q = _train(False)
        assert torch.equal(p, params) and torch.equal(q, probs)
        assert int(ens.status.item()) == 0


@pytest.mark.parametrize('n', [4, 6, 8, 9])
def test_small_fp64_states_take_smaller_tiles(n):
    """The default tile of a small FP64 state against six resident axes: the same maps, grouped otherwise.

    4**n values of at most 2**-n; 12 layers of maps that do not grow them, 3 n roundings of each value
    per layer at 16 terms: 12 * 3 * n * 16 * 2**-53 * 2**-n, doubled for the other grouping."""
    torch = _torch()
    rng = np.random.default_rng(n)
    angles = rng.uniform(0, 6, (12, n, 3))
    pairs = [rng.permutation(n) for _ in range(12)]
    err = {'rx': [1, 0], 'ry': [1, 0], 'rz': [1, 0]}
    states = []
    for axes in (None, 6):
        dev = engine.DeviceState(n, precision='double', tile_axes=axes)
        dev.init_product([[1.0, 0.0, 0.0, 1.0]] * n, 2.0 ** -n)
        for layer, order in zip(angles, pairs):
            for q in range(n):
                dev.map1(q, P.u_gate_ptm('u3', layer[q], err))
                dev.map1(q, P.noise_ptm(0.999, 0.99, 0.998))
            for a, b in zip(order[::2], order[1::2]):
                dev.cx(int(a), int(b), [0.995, 0.01])
        dev.flush()
        states.append(dev.state.clone())
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert engine.DeviceState(n, precision='double').kmax == (5 if 4 ** (n - 5) <= sms else 6)
    assert float((states[0] - states[1]).abs().max()) <= 2 * 12 * 3 * n * 16 * 2.0 ** -53 * 2.0 ** -n
