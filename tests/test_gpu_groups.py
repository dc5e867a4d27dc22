"""Batched tensor-core sweeps on groups of CTAs: the result of an instance does not depend on how many
CTAs run it.  Each batch is compared bit for bit with every instance in a batch of its own (which the
library runs on its largest groups), and with the FP64 batch on the CUDA cores."""
import numpy as np
import pytest

from qiskit_aakash_gb300 import batch as B
from qiskit_aakash_gb300 import surrogate as S
from qiskit_aakash_gb300 import template as TP
from qiskit_aakash_gb300.circuit import random_layer_circuit

pytestmark = pytest.mark.gpu
KMAX = {n: B.TC for n in range(7, 13)}


def _spec(n, depth, seed):
    return {'n': n, 'depth': depth, 'seed': seed, 'depolarisation': 2e-3, 'decoherence': 0.993, 'decay': 0.996}


def _run(specs, precision='single'):
    t = B.compile_sweep(specs, [precision], workers=1, kmax={precision: KMAX if precision == 'single' else {}})
    prog = B.BatchProgram(t[precision])
    prog.launch()
    return prog.results()


@pytest.mark.parametrize('specs', [
    [_spec(7, 3, 1)],                                              # one tile, most of its group idle
    [_spec(8, 4, 2), _spec(7, 2, 3), _spec(9, 3, 4)],              # fewer tiles than group members
    [_spec(11, 4, 5), _spec(10, 5, 6), _spec(9, 1, 7), _spec(8, 3, 8), _spec(7, 6, 9)],
    # one large instance above the even share: groups for it, one CTA each for the others
    [_spec(11, 40, 10)] + [_spec(9, 2, 11 + i) for i in range(310)],
    # fewer than half as many as CTAs, none of them large: groups of two
    [_spec(9, 3, 400 + i) for i in range(120)],
], ids=['one', 'small', 'mixed', 'uneven', 'half'])
def test_batch_does_not_depend_on_grouping(specs):
    got = _run(specs)
    pick = range(len(specs)) if len(specs) < 10 else (0, 1, len(specs) // 2, len(specs) - 1)
    for i in pick:
        assert np.array_equal(got[i], _run([specs[i]])[0]), i
    sub = [specs[i] for i in pick]
    for g, w in zip((got[i] for i in pick), _run(sub, 'double')):
        assert np.abs(g - w).max() < 2e-6


@pytest.mark.parametrize('points', [1, 3, 100, 305, 460])
def test_template_does_not_depend_on_grouping(points):
    """Below one wave of CTAs, one wave and one point more, one wave and half of the next."""
    qc = random_layer_circuit(9, 3, seed=2)
    raw = S.sample_noise(points, seed=points)
    prog = TP.TemplateProgram(qc.to_experiment(), S.options_of(raw[0]), 'single')
    assert prog.tc
    runner = TP.TemplateRunner(prog)
    got = runner.run(S.param_vectors(raw)).cpu().numpy()
    for i in sorted({0, points // 2, points - 1}):
        assert np.array_equal(got[i:i + 1], runner.run(S.param_vectors(raw[i:i + 1])).cpu().numpy()), i


def test_template_of_many_slots():
    """More recipe slots than are composed at a time."""
    qc = random_layer_circuit(9, 60, seed=3)
    raw = S.sample_noise(2, seed=1)
    tc = TP.TemplateProgram(qc.to_experiment(), S.options_of(raw[0]), 'single')
    cc = TP.TemplateProgram(qc.to_experiment(), S.options_of(raw[0]), 'single', tensor_cores=False)
    assert tc.tc and tc.nslots > 600
    got = TP.TemplateRunner(tc).run(S.param_vectors(raw)).cpu().numpy()
    ref = TP.TemplateRunner(cc).run(S.param_vectors(raw)).cpu().numpy()
    assert np.abs(got - ref).max() < 4e-6


@pytest.mark.parametrize('count', [1, 20, 310])
def test_passes_of_many_rounds(count):
    """Passes of 20 rounds (7 qubits, 30 layers): more than one CTA composes at a time, alone and in groups."""
    specs = [_spec(7, 30, 700 + i) for i in range(count)]
    got = _run(specs)
    pick = sorted({0, count // 2, count - 1})
    for i in pick:
        assert np.array_equal(got[i], _run([specs[i]])[0]), i
    for g, w in zip((got[i] for i in pick), _run([specs[i] for i in pick], 'double')):
        assert np.abs(g - w).max() < 2e-6
