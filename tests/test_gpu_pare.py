"""Pared graphs where paring decides the value (csrc/mpx_adjoint.cuh: k_pare_*, k_frozen_*).

A threshold below every weight leaves <O> as it is; these thresholds do not, so that a replay that ignores the keep
set gives another number. The expected values follow from the definition (PareGraph.cpp:103-141): a term past its
last relevant step is neither scaled nor rotated. Products of at most 40 cosines: 1e-12.
"""

import numpy as np
import pytest
from test_gpu_window import circuit

from monoprop_b200 import _native
from monoprop_b200 import workloads as W

pytestmark = pytest.mark.gpu


def pare(eng, circ, threshold):
    eng._check(_native.load().mpx_graph_pare(eng.h, circ.h, float(threshold)))


def graph(wl):
    eng = _native.engine_for(wl)
    circ = eng.upload(wl.gen_words(), wl.angles())
    eng.graph_build(circ)
    return eng, circ


@pytest.mark.parametrize("basis, modes", [("pauli", 30), ("majorana", 130)])
def test_threshold_above_every_weight_keeps_the_initial_operator(basis, modes):
    wl = circuit(basis, modes, 100, modes, 1e-3, None)
    mode = int(wl.gate_slots[0][0]) // 2
    wl.observable[(2 * mode, 2 * mode + 1)] = 0.75 + 0j if basis == "pauli" else 0.75j
    eng, circ = graph(wl)
    plain = eng.graph_expectation(circ)
    pare(eng, circ, 2.0)
    values = [eng.graph_expectation(circ), eng.graph_gradient(circ)[0], eng.graph_gradient(circ, segment_gates=40)[0]]
    pare(eng, circ, -1.0)
    again = eng.graph_expectation(circ)
    eng.reset()
    initial = eng.expectation()
    circ.close()
    eng.close()
    assert abs(again - plain) <= 1e-12 and abs(plain - initial) > 1e-3
    assert all(abs(v - initial) <= 1e-12 for v in values)


def test_schrodinger_threshold_between_two_observable_terms():
    """Small angles under a large lower_atol: no gate pairs anything, every Z string takes one cos per X rotation
    on its qubits. The observable term below the threshold keeps its starting score, the other one its factors."""
    n, layers, angle = 9, 10, 0.02
    slots = [(2 * q,) for _ in range(layers) for q in range(n)]
    wl = W.Workload("pare", "pauli", n, slots, np.ones(len(slots)), np.zeros(len(slots), int), np.array([angle]),
                    {(0, 1): 0.9 + 0j, (2, 3, 4, 5): 0.2 + 0j}, [], n, "support", 0.5)
    wl.extra["schrodinger_cutoff"] = 4
    eng, circ = graph(wl)
    c = np.cos(2 * angle) ** layers
    plain = eng.graph_expectation(circ)
    pare(eng, circ, 0.5)
    values = [eng.graph_expectation(circ), eng.graph_gradient(circ)[0], eng.graph_gradient(circ, segment_gates=31)[0]]
    circ.close()
    eng.close()
    assert abs(plain - (0.9 * c + 0.2 * c * c)) <= 1e-12
    assert all(abs(v - (0.9 * c + 0.2)) <= 1e-12 for v in values)


@pytest.mark.parametrize("threshold", [0.5, 2.0])
@pytest.mark.parametrize("basis, modes", [("pauli", 30), ("majorana", 130)])
def test_pared_gradient_does_not_depend_on_the_segments(basis, modes, threshold):
    wl = circuit(basis, modes, 100, 3 * modes, 1e-3, None)
    eng, circ = graph(wl)
    circ.set_angles(wl.angles(wl.params * 1.03))
    pare(eng, circ, threshold)
    ev0, g0 = eng.graph_gradient(circ)
    ev1, g1 = eng.graph_gradient(circ, segment_gates=30)
    circ.close()
    eng.close()
    assert abs(ev0 - ev1) <= 1e-12 * max(1.0, abs(ev1))
    assert np.max(np.abs(g0 - g1)) <= 1e-11 * max(1.0, float(np.max(np.abs(g1))))
