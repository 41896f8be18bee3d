"""Resident circuits whose path was captured at one set of angles and replayed at others, and replays against segments.

A capture holds a number of windows, then gates one by one, then windows again. Other angles make other stores: the
captured sequence ends early or late, and the host goes on from there. A gradient's forward pass runs the same gates
one by one, with the same arithmetic: coefficients are the same bits, <O> up to the order of its sum.
"""

import dataclasses

import numpy as np
import pytest
from test_gpu_window import circuit

from monoprop_b200 import _native
from monoprop_b200 import workloads as W

pytestmark = pytest.mark.gpu


def lattice():
    slots, g, pmap, params = W.kicked_ising(4, 4, 8, 3, 0.3 * np.pi)
    return W.Workload("lattice", "pauli", 161, slots, g, pmap, params, {(16, 17): 1.0 + 0j}, [], 10, "support", 1e-4)


def schrodinger_line():
    edges = [(i, i + 1) for i in range(13)]
    slots, g, pmap, params = W.kicked_ising(14, 1, 4, 5, np.pi, edges)
    wl = W.Workload("line", "pauli", 150, slots, g, pmap, params, {(14, 15): 1.0 + 0j}, [], 6, "support", 1e-3)
    wl.extra["schrodinger_cutoff"] = 2
    return wl


@pytest.mark.parametrize("make", [lattice, schrodinger_line, lambda: dataclasses.replace(W.ising50(6), lower_atol=1e-4)])
def test_captured_sequence_at_other_angles(make):
    wl = make()
    a = wl.angles()
    half = np.arange(len(a)) < len(a) // 2
    steps = [a, a, a, 0.1 * a, a, np.where(half, 0.05 * a, a), np.where(half, a, 0.05 * a), 1.05 * a, a]

    def run(propagate):
        eng = _native.engine_for(wl)
        eng.set_pair_log(0)
        circ = eng.upload(wl.gen_words(), a)
        out = []
        for x in steps:
            circ.set_angles(x)
            propagate(eng, circ)
            keys, coefs = eng.export()
            order = np.lexsort(keys.T)
            st = eng.gate_stats()
            out.append((keys[order], coefs[order], np.stack([st.n, st.anti, st.emitted, st.appended]), eng.expectation()))
        replays = eng.graph_replay_count()
        circ.close()
        eng.close()
        return out, replays

    def resident(eng, circ):
        eng.reset()
        eng.propagate_circuit(circ)

    windows, replays = run(resident)
    by_gate, _ = run(lambda eng, circ: eng.adjoint_forward(circ))
    assert replays > 0
    for x, y in zip(windows, by_gate):
        assert all(np.array_equal(x[k], y[k]) for k in range(3))
        assert abs(x[3] - y[3]) <= 1e-12


@pytest.mark.parametrize("gates", [8, 63, 64, 65, 129])
@pytest.mark.parametrize("basis, modes", [("pauli", 30), ("majorana", 130), ("pauli", 256)])
def test_windowed_gradient_against_segments(basis, modes, gates):
    """One segment replays in windows, two gate by gate. (A derivative sums some 1e4 products of at most 150 factors
    each rounded to 1e-16: 1e-11 of the largest.)"""
    wl = circuit(basis, modes, gates, 5 * gates + modes, 1e-3, None)
    eng = _native.engine_for(wl)
    circ = eng.upload(wl.gen_words(), wl.angles())
    eng.graph_build(circ)
    circ.set_angles(wl.angles(wl.params * 1.04))
    ev0, g0 = eng.graph_gradient(circ)
    ev1, g1 = eng.graph_gradient(circ, segment_gates=(gates + 1) // 2)
    circ.close()
    eng.close()
    assert abs(ev0 - ev1) <= 1e-11 * max(1.0, abs(ev1))
    assert np.max(np.abs(g0 - g1)) <= 1e-11 * max(1.0, float(np.max(np.abs(g1))))
