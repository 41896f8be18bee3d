"""The windowed replay of a frozen structure (csrc/mpx_replay.cuh) against the gate-by-gate one.

With segment_gates the graph gradient replays gate by gate from checkpoints; without, in windows of gates. Both
evaluate the same structure at the same angles, for circuit lengths around a window's, every key width, odd and
wide generators, and (through the gradient of a propagation) only_rotate_len_k. Their sums run in another order:
a derivative is a sum of up to some 1e6 products of at most 150 factors, each rounded to 1e-16, so with the sums
of their magnitudes within 1e2 of the largest entry they agree to 1e-11 of it.
"""

import numpy as np
import pytest
from test_gpu_window import circuit

from monoprop_b200 import _native

pytestmark = pytest.mark.gpu


def close(a, b):
    assert np.max(np.abs(a - b)) <= 1e-11 * max(1.0, float(np.max(np.abs(b))))


@pytest.mark.parametrize("gates", [1, 8, 63, 64, 65, 129])
@pytest.mark.parametrize("basis, modes", [("pauli", 30), ("majorana", 60), ("majorana", 130), ("pauli", 256)])
def test_windowed_replay_matches_gate_by_gate(basis, modes, gates):
    wl = circuit(basis, modes, gates, 7 * gates + modes, 1e-3, None)
    eng = _native.engine_for(wl)
    circ = eng.upload(wl.gen_words(), wl.angles())
    eng.graph_build(circ)
    circ.set_angles(wl.angles(wl.params + 0.05 * np.random.default_rng(gates).standard_normal(gates)))
    ev0 = eng.graph_expectation(circ)
    ev1, g1 = eng.graph_gradient(circ)
    ev2, g2 = eng.graph_gradient(circ, segment_gates=gates)
    circ.close()
    eng.close()
    assert abs(ev0 - ev2) <= 1e-11 * max(1.0, abs(ev2)) and abs(ev1 - ev2) <= 1e-11 * max(1.0, abs(ev2))
    close(g1, g2)


@pytest.mark.parametrize("basis, modes", [("pauli", 40), ("majorana", 90)])
def test_windowed_gradient_of_a_len_k_propagation(basis, modes):
    """First pass (windowed replay), second pass (logged values, no replay) and no pair log (streaming replay)."""
    wl = circuit(basis, modes, 100, modes, 1e-3, None)
    eng = _native.engine_for(wl)
    circ = eng.upload(wl.gen_words(), wl.angles())
    eng.set_only_rotate_len_k(5)
    grads = []
    for log in (-1, -1, 0):
        eng.set_pair_log(log)
        eng.adjoint_forward(circ)
        grads.append(eng.adjoint_backward(circ))
    circ.close()
    eng.close()
    assert np.count_nonzero(np.abs(grads[2]) > 1e-9) > 0
    close(grads[0], grads[2])
    close(grads[1], grads[2])
