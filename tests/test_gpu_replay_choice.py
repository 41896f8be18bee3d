"""When gates and frozen structures run in windows (csrc/mpx_window.cuh, mpx_replay.cuh) and when gate by gate.

Both give the same numbers (test_gpu_window.py, test_gpu_replay.py); these tests look at what a call costs, in launches or, where a
wrong choice costs a factor of a hundred, in time.
"""

import time

import numpy as np
import pytest

from monoprop_b200 import _native
from monoprop_b200 import workloads as W

pytestmark = pytest.mark.gpu


def on_few_modes(modes, used, gates, seed):
    """Random Pauli generators on `used` of the modes: the operator fills their 4^used strings."""
    rng = np.random.default_rng(seed)
    pool = np.array([2 * m + h for m in rng.choice(modes, size=used, replace=False) for h in (0, 1)])
    slots = [tuple(sorted(int(x) for x in rng.choice(pool, size=int(rng.choice([1, 2, 2, 3, 4])), replace=False)))
             for _ in range(gates)]
    z = 2 * (int(pool[0]) // 2)
    return W.Workload("few", "pauli", modes, slots, np.ones(gates), np.arange(gates), rng.uniform(-0.5, 0.5, size=gates),
                      {(z, z + 1): 1.0 + 0j}, [], 2 * modes, "support", None)


def graph(wl):
    eng = _native.engine_for(wl)
    circ = eng.upload(wl.gen_words(), wl.angles())
    eng.graph_build(circ)
    return eng, circ


def replay_launches(wl):
    eng, circ = graph(wl)
    eng.graph_expectation(circ)  # sorts the pairs, if the structure replays in windows
    before = eng.launch_count()
    eng.graph_expectation(circ)
    used = eng.launch_count() - before
    circ.close()
    eng.close()
    return used


def test_dense_structures_replay_gate_by_gate_and_sparse_ones_in_windows():
    """All of 4^10 terms paired at every gate: windows take 1.7 times as long. A lattice under lower_atol, few of whose
    terms are paired: half as long. Gate by gate is two launches per gate, a window two launches."""
    assert replay_launches(on_few_modes(20, 10, 150, 2)) >= 2 * 150
    assert replay_launches(W.ising50(4)) < W.ising50(4).n_layers


@pytest.mark.parametrize("modes", [20, 161])
def test_generators_on_few_modes_do_not_put_the_store_on_one_block(modes):
    """Two segments replay gate by gate. One block for all terms takes some hundred times as long as that."""
    wl = on_few_modes(modes, 9, 120, 1)
    eng, circ = graph(wl)

    def seconds(segment_gates):
        best = np.inf
        for _ in range(5):
            t = time.perf_counter()
            eng.graph_gradient(circ, segment_gates=segment_gates)
            best = min(best, time.perf_counter() - t)
        return best

    windows, gate_by_gate = seconds(0), seconds(60)
    circ.close()
    eng.close()
    assert windows <= 5 * gate_by_gate


def test_propagation_on_few_modes_does_not_stay_on_one_block():
    """only_rotate_len_k = all slots changes nothing but the path: gate by gate. Windows in which one block takes the
    whole store, as it grows from one term to 1e6 in one coset, take some twenty times as long."""
    wl = on_few_modes(161, 10, 150, 3)
    seconds, results = [], []
    for k in (None, 2 * wl.num_modes):
        best = np.inf
        for _ in range(4):
            eng = _native.engine_for(wl)
            eng.set_only_rotate_len_k(k)
            t = time.perf_counter()
            eng.propagate(wl.gen_words(), wl.angles())
            best = min(best, time.perf_counter() - t)
            result = (eng.size(), eng.expectation())
            eng.close()
        seconds.append(best)
        results.append(result)
    assert results[0][0] == results[1][0] and abs(results[0][1] - results[1][1]) <= 1e-12
    assert seconds[0] <= 5 * seconds[1]
