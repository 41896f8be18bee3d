"""Profiling times the kernels that run without it (mpx_set_profiling): the same windows and the same gates one by one."""

import time

import numpy as np
import pytest

from monoprop_b200 import _native
from monoprop_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_profiled_propagation_takes_the_same_path():
    """The 10x10 lattice on a wide register (no shared-memory path), which changes between windows and single gates.
    Window lengths are chosen from a sample of terms, so the launches of two runs may differ by a few."""
    slots, g, pmap, params = W.kicked_ising(10, 10, 10, 3, 0.3 * np.pi)
    wl = W.Workload("wide", "pauli", 161, slots, g, pmap, params, {(100, 101): 1.0 + 0j}, [], 10, "support", 1e-4)
    launches, values = [], []
    for on in (False, True):
        eng = _native.engine_for(wl)
        eng.set_profiling(on)
        before = eng.launch_count()
        t = time.perf_counter()
        eng.propagate(wl.gen_words(), wl.angles())
        wall = 1e3 * (time.perf_counter() - t)
        launches.append(eng.launch_count() - before)
        values.append(eng.expectation())
        if on:
            first, rest, _, gates = eng.kernel_times()
            assert gates == wl.n_layers and first > 0 and rest > 0 and first + rest <= wall
        eng.close()
    assert abs(launches[1] - launches[0]) <= 0.1 * launches[0]
    assert abs(values[1] - values[0]) <= 1e-12


def test_windows_that_are_run_again_are_timed():
    """A store that starts at its smallest grows several times within the windows of one short circuit."""
    rng = np.random.default_rng(2)
    slots = [tuple(sorted(rng.choice(24, size=2, replace=False).tolist())) for _ in range(40)]
    wl = W.Workload("grow", "pauli", 161, slots, np.ones(40), np.arange(40), rng.uniform(0.3, 1.0, size=40),
                    {(0, 1): 1.0 + 0j, (4, 5): 0.5 + 0j}, [], 12, "support", 1e-6)
    out = []
    for on in (False, True):
        eng = _native.engine_for(wl, capacity_hint=1)
        eng.set_profiling(on)
        eng.propagate(wl.gen_words(), wl.angles())
        out.append((eng.size(), eng.expectation()))
        eng.close()
    assert out[0][0] == out[1][0] and abs(out[0][1] - out[1][1]) <= 1e-12
