"""Calls that fit into the device's memory keep working when what only makes them faster has no room.

A torch tensor holds the rest of the device's memory meanwhile.
"""

import contextlib

import numpy as np
import pytest
from test_gpu_window import circuit

from monoprop_b200 import _native
from monoprop_b200 import workloads as W

pytestmark = pytest.mark.gpu

MIB = 1 << 20


@contextlib.contextmanager
def only_free(nbytes):
    """Leaves about this much of the device's memory."""
    import torch

    _native.load().mpx_trim_device_memory(0)
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    rest, hold = max(torch.cuda.mem_get_info()[0] - nbytes, 0), None
    for _ in range(8):  # the last few MiB may not be had in one block
        with contextlib.suppress(torch.cuda.OutOfMemoryError):
            hold = torch.empty(rest, dtype=torch.uint8, device="cuda")
            break
        rest -= 16 * MIB
    assert hold is not None
    try:
        yield
    finally:
        del hold
        torch.cuda.empty_cache()


def test_window_scratch_is_given_back():
    """The windows' scratch of a store of 2^22 terms takes some 250 MiB; only_rotate_len_k needs another array of 32 MiB."""
    wl = circuit("majorana", 130, 100, 11, 1e-3, None)
    eng = _native.engine_for(wl, capacity_hint=1 << 22)
    eng.propagate(wl.gen_words(), wl.angles())
    plain = eng.expectation()
    eng.set_only_rotate_len_k(2 * wl.num_modes)  # every term: no effect on the result
    with only_free(24 * MIB):
        eng.reset()
        eng.propagate(wl.gen_words(), wl.angles())
        limited = eng.expectation()
    eng.close()
    assert abs(limited - plain) <= 1e-12


def test_a_graph_replays_in_windows_once_there_is_room():
    """Without memory for the sorted pairs (some 500 MiB) a graph replays gate by gate, two launches a gate; later calls
    try again."""
    wl = W.ising50(8)
    eng = _native.engine_for(wl)
    circ = eng.upload(wl.gen_words(), wl.angles())
    eng.graph_build(circ)

    def launches():
        before = eng.launch_count()
        return eng.graph_expectation(circ), eng.launch_count() - before

    with only_free(16 * MIB):
        limited = launches()
    launches()
    free = launches()
    circ.close()
    eng.close()
    assert abs(limited[0] - free[0]) <= 1e-12
    assert limited[1] >= 2 * wl.n_layers > wl.n_layers > free[1]


def test_gradient_pass_without_room_for_the_log():
    """A pass at tiny angles says that the log needs next to nothing. At the angles that follow, 5.5e6 terms are
    checkpointed at every replay window: some 100 blocks of 64 MiB, where 5.2 GiB are free. The forward pass
    then keeps one checkpoint, as it did for the first call."""
    gates = 2200
    rng = np.random.default_rng(8)
    slots = [tuple(sorted(rng.choice(42, size=int(rng.choice([1, 2, 2, 3])), replace=False).tolist())) for _ in range(gates)]
    wl = W.Workload("log", "pauli", 21, slots, np.ones(gates), np.arange(gates), rng.uniform(0.2, 0.6, size=gates),
                    {(0, 1): 1.0 + 0j, (20, 21): 1.0 + 0j}, [], 5, "support", 1e-12)
    angles = wl.angles()
    eng = _native.engine_for(wl)
    eng.set_pair_log(1 << 20)
    circ = eng.upload(wl.gen_words(), angles)
    eng.propagate_circuit(circ)
    plain, terms = eng.expectation(), eng.size()
    circ.set_angles(np.full(gates, 1e-13))
    eng.adjoint_forward(circ)
    circ.set_angles(angles)
    with only_free(5325 * MIB):
        value = eng.adjoint_forward(circ)
        logged = eng.adjoint_logged()
    circ.close()
    eng.close()
    assert terms > 1 << 22 and not logged
    assert abs(value - plain) <= 1e-10 * max(1.0, abs(plain))
