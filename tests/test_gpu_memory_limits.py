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
    hold = torch.empty(max(torch.cuda.mem_get_info()[0] - nbytes, 0), dtype=torch.uint8, device="cuda")
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
