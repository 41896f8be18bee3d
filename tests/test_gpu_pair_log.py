"""The pair log of a recording forward pass (mpx_graph_build, mpx_adjoint_forward) on an engine that has recorded before,
and what a graph is reported to hold."""

import ctypes as C

import pytest

from monoprop_b200 import _native
from monoprop_b200 import workloads as W

pytestmark = pytest.mark.gpu


def used_bytes():
    import torch

    _native.load().mpx_trim_device_memory(0)
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_rebuilding_a_graph_holds_no_more_memory():
    """The first build sizes the log as it goes (at most four times too large); the second knows what the circuit
    needs: a quarter more than its 1.8e7 records of 9 bytes, in power-of-two blocks. It may not hold more than the
    first but for the rounding of one block (128 MiB)."""
    wl = W.ising50(8)
    eng = _native.engine_for(wl)
    circ = eng.upload(wl.gen_words(), wl.angles())
    used = []
    for _ in range(3):
        eng.graph_build(circ)
        used.append(used_bytes())
    circ.close()
    eng.close()
    assert used[1] <= used[0] + (128 << 20) and used[2] <= used[0] + (128 << 20)


def test_reported_graph_bytes_count_the_replay_order():
    """Sorted for windowed replays, a pair takes another 17 bytes: two terms, the phase and the gate mask."""
    wl = W.ising50(5)
    eng = _native.engine_for(wl)
    circ = eng.upload(wl.gen_words(), wl.angles())
    eng.graph_build(circ)

    def memory():
        info = _native.MemoryInfo()
        eng._check(eng.lib.mpx_memory(eng.h, C.byref(info)))
        return info

    built = memory()
    eng.graph_expectation(circ)
    replayed = memory()
    circ.close()
    eng.close()
    assert built.graph_pairs == replayed.graph_pairs > 0
    assert replayed.graph_bytes >= built.graph_bytes + 17 * built.graph_pairs
