"""Calls that fit into the device's memory keep working when what only makes them faster has no room.

A torch tensor holds the rest of the device's memory meanwhile.
"""

import contextlib

import numpy as np
import pytest
from test_gpu_window import circuit

from monoprop_b200 import _native

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
