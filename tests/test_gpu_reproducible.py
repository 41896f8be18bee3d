"""Gradients over one frozen structure are the same bits on every call, and on a clone of the engine.

The windowed reverse sweep sums over some thousand blocks; no sum may depend on which of them comes first, nor the
order of the pairs on how a sort's threads ran.
"""

import ctypes as C

import numpy as np
import pytest
from test_gpu_window import circuit

from monoprop_b200 import _native
from monoprop_b200 import workloads as W

pytestmark = pytest.mark.gpu


def clone(eng, circ):
    """The engine's clone and its copy of the circuit, as objects of the host layer."""
    h, hc = C.c_void_p(), C.c_void_p()
    eng._check(eng.lib.mpx_clone(eng.h, circ.h, C.byref(h), C.byref(hc)))
    e2, c2 = object.__new__(_native.Engine), object.__new__(_native.Circuit)
    e2.lib, e2.h, e2.words, e2.num_modes = eng.lib, h, eng.words, eng.num_modes
    c2.engine, c2.h, c2.n_layers = e2, hc, circ.n_layers
    return e2, c2


@pytest.mark.parametrize("make", [lambda: W.ising50(5), lambda: circuit("majorana", 130, 129, 4, 1e-4, None)])
def test_graph_gradient_bits(make):
    wl = make()
    eng = _native.engine_for(wl)
    circ = eng.upload(wl.gen_words(), wl.angles())
    eng.graph_build(circ)
    e2, c2 = clone(eng, circ)
    angles = wl.angles(wl.params * 1.01)
    circ.set_angles(angles)
    c2.set_angles(angles)
    first = eng.graph_gradient(circ)
    others = [eng.graph_gradient(circ) for _ in range(4)] + [e2.graph_gradient(c2) for _ in range(2)]
    for x in (circ, eng, c2, e2):
        x.close()
    for value, gradient in others:
        assert value == first[0] and np.array_equal(gradient, first[1])
