"""A window whose lists outgrow their scratch is given up: its gates run one by one, and the store, which has room, stays.

8e6 terms, a quarter of them active: two gates make the other three quarters join them, and a third, which emits nothing,
anticommutes with half of the terms. The lists then ask for 1.5 times as many places as there are terms; the scratch
has places for half the store's capacity and two chunks of 1024 per sector.
"""

import ctypes as C

import numpy as np
import pytest

from monoprop_b200 import _native

pytestmark = pytest.mark.gpu

QUARTER, CAPACITY = 1_950_000, 1 << 24


def key(*slots):
    return np.uint64(sum(1 << (63 - s) for s in slots))


def engine(len_k):
    rng = np.random.default_rng(5)
    base = np.unique(rng.integers(0, 1 << 44, size=2_200_000, dtype=np.uint64) << np.uint64(20))
    base, idle = base[:QUARTER], base[QUARTER:QUARTER + 50_000]  # strings on qubits 0 to 21
    keys = np.concatenate([base | key(44, 46), idle])  # X on qubits 22 and 23
    coefs = np.full(len(keys), 1e-9)
    coefs[:QUARTER] = rng.choice([-1.0, 1.0], size=QUARTER) * rng.uniform(0.5, 1.0, size=QUARTER)
    eng = _native.Engine(basis="pauli", cutoff_type="support", cutoff=32, num_modes=25, keys=keys[:, None], coefs=coefs, core=0.0,
                         state_mask=np.zeros(1, np.uint64), capacity_hint=CAPACITY)
    # their partners with Y, far below the lower_atol of the test (appended here, so that the store is half full)
    eng.propagate(np.array([[key(46, 47)], [key(44, 45)]], np.uint64), np.array([5e-10, 5e-10]))
    eng.set_lower_atol(1e-3)
    eng.set_only_rotate_len_k(len_k)
    return eng


def capacity(eng):
    info = _native.MemoryInfo()
    eng._check(eng.lib.mpx_memory(eng.h, C.byref(info)))
    return info.capacity


def test_full_lists_leave_the_store_as_it_is():
    # applied last to first: Z on qubits 22, 23 and 0, then 29 gates on qubit 24, where every term is the identity
    gens = np.array([key(48, 49)] * 29 + [key(0, 1), key(46, 47), key(44, 45)], np.uint64)[:, None]
    angles = np.array([0.3] * 29 + [1e-4, 0.35, 0.4])
    out = []
    for len_k in (None, 50):  # 50: every slot, which only keeps the gates out of windows
        eng = engine(len_k)
        before = capacity(eng)
        eng.propagate(gens, angles)
        keys, coefs = eng.export()
        order = np.argsort(keys[:, 0])
        st = eng.gate_stats()
        out.append((before, capacity(eng), keys[order, 0], coefs[order], np.stack([st.n, st.anti, st.emitted, st.appended])))
        eng.close()
    windows, by_gate = out
    assert by_gate[0] == by_gate[1] and windows[0] == windows[1]
    for a, b in zip(windows[2:], by_gate[2:]):
        assert np.array_equal(a, b)
    assert windows[4][2].sum() > 5_000_000 and windows[4][3].sum() == 0
