"""Gates applied in windows over the active terms (csrc/mpx_window.cuh), against the oracle.

Key widths above four words have no shared-memory path, so a propagation runs in windows from its first gate:
circuits of every length around a window's (8 to 64 gates), with repeated and dependent generators, generators
of more than eight slots (more columns than are read together) and odd Majorana generators. Keys and the
per-gate counters must be equal, coefficients bit-identical up to the order of two runs (1e-10 relative).
"""

import numpy as np
import pytest

import oracle
from monoprop_b200 import _native
from monoprop_b200 import workloads as W
from monoprop_b200.encoding import canonical_order

pytestmark = pytest.mark.gpu


def circuit(basis, modes, gates, seed, lower, upper):
    """Generators on a few scattered modes, a third of them repeats or products of earlier ones."""
    rng = np.random.default_rng(seed)
    pool = np.array([2 * m + h for m in rng.choice(modes, size=10, replace=False) for h in (0, 1)])
    slots = []
    for k in range(gates):
        if k > 3 and rng.random() < 0.33:
            a, b = (set(slots[i]) for i in rng.integers(0, k, size=2))
            s = a ^ b if rng.random() < 0.5 else a
        else:
            s = set(rng.choice(pool, size=int(rng.choice([1, 2, 3, 4, 11], p=[0.2, 0.25, 0.2, 0.25, 0.1])), replace=False).tolist())
        slots.append(tuple(sorted(int(x) for x in s)))  # () is the identity: a gate without effect
    obs = {tuple(sorted(int(x) for x in rng.choice(pool, size=2, replace=False))): 1.0 + 0j for _ in range(3)}
    if basis == "majorana":
        obs = {k: 1j for k in obs}
    return W.Workload("window", basis, modes, slots, rng.choice([-1.0, -0.5, 0.5, 1.0], size=gates),
                      np.arange(gates), rng.uniform(-1.5, 1.5, size=gates), obs, [0, 3], 7 if basis == "pauli" else 9,
                      "support" if basis == "pauli" else "length", lower, upper)


def check(wl, **kw):
    ref = oracle.run_port(wl)
    eng = _native.engine_for(wl, **kw)
    eng.propagate(wl.gen_words(), wl.angles())
    keys, coefs = eng.export()
    st = eng.gate_stats()
    eng.close()
    ia, ib = canonical_order(keys), canonical_order(ref.keys)
    assert np.array_equal(keys[ia], ref.keys[ib])
    a, b = coefs[ia], ref.coefs[ib]
    assert np.all(np.abs(a - b) <= 1e-10 * np.maximum(np.abs(a), np.abs(b)) + 1e-15)
    for got, col in ((st.n, 0), (st.anti, 1), (st.emitted, 2), (st.appended, 3)):
        np.testing.assert_array_equal(got, ref.counts[:, col])


@pytest.mark.parametrize("gates", [1, 7, 8, 9, 63, 64, 65, 150])
@pytest.mark.parametrize("basis", ["pauli", "majorana"])
def test_window_lengths(basis, gates):
    check(circuit(basis, 160, gates, gates, 1e-3, None))


@pytest.mark.parametrize("modes", [161, 200, 256])
@pytest.mark.parametrize("lower, upper", [(None, None), (1e-4, None), (1e-3, 0.05)])
def test_widths_and_truncation(modes, lower, upper):
    check(circuit("majorana", modes, 90, modes, lower, upper), capacity_hint=1)


def test_store_grows_inside_a_window():
    """A window whose appends do not fit is run again: the result does not depend on the starting capacity."""
    wl = W.ising50(4)
    check(wl, capacity_hint=1)
