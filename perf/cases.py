"""The calls that the framework's speed is measured on, as a user's program makes them.

A case names a circuit family (``ising``: kicked Ising on an nx x ny lattice, ``line``: kicked Ising on a line of
nx qubits with angles up to pi, ``hubbard``: spinful Fermi-Hubbard Trotter steps on an nx x ny lattice), its
truncation, and the call:

* ``fresh``     create an engine from host arrays, propagate, read <O>, close;
* ``evolve``    reset a resident engine, propagate its resident circuit, read <O> and the per-gate counters;
* ``frontend``  ``from_circuit(...)`` of the Python propagators, its expectation value and evolved operator;
* ``gradient``  <O> and its gradient through ``DifferentiablePropagation`` (torch autograd);
* ``loop``      <O> and its gradient at new parameters over a structure built once (``build_graph``);
* ``batch``     many 5x10 kicked-Ising instances of uneven depth in one ``run_batch`` call.

``operator`` adds the evolved operator in canonical key order (small stores; a large one stays on the device).
"""

import dataclasses
import math

import numpy as np
import torch

from monoprop_b200 import Circuit, ExpGate, MajoranaOperator, MajoranaPropagator, Pauli, PauliOperator, PauliPropagator
from monoprop_b200 import _native
from monoprop_b200 import workloads as W
from monoprop_b200.autograd import DifferentiablePropagation
from monoprop_b200.batch import BatchConfig, run_batch

#: atol 0.0 stands for "no lower_atol"; schrodinger 0 for the Heisenberg picture; len_k 0 for no only_rotate_len_k.
BASE = {"kind": "ising", "nx": 10, "ny": 10, "layers": 1, "cutoff": 10, "atol": 1e-5, "call": "evolve",
        "operator": False, "schrodinger": 0, "len_k": 0, "jordan_wigner": False, "instances": 0}


def listed():
    def case(name, **kw):
        return {"name": name, **BASE, **kw}

    return [
        # the smallest calls: a short line through the Python front-end, its evolved operator read back, ...
        case("line16-frontend", kind="line", nx=16, ny=1, layers=5, cutoff=4, atol=0.0, call="frontend"),
        # ... and the 20-qubit line benchmark from host arrays, engine included (latency)
        case("line20-fresh", kind="line", nx=20, ny=1, layers=10, cutoff=8, atol=1e-4, call="fresh"),
        # truncation by weight alone (no lower_atol): every anticommuting term may emit; an odd line length
        case("line27-weight", kind="line", nx=27, ny=1, layers=9, cutoff=7, atol=0.0),
        # the Schrodinger picture: the reference state's monomials evolved, observable dotted in at the end
        case("line20-schrodinger", kind="line", nx=20, ny=1, layers=5, cutoff=8, atol=1e-4, schrodinger=4),
        # the 6x6 Hubbard benchmark, resident
        case("hubbard6x6", kind="hubbard", nx=6, ny=6, layers=8, cutoff=8),
        # a ragged Hubbard lattice whose cutoff is judged on the Jordan-Wigner image
        case("hubbard5x3-jw", kind="hubbard", nx=5, ny=3, layers=5, cutoff=6, jordan_wigner=True, call="fresh"),
        # the variational loop on a Hubbard circuit: structure built once, new parameters on every call
        case("hubbard6x6-loop", kind="hubbard", nx=6, ny=6, layers=4, cutoff=8, call="loop"),
        # one 50-qubit instance from host arrays: the store grows as it goes
        case("ising50-fresh", nx=10, ny=5, layers=12, cutoff=8, call="fresh"),
        # the gradient of a 50-qubit instance
        case("ising50-gradient", nx=10, ny=5, layers=8, cutoff=8, call="gradient"),
        # sixteen instances at once, as a parameter study or a data set needs them
        case("ising50-batch", nx=10, ny=5, layers=8, cutoff=8, call="batch", instances=16),
        # the variational loop at 100 qubits
        case("ising100-loop", layers=8, call="loop"),
        # the headline: the 100-qubit circuit of 5600 gates, resident
        case("ising100", layers=20),
    ]


def draw(rng):
    def log_int(lo, hi):
        return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5))))))

    c = dict(BASE)
    kind = rng.choice(["ising", "ising", "line", "hubbard", "hubbard", "schrodinger", "batch"])
    if kind == "ising":
        c.update(nx=rng.randint(3, 10), ny=rng.randint(2, 10), layers=log_int(2, 9), cutoff=rng.randint(4, 10),
                 atol=rng.choice([1e-5, 3e-5, 1e-4]), call=rng.choice(["evolve", "fresh", "gradient", "loop"]))
    elif kind == "line":
        c.update(kind="line", nx=rng.randint(8, 40), ny=1, layers=log_int(2, 10), cutoff=rng.randint(3, 8),
                 atol=rng.choice([1e-4, 3e-4, 1e-3]), call=rng.choice(["evolve", "fresh", "gradient"]))
        if c["cutoff"] <= 6 and rng.random() < 0.6:  # by weight alone: the set of terms does not depend on the angles
            c.update(nx=min(c["nx"], 30), atol=0.0)
            c["operator"] = c["cutoff"] <= 5 and c["call"] != "gradient"
            if c["cutoff"] <= 4 and c["layers"] <= 6:
                c.update(call="frontend", operator=False)
    elif kind == "hubbard":
        c.update(kind="hubbard", nx=rng.randint(2, 6), ny=rng.randint(2, 6), layers=log_int(1, 8),
                 cutoff=rng.randint(4, 8), atol=rng.choice([1e-5, 1e-4]),
                 call=rng.choice(["evolve", "fresh", "loop"]))
        if c["call"] == "fresh":
            c["jordan_wigner"] = rng.random() < 0.5
        elif c["call"] == "evolve" and rng.random() < 0.4:
            c["len_k"] = rng.randint(2, c["cutoff"])
    elif kind == "schrodinger":
        c.update(kind="line", nx=rng.randint(8, 20), ny=1, layers=log_int(2, 5), cutoff=rng.randint(4, 8), atol=1e-4,
                 schrodinger=4)
    else:
        c.update(nx=10, ny=5, layers=rng.randint(3, 8), cutoff=8, call="batch", instances=rng.randint(4, 16))
    return c


# ----- inputs ---------------------------------------------------------------------------------------------------


def _problem(case, seed):
    """The case's circuit, observable and truncation; the angles come from the seed."""
    kind, nx, ny, layers = case["kind"], case["nx"], case["ny"], case["layers"]
    atol = case["atol"] if case["atol"] > 0 else None
    if kind == "hubbard":
        wl = W.hubbard6x6(seed=seed, steps=layers, lx=nx, ly=ny)
        wl = dataclasses.replace(wl, cutoff=case["cutoff"], lower_atol=atol)
    else:
        if kind == "line":
            edges = [(i, i + 1) for i in range(nx - 1)]
            slots, g, pmap, params = W.kicked_ising(nx, 1, layers, seed, np.pi, edges)
            obs = {(2 * (nx // 2), 2 * (nx // 2) + 1): 1.0 + 0j}
        else:
            slots, g, pmap, params = W.kicked_ising(nx, ny, layers, seed, 0.3 * np.pi)
            n = nx * ny
            if n > 50:  # the average magnetisation
                obs = {(2 * i, 2 * i + 1): 1.0 / n + 0j for i in range(n)}
            else:
                obs = {(2 * (n // 2), 2 * (n // 2) + 1): 1.0 + 0j}
        wl = W.Workload(kind, "pauli", nx * ny, slots, g, pmap, params, obs, [], case["cutoff"], "support", atol)
    if case["schrodinger"]:
        wl.extra["schrodinger_cutoff"] = case["schrodinger"]
    if case["jordan_wigner"]:
        wl.extra["basis_change"] = _jordan_wigner(wl.num_modes)
    return wl


def _jordan_wigner(num_modes):
    return [[s] if s % 2 == 0 else [s - 1, s] for s in range(2 * num_modes)]


def _instances(case, seed):
    """Instances of the batched workload: uneven depths from 2 to the case's layers, one observable qubit each."""
    rng = np.random.default_rng(seed)
    depths = [2 + (5 * i + case["layers"] - 2) % (case["layers"] - 1) for i in range(case["instances"])]
    return [W.ising50(d, seed=1000 * seed + i, observable_qubit=int(rng.integers(0, 50)))
            for i, d in enumerate(depths)]


def _new_parameters(wl, seed):
    """Where an optimiser's next step would evaluate the structure built at wl.params."""
    return wl.params * (1.0 + 0.02 * np.random.default_rng(seed + 1).standard_normal(wl.params.shape))


def _frontend(wl):
    """The front-end's circuit and observable of a workload."""
    if wl.basis == "pauli":
        letters = {(0,): "X", (1,): "Y", (0, 1): "Z"}

        def pauli(slots):
            per = {}
            for s in slots:
                per.setdefault(s // 2, []).append(s % 2)
            return Pauli("".join(letters[tuple(v)] for v in per.values()), list(per))

        gates = [ExpGate(PauliOperator({pauli(m): float(g)}, wl.num_modes)) for m, g in zip(wl.gate_slots, wl.gen_coeffs)]
        circuit = Circuit(gates, wl.num_modes, wl.params, wl.initial_state)
        return circuit, PauliOperator({pauli(m): c for m, c in wl.observable.items()}, wl.num_modes), PauliPropagator
    circuit = Circuit.from_dense_arrays(wl.gate_slots, wl.gen_coeffs, wl.param_map, wl.num_modes, wl.params,
                                        wl.initial_state)
    return circuit, MajoranaOperator(dict(wl.observable), wl.num_modes), MajoranaPropagator


def _truncation(wl):
    return {"cutoff": wl.cutoff, "lower_atol": wl.lower_atol}


class _Fresh:
    """Host arrays of a problem, for an engine made anew on every call."""

    def __init__(self, wl, operator):
        keys, coefs, core = wl.encoded_observable()
        self.kw = dict(basis=wl.basis, cutoff_type=wl.cutoff_type, cutoff=wl.cutoff, num_modes=wl.num_modes, keys=keys,
                       coefs=coefs, core=core, state_mask=wl.state_mask(), lower_atol=wl.lower_atol,
                       schrodinger_cutoff=wl.extra.get("schrodinger_cutoff"))
        self.basis_change = wl.extra.get("basis_change")
        self.gens, self.angles, self.operator = wl.gen_words(), wl.angles(), operator


def prepare(case, seed):
    call = case["call"]
    state = {"call": call, "operator": case["operator"]}
    if call == "batch":
        state["workloads"] = _instances(case, seed)
        return state
    wl = _problem(case, seed)
    if call == "fresh":
        state["fresh"] = _Fresh(wl, case["operator"])
    elif call == "evolve":
        eng = _native.engine_for(wl)
        if case["len_k"]:
            eng.set_only_rotate_len_k(case["len_k"])
        state.update(engine=eng, circuit=eng.upload(wl.gen_words(), wl.angles()))
    elif call == "gradient":
        state["propagation"] = DifferentiablePropagation(wl)
        state["theta"] = torch.tensor(wl.params, dtype=torch.float64, device="cuda", requires_grad=True)
    else:
        circuit, observable, cls = _frontend(wl)
        state.update(circuit=circuit, observable=observable, cls=cls, truncation=_truncation(wl))
        if call == "loop":
            prop = cls(observable, wl.initial_state, **_truncation(wl))
            prop.build_graph(circuit)
            state["functional"] = prop.expectation_value_and_gradient_functional()
            state["parameters"] = _new_parameters(wl, seed)
    return state


# ----- one pass -------------------------------------------------------------------------------------------------


def _counters(eng):
    s = eng.gate_stats()
    return {"terms": s.n.astype(np.int64), "anticommuting": s.anti.astype(np.int64),
            "emitted": s.emitted.astype(np.int64), "appended": s.appended.astype(np.int64)}


def _sorted_operator(eng):
    keys, coefs = eng.export()
    order = np.lexsort([keys[:, w] for w in range(keys.shape[1])])
    return {"keys": keys[order], "coefs": coefs[order]}


def run(state):
    call = state["call"]
    if call == "fresh":
        f = state["fresh"]
        eng = _native.Engine(**f.kw)
        if f.basis_change is not None:
            eng.set_basis_change(f.basis_change)
        eng.propagate(f.gens, f.angles)
        out = {"value": np.float64(eng.expectation()), **_counters(eng), **(_sorted_operator(eng) if f.operator else {})}
        eng.close()
        return out
    if call == "evolve":
        eng = state["engine"]
        eng.reset()
        eng.propagate_circuit(state["circuit"])
        return {"value": np.float64(eng.expectation()), **_counters(eng), **(_sorted_operator(eng) if state["operator"] else {})}
    if call == "frontend":
        prop = state["cls"].from_circuit(state["circuit"], state["observable"], **state["truncation"])
        terms = prop.evolved_operator(atol=0.0).terms
        order = sorted(terms, key=lambda p: p.slots())
        return {"value": np.float64(prop.expectation_value()), "coefs": np.array([terms[p].real for p in order])}
    if call == "gradient":
        theta = state["theta"]
        theta.grad = None
        value = state["propagation"](theta)
        value.backward()
        return {"value": value.detach(), "gradient": theta.grad}
    if call == "loop":
        value, gradient = state["functional"](state["parameters"])
        return {"value": np.float64(value), "gradient": gradient}
    res = run_batch(state["workloads"], BatchConfig(), gradient=True)
    return {"values": res.expectations, "terms": res.final_terms.astype(np.int64), "gradients": np.concatenate(res.grads)}


def work(case):
    """Bytes: per gate, the coefficients of the anticommuting terms read and written and the appended terms
    written, as the per-gate counters of the case at one seed count them; a gradient also reads those
    coefficients again and updates their adjoints."""
    wls = _instances(case, 1) if case["call"] == "batch" else [_problem(case, 1)]
    nbytes = flops = 0.0
    for wl in wls:
        eng = _native.engine_for(wl)
        if case["len_k"]:
            eng.set_only_rotate_len_k(case["len_k"])
        eng.propagate(wl.gen_words(), wl.angles())
        s = eng.gate_stats()
        eng.close()
        anti, emitted, appended = (float(x.sum()) for x in (s.anti, s.emitted, s.appended))
        grad = case["call"] in ("gradient", "loop", "batch")
        nbytes += (40 if grad else 16) * anti + (8 * wl.words + 8) * appended
        flops += (4 if grad else 1) * anti + (18 if grad else 6) * emitted
    return {"bytes": nbytes, "flops": flops}


# ----- the same numbers from numpy, in 64 bits --------------------------------------------------------------------

EVEN = np.uint64(0x5555555555555555)
LIMIT = 4e7  # term-gate pairs (times key words) above which the numpy propagation would take too long


class _TooLong(Exception):
    pass


def _key(slots, words):
    out = np.zeros(words, np.uint64)
    for s in slots:
        bit = 64 * words - 1 - s
        out[bit // 64] |= np.uint64(1 << (bit % 64))
    return out


def _pop(k):
    return np.bitwise_count(k).astype(np.int64).sum(axis=-1)


def _score(keys, occupied, pauli):
    """<state|M|state> of every key: zero unless both slots of each mode are set or clear."""
    unpaired = ((keys & EVEN) ^ ((keys >> np.uint64(1)) & EVEN)).any(axis=1)
    sign = _pop(keys & occupied) + (0 if pauli else _pop(keys) // 2)
    return np.where(unpaired, 0.0, 1.0 - 2.0 * (sign & 1))


class _Numpy:
    """Truncated propagation in plain numpy: the store, and per gate which terms it touched."""

    def __init__(self, wl, len_k=0):
        self.words = words = wl.words
        self.pauli = wl.basis == "pauli"
        self.occupied = _key([2 * m for m in wl.initial_state], words)
        self.schrodinger = wl.extra.get("schrodinger_cutoff")
        rows = wl.extra.get("basis_change")
        self.rows = None if rows is None else np.array([_key(r, words) for r in rows])
        self.wl, self.len_k = wl, len_k
        order = sorted(wl.observable)
        self.core = sum(W.encode_coefficient(wl.basis, m, wl.observable[m]) for m in order if not m)
        self.obs = {_key(m, words).tobytes(): W.encode_coefficient(wl.basis, m, wl.observable[m]) for m in order if m}
        if self.schrodinger:
            import itertools

            start = [sum(((2 * q, 2 * q + 1) for q in sel), ()) for k in range((self.schrodinger + 1) // 2 + 1)
                     for sel in itertools.combinations(range(wl.num_modes), k)]
            self.keys = np.array([_key(m, words) for m in start])
            self.coefs = _score(self.keys, self.occupied, self.pauli)
        else:
            self.keys = np.array([np.frombuffer(k, np.uint64) for k in self.obs])
            self.coefs = np.array(list(self.obs.values()))
        self.start = self.coefs.copy()
        self.index = {k.tobytes(): i for i, k in enumerate(self.keys)}
        self.tape = []

    def _gate_order(self, angles):
        layers = range(self.wl.n_layers) if self.schrodinger else reversed(range(self.wl.n_layers))
        return [(layer, -angles[layer] if self.schrodinger else angles[layer]) for layer in layers]

    def _kept(self, p):
        if self.rows is not None:
            image = np.zeros_like(p)
            for s, row in enumerate(self.rows):
                b = 64 * self.words - 1 - s
                image ^= np.where(((p[:, b // 64] >> np.uint64(b % 64)) & np.uint64(1))[:, None] != 0, row, np.uint64(0))
            p = image
        a, b = p & EVEN, (p >> np.uint64(1)) & EVEN
        size = _pop(a | b) if self.wl.cutoff_type == "support" else _pop(p)
        return (_pop(a ^ b) == 0) | (size <= self.wl.cutoff)

    def _phase(self, m, p, g):
        one = np.uint64(1)
        if self.pauli:
            def y(k):
                return _pop((k & EVEN) & ~((k >> one) & EVEN))

            e = y(g) + y(m) - y(p) + 2 * _pop((m & EVEN) & (((g >> one) ^ g) & EVEN))
            return np.where((e & 3) == 1, -1.0, 1.0)
        above, mask = 0, np.zeros_like(g)
        for c in reversed(range(64 * self.words)):
            if above & 1:
                mask[c // 64] |= np.uint64(1 << (c % 64))
            above += int(g[c // 64] >> np.uint64(c % 64)) & 1
        a, b, c = _pop(m), int(_pop(g)), _pop(p)
        power = (a * (a - 1) // 2 + b * (b - 1) // 2 - c * (c - 1) // 2 + 3) & 3
        return np.array([1.0, 0.0, -1.0, 0.0])[power] * (1.0 - 2.0 * (_pop(m & mask) & 1))

    def propagate(self, angles):
        wl, spent = self.wl, 0
        gens = np.array([_key(m, self.words) for m in wl.gate_slots])
        for layer, angle in self._gate_order(angles):
            g, n = gens[layer], len(self.keys)
            spent += n * self.words
            if spent > LIMIT:
                raise _TooLong
            cos, sin = math.cos(2 * angle), math.sin(2 * angle)
            if self.pauli:
                anti = _pop(self.keys & (((g & EVEN) << np.uint64(1)) | ((g >> np.uint64(1)) & EVEN))) & 1
            else:
                anti = (_pop(self.keys & g) ^ (_pop(g) & _pop(self.keys))) & 1
            inside = _pop(self.keys) <= self.len_k if self.len_k else True
            idx = np.nonzero((anti == 1) & inside)[0]
            before = self.coefs.copy()
            self.coefs[idx] *= cos
            big = idx if wl.lower_atol is None else idx[~(abs(sin) * np.abs(before[idx]) <= wl.lower_atol)]
            src = big[self._kept(self.keys[big] ^ g)]
            partner = self.keys[src] ^ g
            tgt = np.array([self.index.get(p.tobytes(), -1) for p in partner], np.int64)
            word = int(np.nonzero(g)[0][0])
            follower = (self.keys[src, word] & (g[word] & (~g[word] + np.uint64(1)))) != 0
            emitted = np.zeros(n, bool)
            emitted[src[~follower]] = True
            phase = self._phase(self.keys[src], partner, g)
            use = ~(follower & (tgt >= 0) & emitted[tgt])
            src, tgt, phase, partner = src[use], tgt[use], phase[use], partner[use]
            new = tgt < 0
            tgt[new] = n + np.arange(int(new.sum()))
            if new.any():
                self.keys = np.concatenate([self.keys, partner[new]])
                first = _score(partner[new], self.occupied, self.pauli) if self.schrodinger else np.zeros(int(new.sum()))
                before = np.concatenate([before, first])
                self.coefs = np.concatenate([self.coefs, cos * first])
                self.index.update((p.tobytes(), int(t)) for p, t in zip(partner[new], tgt[new]))
            self.coefs[src] -= sin * phase * before[tgt]
            self.coefs[tgt] += sin * phase * before[src]
            self.tape.append((layer, np.concatenate([idx, tgt[new]]), src, tgt, phase))

    def value(self, coefs):
        if self.schrodinger:
            return self.core + sum(c * coefs[self.index[k]] for k, c in self.obs.items() if k in self.index)
        return self.core + float(np.sum(_score(self.keys, self.occupied, self.pauli) * coefs))

    def replay(self, angles):
        """<O> and its derivative by every angle over the structure that propagate() found."""
        c = np.zeros(len(self.keys))
        c[: len(self.start)] = self.start
        saved = []
        for layer, idx, src, tgt, phase in self.tape:
            cos, sin = math.cos(2 * angles[layer]), math.sin(2 * angles[layer])
            x, a, b = c[idx], c[src], c[tgt]
            saved.append((x, a, b))
            c[idx] *= cos
            c[src] -= sin * phase * b
            c[tgt] += sin * phase * a
        value, lam, grad = self.value(c), _score(self.keys, self.occupied, self.pauli), np.zeros(self.wl.n_layers)
        for (layer, idx, src, tgt, phase), (x, a, b) in zip(reversed(self.tape), reversed(saved)):
            cos, sin = math.cos(2 * angles[layer]), math.sin(2 * angles[layer])
            ls, lt = lam[src], lam[tgt]
            grad[layer] = -2 * sin * np.dot(lam[idx], x) + 2 * cos * np.dot(phase, lt * a - ls * b)
            lam[idx] *= cos
            lam[src] += sin * phase * lt
            lam[tgt] -= sin * phase * ls
        return value, grad


def exact(case, seed):
    call = case["call"]
    try:
        if call == "batch":
            values, grads = [], []
            for wl in _instances(case, seed):
                ref = _Numpy(wl)
                ref.propagate(wl.angles())
                value, grad = ref.replay(wl.angles())
                values.append(value)
                grads.append(grad)
            return {"values": np.array(values), "terms": None, "gradients": np.concatenate(grads)}
        wl = _problem(case, seed)
        ref = _Numpy(wl, case["len_k"])
        ref.propagate(wl.angles())
    except _TooLong:
        return None
    if call in ("gradient", "loop"):
        params = wl.params if call == "gradient" else _new_parameters(wl, seed)
        value, by_angle = ref.replay(wl.angles(params))
        grad = np.zeros(len(params))
        np.add.at(grad, wl.param_map, wl.gen_coeffs * by_angle)
        return {"value": np.float64(value), "gradient": grad}
    out = {"value": np.float64(ref.value(ref.coefs))}
    if call == "frontend":
        bits = np.unpackbits(ref.keys[:, ::-1].copy().byteswap().view(np.uint8), axis=1)
        slots = [tuple(np.nonzero(b)[0]) for b in bits]
        out["coefs"] = ref.coefs[sorted(range(len(slots)), key=slots.__getitem__)]
        return out
    out.update(terms=None, anticommuting=None, emitted=None, appended=None)
    if case["operator"]:
        out.update(keys=None, coefs=ref.coefs[np.lexsort([ref.keys[:, w] for w in range(ref.words)])])
    return out
