"""Performance cases of the engine: the work a user's program has it do.

Every case goes through a public entry point, with the circuit families of the
repository's benchmark and tests (random layered circuits, hardware-efficient
ansaetze, mid-circuit measurement, noise channels) over the sizes users run:

  simulate      quafu.simulate's call: ``qfvm.simulate_circuit`` on a circuit
                object, host arrays in and out, seeded shots
  plan          a compiled circuit (``engine.Plan``) on a device-resident state
  adjoint       energy and gradient of one ansatz (``gradients.adjoint``)
  batch         many circuits of uneven sizes, expectation values and
                gradients in one run (``batch.BatchSession``)
  qnn           a training step's forward and backward (``interface.QuantumLayer``)
  measure       Pauli expectation values and seeded shots of a device state
  trajectories  per-shot runs of a circuit with measurement, reset and
                classical control in its middle (``qfvm.simulate_circuit``)
  noise         noisy trajectories with unitary and Kraus channels
                (``noise.simulate_noise``)

A case's ``circuit`` number fixes the structure of its random circuits; the
seed gives the angles, inputs, states and uniforms, as in a variational or
sampling loop that runs one circuit structure on new values.
"""

import math

import numpy as np
import torch

from pyquafu_gb300 import ir, qfvm, workloads
from pyquafu_gb300 import gradients as gradients_mod
from pyquafu_gb300 import noise as noise_mod
from pyquafu_gb300.batch import BatchSession
from pyquafu_gb300.engine import DeviceState, Plan
from pyquafu_gb300.interface import QuantumLayer

AMP_BYTES = {"c128": 16, "c128_ds": 16, "c64": 8}


def listed():
    return [
        # the smallest calls: a classroom-sized circuit through quafu.simulate, latency bound
        {"name": "simulate_6q", "kind": "simulate", "n": 6, "depth": 6, "shots": 1000, "circuit": 1},
        # an ordinary small study (QAOA / VQE prototypes)
        {"name": "simulate_13q", "kind": "simulate", "n": 13, "depth": 13, "shots": 1024, "circuit": 2},
        # the benchmark's 20-qubit circuit: depth 20, 4096 shots, host arrays in and out
        {"name": "simulate_20q", "kind": "simulate", "n": 20, "depth": 20, "shots": 4096, "circuit": 0},
        # the benchmark's headline: 30 qubits, depth 40, complex128 in the engine's default arithmetic
        {"name": "plan_30q_c128_ds", "kind": "plan", "n": 30, "depth": 40, "precision": "c128_ds", "circuit": 0},
        # the same family in complex64, an odd size
        {"name": "plan_27q_c64", "kind": "plan", "n": 27, "depth": 40, "precision": "c64", "circuit": 3},
        # and in IEEE FP64, for users who need its last digits
        {"name": "plan_25q_fp64", "kind": "plan", "n": 25, "depth": 30, "precision": "c128", "circuit": 4},
        # the benchmark's adjoint gradient: 24 qubits, 960 parameters
        {"name": "adjoint_24q", "kind": "adjoint", "n": 24, "layers": 20, "precision": "c128_ds"},
        # the benchmark's batch of uneven circuits, complex64
        {"name": "batch_2048", "kind": "batch", "circuits": 2048, "nmin": 10, "nmax": 18, "layers": 6,
         "precision": "c64"},
        # the benchmark's QNN training step
        {"name": "qnn_1024x16q", "kind": "qnn", "batch": 1024, "n": 16, "layers": 12},
        # observables and shots of a large state that is on the device already
        {"name": "measure_28q", "kind": "measure", "n": 28, "precision": "c128", "shots": 4096},
        # mid-circuit measurement, reset and classical control, one trajectory per shot
        {"name": "trajectories_17q", "kind": "trajectories", "n": 17, "layers": 6, "shots": 2048, "circuit": 7},
        # noisy trajectories: depolarizing and amplitude-damping channels
        {"name": "noise_16q", "kind": "noise", "n": 16, "layers": 8, "shots": 1024, "circuit": 100},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["simulate", "simulate", "plan", "plan", "adjoint", "batch", "qnn", "measure", "trajectories",
                       "noise"])
    circuit = rng.randrange(1000)
    if kind == "simulate":
        n = rng.randint(2, 22)
        return {"kind": kind, "n": n, "depth": _log_int(rng, 3, 30), "shots": _log_int(rng, 1, 8192),
                "circuit": circuit}
    if kind == "plan":
        precision = rng.choice(["c128_ds", "c64", "c128"])
        return {"kind": kind, "n": rng.randint(12, 25 if precision == "c128" else 27),
                "depth": _log_int(rng, 4, 40), "precision": precision, "circuit": circuit}
    if kind == "adjoint":
        return {"kind": kind, "n": rng.randint(3, 23), "layers": _log_int(rng, 1, 16),
                "precision": rng.choice(["c128_ds", "c64", "c128"])}
    if kind == "batch":
        nmin = rng.randint(3, 12)
        return {"kind": kind, "circuits": _log_int(rng, 4, 1024), "nmin": nmin, "nmax": nmin + rng.randint(0, 5),
                "layers": rng.randint(1, 6), "precision": rng.choice(["c64", "c64", "c128_ds"])}
    if kind == "qnn":
        return {"kind": kind, "batch": _log_int(rng, 1, 700), "n": rng.randint(3, 16), "layers": rng.randint(1, 10)}
    if kind == "measure":
        return {"kind": kind, "n": rng.randint(8, 27), "precision": rng.choice(["c128", "c64"]),
                "shots": _log_int(rng, 1, 16384)}
    if kind == "trajectories":
        return {"kind": kind, "n": rng.randint(4, 16), "layers": rng.randint(1, 6), "shots": _log_int(rng, 1, 2000),
                "circuit": circuit}
    return {"kind": kind, "n": rng.randint(3, 15), "layers": 2 * rng.randint(1, 3), "shots": _log_int(rng, 1, 1000),
            "circuit": circuit}


# ------------------------------------------------------------------ circuits
# A gate is (name, qubits with controls first, angle or None).

CONTROLS = {"cx": 1, "cz": 1, "ccx": 2}


def random_layers(n, depth, circuit, angles, extras=False):
    """Layers of random one-qubit gates and cx on a random matching; with
    ``extras`` about 5% of the layers also get cz, swap, rzz and ccx.
    ``circuit`` fixes the structure, ``angles`` (a generator) the values."""
    rng = np.random.default_rng(circuit)
    turn = lambda: float(angles.uniform(0.0, 2 * np.pi))  # noqa: E731
    gates = []
    for _ in range(depth):
        for q in range(n):
            g = workloads.ONE_QUBIT[int(rng.integers(len(workloads.ONE_QUBIT)))]
            gates.append((g, (q,), turn() if g in ("rx", "ry", "rz") else None))
        perm = rng.permutation(n)
        for i in range(0, n - 1, 2):
            gates.append(("cx", (int(perm[i]), int(perm[i + 1])), None))
        if extras and n >= 3 and rng.random() < 0.05:
            for g, k in (("cz", 2), ("swap", 2), ("rzz", 2), ("ccx", 3)):
                qs = tuple(int(x) for x in rng.choice(n, k, replace=False))
                gates.append((g, qs, turn() if g == "rzz" else None))
    return gates


def hea(n, layers, encode):
    """Hardware-efficient ansatz as (name, qubits, slot or None) gates: slots
    0..2*n*layers-1 are the weights, then (with ``encode``) n input angles."""
    gates = [("ry", (q,), 2 * n * layers + q) for q in range(n)] if encode else []
    k = 0
    for _ in range(layers):
        for name in ("ry", "rz"):
            for q in range(n):
                gates.append((name, (q,), k))
                k += 1
        gates += [("cx", (q, q + 1), None) for q in range(n - 1)]
    return gates


def to_ops(gates, slotted=False, values=None):
    """The engine's packed input for a gate list."""
    ops = []
    for name, qs, a in gates:
        if name == "swap":
            ops.append(workloads.matrix_gate("swap", qs, workloads.SWAP))
        elif a is None:
            ops.append(workloads.named(name, qs, ncontrols=CONTROLS.get(name, 0)))
        elif slotted:
            ops.append(ir.Op(name, ir.NAMED_KIND[name], qs, 0, (float(values[a]) if values is not None else 0.0,),
                             slot=a))
        else:
            ops.append(workloads.named(name, qs, (a,)))
    return ops


def observable(n, rng):
    """sum a_i Z_i Z_{i+1} + sum b_i X_i, a and b normal."""
    a, b = rng.normal(size=n - 1), rng.normal(size=n)
    return [(float(a[i]), "ZZ", [i, i + 1]) for i in range(n - 1)] + [(float(b[i]), "X", [i]) for i in range(n)]


def pauli_strings(n):
    """What a program measures on a large state: neighbours, fields and a few long strings."""
    terms = [("ZZ", [i, i + 1]) for i in range(0, n - 1, 2)] + [("X", [i]) for i in range(0, n, 4)]
    return terms + [("Z" * n, list(range(n))), ("XYZ", [0, n // 2, n - 1]), ("YY", [1, n - 2])]


class _Instruction:
    """An instruction of quafu's circuit protocol."""

    def __init__(self, name, **fields):
        self.name = name
        self.__dict__.update(fields)


class _Circuit:
    """quafu's circuit protocol: instructions, qubit and classical-bit counts."""

    def __init__(self, num, cbits_num, instructions):
        self.num, self.cbits_num, self.instructions = num, cbits_num, instructions


def _gate_objects(n, gates):
    return workloads.as_protocol(n, to_ops(gates)).instructions


class _DeviceArray:
    """A state's device buffer as a CUDA array (interop through ``device_ptr``)."""

    def __init__(self, state, precision):
        real = "<f4" if precision == "c64" else "<f8"
        self.state = state
        self.__cuda_array_interface__ = {"shape": (state.size, 2), "typestr": real, "version": 2,
                                         "data": (state.device_ptr()[0], False), "strides": None}


def _view(state, precision):
    return torch.view_as_complex(torch.as_tensor(_DeviceArray(state, precision), device="cuda"))


X, Y, Z = np.array([[0, 1], [1, 0]], complex), np.array([[0, -1j], [1j, 0]]), np.diag([1.0, -1.0]).astype(complex)
P_DEPOL, G_DAMP = 0.02, 0.05
DEPOL = ([X, Y, Z, np.eye(2, dtype=complex)], [P_DEPOL / 3, P_DEPOL / 3, P_DEPOL / 3, 1 - P_DEPOL])
DAMP = [np.array([[1, 0], [0, np.sqrt(1 - G_DAMP)]], complex), np.array([[0, np.sqrt(G_DAMP)], [0, 0]], complex)]


def noisy_circuit(n, layers, circuit, angles):
    """Random layers; after every second one a depolarizing and an
    amplitude-damping channel on each qubit."""
    gates = []
    for layer in range(layers):
        gates += random_layers(n, 1, circuit + layer, angles)
        if layer % 2:
            for q in range(n):
                gates += [("depolarize", (q,), None), ("damp", (q,), None)]
    return gates


def noise_terms(n):
    return [(1.0, "Z", [0]), (0.5, "ZZ", [0, 1]), (0.25, "X", [n - 1])]


def _mid_circuit(case, seed):
    """(gates before, gates after) a measurement of qubits 0 and 1, a reset
    of qubit 2 and a block run where both outcomes are 1."""
    n, angles = case["n"], np.random.default_rng(seed)
    return (random_layers(n, case["layers"], case["circuit"], angles),
            random_layers(n, case["layers"], case["circuit"] + 1, angles))


def uneven_sizes(case, seed):
    ns = np.random.default_rng(case["circuits"]).integers(case["nmin"], case["nmax"] + 1, size=case["circuits"])
    rng = np.random.default_rng(seed)
    groups = {}
    for n in range(case["nmin"], case["nmax"] + 1):
        count = int(np.sum(ns == n))
        if count:
            nw = 2 * n * case["layers"]
            groups[n] = np.concatenate([rng.uniform(0.0, 2 * np.pi, (count, nw)),
                                        rng.uniform(-np.pi, np.pi, (count, n))], axis=1)
    return groups


def _qnn_data(case, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(case["batch"], case["n"]))
    y = np.where(x @ rng.normal(size=case["n"]) >= 0, 1.0, -1.0)
    return rng.uniform(0.0, 2 * np.pi, 2 * case["n"] * case["layers"]), x, y


# ---------------------------------------------------------- prepare and run


def prepare(case, seed):
    kind = case["kind"]
    if kind == "simulate":
        gates = random_layers(case["n"], case["depth"], case["circuit"], np.random.default_rng(seed), extras=True)
        circ = workloads.as_protocol(case["n"], to_ops(gates), measures=[(q, q) for q in range(case["n"])])
        return {"kind": kind, "circuit": circ, "shots": case["shots"], "seed": seed}
    if kind == "plan":
        gates = random_layers(case["n"], case["depth"], case["circuit"], np.random.default_rng(seed), extras=True)
        state = DeviceState(case["n"], case["precision"])
        return {"kind": kind, "state": state, "plan": Plan(case["n"], to_ops(gates), case["precision"]),
                "view": _view(state, case["precision"])}
    if kind == "adjoint":
        rng = np.random.default_rng(seed)
        n, layers = case["n"], case["layers"]
        ops = to_ops(hea(n, layers, False), True, rng.uniform(0.0, 2 * np.pi, 2 * n * layers))
        return {"kind": kind, "n": n, "ops": ops, "terms": observable(n, rng), "precision": case["precision"]}
    if kind == "batch":
        session, values = BatchSession(case["precision"], grads=True), []
        for n, vals in uneven_sizes(case, seed).items():
            session.add_group(n, to_ops(hea(n, case["layers"], True), True), [(1.0, "Z", [0])], len(vals),
                              vals.shape[1])
            values.append(vals)
        return {"kind": kind, "session": session, "values": values, "precision": case["precision"]}
    if kind == "qnn":
        n, layers = case["n"], case["layers"]
        weights, x, y = _qnn_data(case, seed)
        nw = len(weights)
        layer = QuantumLayer(n, to_ops(hea(n, layers, True), True), [(1.0, "Z", [0])], range(nw), range(nw, nw + n),
                             init=weights)
        return {"kind": kind, "layer": layer, "x": torch.from_numpy(x), "y": torch.from_numpy(y)}
    if kind == "measure":
        state = DeviceState(case["n"], case["precision"])
        _view(state, case["precision"]).copy_(_random_state(case["n"], seed, case["precision"]))
        torch.cuda.synchronize()
        return {"kind": kind, "state": state, "terms": pauli_strings(case["n"]),
                "uniforms": np.random.default_rng(seed).random(case["shots"])}
    if kind == "trajectories":
        n = case["n"]
        before, after = _mid_circuit(case, seed)
        ins = _gate_objects(n, before)
        ins += [_Instruction("measure", qbits=[0, 1], cbits=[0, 1]), _Instruction("reset", pos=[2]),
                _Instruction("cif", cbits=[0, 1], condition=3,
                             instructions=_gate_objects(n, [("x", (2,), None), ("h", (3,), None)]))]
        ins += _gate_objects(n, after) + [_Instruction("measure", qbits=[0, 1, 2, 3], cbits=[2, 3, 4, 5])]
        return {"kind": kind, "circuit": _Circuit(n, 6, ins), "shots": case["shots"], "seed": seed}
    rng = np.random.default_rng(seed)
    n = case["n"]
    ops = []
    for name, qs, a in noisy_circuit(n, case["layers"], case["circuit"], rng):
        if name == "depolarize":
            ops.append(ir.channel_op(ir.OP_UCHANNEL, qs[0], *DEPOL))
        elif name == "damp":
            ops.append(ir.channel_op(ir.OP_KRAUS, qs[0], DAMP))
        else:
            ops += to_ops([(name, qs, a)])
    return {"kind": "noise", "n": n, "ops": ops, "shots": case["shots"], "terms": noise_terms(n),
            "uniforms": rng.random((case["shots"], ir.noise_draws(ops)))}


def run(state):
    kind = state["kind"]
    if kind in ("simulate", "trajectories"):
        qfvm.set_seed(state["seed"])  # reproducible shots
        counts, psi = qfvm.simulate_circuit(state["circuit"], shots=state["shots"])
        keys = sorted(counts)  # every shot's outcome, in ascending order
        return {"state": psi, "outcomes": np.repeat(np.array(keys, np.int64), [counts[k] for k in keys])}
    if kind == "plan":
        state["plan"].run(state["state"].set_zero())
        return state["view"]
    if kind == "adjoint":
        energy, grads = gradients_mod.adjoint(state["n"], state["ops"], state["terms"], state["precision"])
        # a complex64 run's results carry single precision: kept as such
        return (np.float32(energy), grads.astype(np.float32)) if state["precision"] == "c64" else (energy, grads)
    if kind == "batch":
        exps, grads = state["session"].run(state["values"], grads=True)
        if state["precision"] == "c64":  # as above
            exps, grads = [e.astype(np.float32) for e in exps], [g.astype(np.float32) for g in grads]
        return {"expectations": exps, "gradients": grads}
    if kind == "qnn":
        layer = state["layer"]
        layer.zero_grad(set_to_none=True)
        out = layer(state["x"])[:, 0].float()  # the layer computes in complex64; the loss is a float32 one
        loss = torch.mean((out - state["y"].float()) ** 2)
        loss.backward()
        return {"out": out.detach(), "loss": loss.detach(), "grad": layer.weight.grad.float()}
    if kind == "measure":
        return {"expectations": state["state"].expect(state["terms"]),
                "shots": state["state"].sample(state["uniforms"]).view(np.int64)}
    samples, expv = noise_mod.simulate_noise(state["n"], state["ops"], state["shots"], terms=state["terms"],
                                             uniforms=state["uniforms"])
    return {"samples": samples.view(np.int64), "expectations": expv}


# --------------------------------------------------------------------- work


def _gate_flops(gates, n):
    """Real operations on the amplitudes a gate has to change."""
    per_amp = {"h": 4, "rx": 6, "ry": 6, "rz": 6, "s": 1, "t": 3, "rzz": 6, "cz": 0.5}
    return sum(per_amp.get(g[0], 0) for g in gates) * 2.0**n


def work(case):
    kind = case["kind"]
    rng = np.random.default_rng(0)
    if kind == "simulate":
        n = case["n"]
        gates = random_layers(n, case["depth"], case["circuit"], rng, extras=True)
        return {"bytes": 16.0 * 2**n + 16 * case["shots"], "flops": _gate_flops(gates, n)}
    if kind == "plan":
        n = case["n"]
        gates = random_layers(n, case["depth"], case["circuit"], rng, extras=True)
        return {"bytes": float(AMP_BYTES[case["precision"]]) * 2**n, "flops": _gate_flops(gates, n)}
    if kind == "adjoint":
        n = case["n"]
        # forward, then both states back, with an inner product per parameter
        gates = hea(n, case["layers"], False)
        return {"bytes": 16.0 * 2 * n * case["layers"],
                "flops": 3 * _gate_flops(gates, n) + 2 * n * case["layers"] * 4 * 2.0**n}
    if kind == "batch":
        b = f = 0.0
        for n, vals in uneven_sizes(case, 0).items():
            b += 16.0 * vals.size + 8 * len(vals)
            f += len(vals) * (3 * _gate_flops(hea(n, case["layers"], True), n) + vals.shape[1] * 4 * 2.0**n)
        return {"bytes": b, "flops": f}
    if kind == "qnn":
        n, b = case["n"], case["batch"]
        slots = 2 * n * case["layers"] + n
        return {"bytes": 8.0 * (b * (n + 2) + 2 * (slots - n)),
                "flops": b * (3 * _gate_flops(hea(n, case["layers"], True), n) + slots * 4 * 2.0**n)}
    if kind == "measure":
        n = case["n"]
        return {"bytes": float(AMP_BYTES[case["precision"]]) * 2**n + 16 * case["shots"],
                "flops": (3 + len(pauli_strings(n))) * 2.0**n}
    n, shots = case["n"], case["shots"]
    if kind == "trajectories":
        before, after = _mid_circuit(case, 0)
        return {"bytes": 16.0 * 2**n + 16 * shots,
                "flops": _gate_flops(before, n) + shots * (_gate_flops(after, n) + 12 * 2.0**n)}
    gates = noisy_circuit(n, case["layers"], case["circuit"], rng)
    channels = sum(1 for g in gates if g[0] == "damp")
    return {"bytes": 8.0 * shots * (2 * channels + 5), "flops": shots * (_gate_flops(gates, n) + channels * 6 * 2.0**n)}


# -------------------------------------------------------------------- exact
# The same results in plain torch, complex128, without the engine.


def _random_state(n, seed, precision):
    """A normalised complex Gaussian state: what a deep random circuit ends in."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    real = torch.float32 if precision == "c64" else torch.float64
    psi = torch.view_as_complex(torch.randn(1 << n, 2, generator=g, device="cuda", dtype=real))
    return psi.mul_(float(1.0 / torch.sqrt(psi.abs().square().sum(dtype=torch.float64))))


def _zero(b, n):
    psi = torch.zeros(b, 1 << n, dtype=torch.complex128, device="cuda")
    psi[:, 0] = 1.0
    return psi


def _halves(psi, q):
    v = psi.view(psi.shape[0], -1, 2, 1 << q)
    return v[:, :, 0], v[:, :, 1]


def _bits(psi, fixed):
    """The view of psi whose qubits in ``fixed`` (a dict) have the given values."""
    qs = sorted(fixed, reverse=True)
    n = psi.shape[1].bit_length() - 1
    shape, index, top = [psi.shape[0]], [slice(None)], n
    for q in qs:
        shape += [1 << (top - 1 - q), 2]
        index += [slice(None), fixed[q]]
        top = q
    return psi.view(*shape, 1 << top)[tuple(index)]


def _per_item(v):
    """A coefficient: a number, or one per item (broadcast over a half state)."""
    return v.view(-1, 1, 1) if isinstance(v, torch.Tensor) else v


def _apply(psi, name, qs, a=None):
    """In place; ``a``: the angle, a number or one per item."""
    if name in ("h", "rx", "ry"):
        lo, hi = _halves(psi, qs[-1])
        if name == "h":
            s = 1 / math.sqrt(2)
            new_lo = (lo + hi) * s
            hi.copy_((lo - hi) * s)
        else:
            half = a / 2
            c, s = (torch.cos(half), torch.sin(half)) if isinstance(a, torch.Tensor) else (math.cos(half), math.sin(half))
            c, s = _per_item(c), _per_item(s)
            f, g = (-s, s) if name == "ry" else (-1j * s, -1j * s)
            new_lo = c * lo + f * hi
            hi.copy_(g * lo + c * hi)
        lo.copy_(new_lo)
    elif name in ("x", "cx", "ccx"):
        ctl = {q: 1 for q in qs[:-1]}
        lo, hi = _bits(psi, {**ctl, qs[-1]: 0}), _bits(psi, {**ctl, qs[-1]: 1})
        keep = lo.clone()
        lo.copy_(hi)
        hi.copy_(keep)
    elif name == "swap":
        u, v = _bits(psi, {qs[0]: 0, qs[1]: 1}), _bits(psi, {qs[0]: 1, qs[1]: 0})
        keep = u.clone()
        u.copy_(v)
        v.copy_(keep)
    elif name in ("s", "t"):
        _halves(psi, qs[0])[1].mul_(1j if name == "s" else complex(math.sqrt(0.5), math.sqrt(0.5)))
    elif name == "cz":
        _bits(psi, {qs[0]: 1, qs[1]: 1}).neg_()
    elif name == "rz":
        d = torch.exp(0.5j * a) if isinstance(a, torch.Tensor) else complex(math.cos(a / 2), math.sin(a / 2))
        d = _per_item(d)
        lo, hi = _halves(psi, qs[0])
        lo.mul_(d.conj() if isinstance(d, torch.Tensor) else d.conjugate())
        hi.mul_(d)
    elif name == "rzz":
        d = complex(math.cos(a / 2), math.sin(a / 2))
        for i in (0, 1):
            for j in (0, 1):
                _bits(psi, {qs[0]: i, qs[1]: j}).mul_(d if i != j else d.conjugate())
    else:
        raise ValueError(name)


def _pauli(psi, string, pos):
    out = psi.clone()
    for ch, q in zip(string, pos):
        lo, hi = _halves(out, q)
        if ch == "Z":
            hi.neg_()
        else:
            new_lo = hi * (-1j if ch == "Y" else 1)
            hi.copy_(lo * (1j if ch == "Y" else 1))
            lo.copy_(new_lo)
    return out


def _inner(u, v):
    """Per item Re and Im of <u|v>."""
    z = torch.linalg.vecdot(u, v, dim=1)
    return z.real, z.imag


def _exact_gradient(n, gates, values, terms):
    """(<H> per item, d<H>/d value) of a slotted circuit, by the adjoint method."""
    b = values.shape[0]
    psi = _zero(b, n)
    for name, qs, k in gates:
        _apply(psi, name, qs, None if k is None else values[:, k])
    lam = sum(c * _pauli(psi, p, pos) for c, p, pos in terms)
    energy, _ = _inner(psi, lam)
    grads = torch.zeros(b, values.shape[1], dtype=torch.float64, device="cuda")
    for name, qs, k in reversed(gates):
        if k is not None:  # d/dtheta exp(-i theta Q / 2): Im <lam|Q|psi>
            l0, l1 = _halves(lam, qs[0])
            p0, p1 = _halves(psi, qs[0])
            dot = lambda u, v: (u.conj() * v).sum(dim=(1, 2))  # noqa: E731
            z = dot(l0, p0) - dot(l1, p1) if name == "rz" else -1j * dot(l0, p1) + 1j * dot(l1, p0)
            grads[:, k] += z.imag
        for s in (psi, lam):
            _apply(s, name, qs, None if k is None else -values[:, k])
    return energy, grads


def _exact_shot(case, seed):
    """The last shot's state: the engine's uniforms, outcome m the first with u * total < cum[m]."""
    n = case["n"]
    before, after = _mid_circuit(case, seed)
    uni = np.random.default_rng(seed).random(case["shots"] * 3).reshape(case["shots"], 3)[-1]
    psi = _zero(1, n)
    for g in before:
        _apply(psi, *g)

    def outcome(qs, u):
        p = np.array([float(_bits(psi, {q: (m >> k) & 1 for k, q in enumerate(qs)}).abs().square().sum())
                      for m in range(1 << len(qs))])
        m = min(int(np.searchsorted(np.cumsum(p), u * p.sum(), side="right")), len(p) - 1)
        for other in range(1 << len(qs)):
            part = _bits(psi, {q: (other >> k) & 1 for k, q in enumerate(qs)})
            part.mul_(1 / math.sqrt(p[m]) if other == m else 0.0)
        return m

    both = outcome([0, 1], uni[0]) == 3
    if outcome([2], uni[1]) == 1:
        _apply(psi, "x", (2,))
    if both:
        _apply(psi, "x", (2,))
        _apply(psi, "h", (3,))
    for g in after:
        _apply(psi, *g)
    outcome([0, 1, 2, 3], uni[2])
    return psi[0]


def _exact_noise(case, seed):
    n, shots = case["n"], case["shots"]
    rng = np.random.default_rng(seed)
    gates = noisy_circuit(n, case["layers"], case["circuit"], rng)
    nu = sum(1 for g in gates if g[0] == "depolarize")
    uni = rng.random((shots, 2 * nu + 1))  # unitary channels, Kraus channels, sample
    pick = np.searchsorted(np.cumsum(DEPOL[1]), uni[:, :nu], side="right")
    unitaries = torch.tensor(np.array(DEPOL[0]), device="cuda")
    psi = _zero(shots, n)
    iu = ik = 0
    for name, qs, a in gates:
        if name == "depolarize":
            m = unitaries[torch.from_numpy(np.minimum(pick[:, iu], 3)).cuda()]
            iu += 1
        elif name == "damp":
            u = torch.from_numpy(uni[:, nu + ik]).cuda()
            ik += 1
            lo, hi = _halves(psi, qs[0])
            p0 = lo.abs().square().sum(dim=(1, 2)), hi.abs().square().sum(dim=(1, 2))
            norm0, norm1 = torch.sqrt(p0[0] + (1 - G_DAMP) * p0[1]), torch.sqrt(G_DAMP * p0[1])
            first = u < norm0 / torch.sqrt(p0[0] + p0[1])
            k = torch.tensor(np.array(DAMP), device="cuda")
            m = torch.where(first.view(-1, 1, 1), k[0] / norm0.view(-1, 1, 1), k[1] / norm1.view(-1, 1, 1))
        else:
            _apply(psi, name, qs, a)
            continue
        lo, hi = _halves(psi, qs[0])
        e = lambda r, c: m[:, r, c].view(-1, 1, 1)  # noqa: E731
        new_lo = e(0, 0) * lo + e(0, 1) * hi
        hi.copy_(e(1, 0) * lo + e(1, 1) * hi)
        lo.copy_(new_lo)
    return torch.stack([c * _inner(psi, _pauli(psi, p, pos))[0] for c, p, pos in noise_terms(n)], dim=1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("simulate", "plan"):
        n = case["n"]
        gates = random_layers(n, case["depth"], case["circuit"], np.random.default_rng(seed), extras=True)
        if len(gates) * 2.0**n > 3e11:  # over 20 seconds
            return None
        psi = _zero(1, n)
        for g in gates:
            _apply(psi, *g)
        if kind == "plan":
            return psi[0]
        return {"state": psi[0], "outcomes": None}
    if kind == "trajectories":
        return {"state": _exact_shot(case, seed), "outcomes": None}
    if kind == "adjoint":
        rng = np.random.default_rng(seed)
        n, layers = case["n"], case["layers"]
        values = torch.from_numpy(rng.uniform(0.0, 2 * np.pi, 2 * n * layers)).cuda().view(1, -1)
        energy, grads = _exact_gradient(n, hea(n, layers, False), values, observable(n, rng))
        return energy[0], grads[0]
    if kind == "batch":
        exps, grads = [], []
        for n, vals in uneven_sizes(case, seed).items():
            e, g = _exact_gradient(n, hea(n, case["layers"], True), torch.from_numpy(vals).cuda(), [(1.0, "Z", [0])])
            exps.append(e.view(-1, 1))
            grads.append(g)
        return {"expectations": exps, "gradients": grads}
    if kind == "qnn":
        n = case["n"]
        weights, x, y = _qnn_data(case, seed)
        values = np.concatenate([np.broadcast_to(weights, (len(x), len(weights))), x], axis=1)
        e, g = _exact_gradient(n, hea(n, case["layers"], True), torch.from_numpy(values).cuda(), [(1.0, "Z", [0])])
        d = e - torch.from_numpy(y).cuda()
        grad = (2 * d / len(x)).view(1, -1) @ g[:, : len(weights)]
        return {"out": e, "loss": d.square().mean(), "grad": grad[0]}
    if kind == "measure":
        psi = _random_state(case["n"], seed, case["precision"]).to(torch.complex128).view(1, -1)
        return {"expectations": torch.cat([_inner(psi, _pauli(psi, p, pos))[0] for p, pos in
                                           pauli_strings(case["n"])]), "shots": None}
    return {"samples": None, "expectations": _exact_noise(case, seed)}
