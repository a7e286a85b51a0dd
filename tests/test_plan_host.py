"""The fuser (host planner) checked on CPU: host-built plans are executed by
a numpy interpreter (tests/helpers.py) and compared with the oracle."""

import numpy as np
import pytest

import helpers
import oracle
from pyquafu_gb300 import workloads


SHAPES_C128 = [(11, 4), (12, 4), (12, 5), (12, 3), (11, 3)]
SHAPES_C64 = [(12, 5), (13, 5), (12, 4), (13, 4)]


@pytest.mark.parametrize("T,R", SHAPES_C128)
def test_random_layers_plans(T, R):
    for n in (T, T + 1, T + 3):
        ops = workloads.random_layers(n, 5, seed=100 + n, extras=True, extra_rate=0.6)
        plan = helpers.host_plan(n, ops, 0, T, R)
        got = helpers.interpret(plan, oracle.zero_state(n))
        ref = oracle.simulate(n, ops)
        assert np.abs(got - ref).max() < 1e-13
        # every gate applied once at most (one-qubit merges and merged
        # register-round diagonals fold some)
        applied = sum(int(s["op_count"]) for s in plan["steps"])
        applied += sum(int(p["op_count"]) for p in plan["passes"] if p["type"] != 0)
        assert 0.7 * len(ops) <= applied <= len(ops)


def plan_op_count(plan):
    return sum(int(s["op_count"]) for s in plan["steps"]) + sum(
        int(p["op_count"]) for p in plan["passes"] if p["type"] != 0)


def test_single_qubit_fusion():
    """Commuting one-qubit merges of plain plans: a diagonal passes a gate
    that uses its qubit as a control, RX passes CX on its target, X X
    vanishes; a Hadamard between, or a diagonal on a CX target, blocks."""
    n = 5
    named = workloads.named
    merged = [named("t", (0,)), named("cx", (0, 1), ncontrols=1), named("s", (0,)),          # 1 merge
              named("rx", (2,), (0.3,)), named("cx", (3, 2), ncontrols=1), named("rx", (2,), (1.1,)),  # 1 merge
              named("x", (4,)), named("x", (4,)),                                              # both removed
              named("rz", (3,), (0.7,)), named("cz", (3, 4), ncontrols=1), named("rz", (3,), (0.2,))]  # 1 merge
    blocked = [named("rz", (0,), (0.5,)), named("h", (0,)), named("rz", (0,), (0.4,)),
               named("t", (1,)), named("cx", (0, 1), ncontrols=1), named("t", (1,))]
    for ops, removed in ((merged, 5), (blocked, 0)):
        ops = [named("h", (q,)) for q in range(n)] + ops
        plan = helpers.host_plan(n, ops, 0, 0, 0)
        got = helpers.interpret(plan, oracle.zero_state(n))
        assert np.abs(got - oracle.simulate(n, ops)).max() < 1e-13
        assert plan_op_count(plan) == len(ops) - removed


@pytest.mark.parametrize("T,R", SHAPES_C64)
def test_c64_shapes_plans(T, R):
    n = T + 2
    ops = workloads.random_layers(n, 4, seed=7, extras=True, extra_rate=0.5)
    plan = helpers.host_plan(n, ops, 1, T, R)
    got = helpers.interpret(plan, oracle.zero_state(n))
    assert np.abs(got - oracle.simulate(n, ops)).max() < 1e-13


def test_all_gate_kinds_in_tile_passes(golden):
    meta, states = golden
    case = [c for c in meta["cases"] if c["tag"] == "allgates_n12"][0]
    ops = [helpers.op_from_json(d) for d in case["ops"]]
    plan = helpers.host_plan(12, ops, 0, 11, 4)
    kinds = {int(o["kind"]) for o in plan["ops"]}
    assert helpers.K_DENSE2 in kinds and helpers.K_SWAP in kinds and helpers.K_DIAG in kinds
    got = helpers.interpret(plan, oracle.zero_state(12))
    assert np.abs(got - states["allgates_n12__out"]).max() < 1e-13


def test_dense_k_gate_becomes_global_pass():
    rng = np.random.default_rng(0)
    m = np.linalg.qr(rng.normal(size=(8, 8)) + 1j * rng.normal(size=(8, 8)))[0]
    ops = [workloads.named("h", (q,)) for q in range(13)]
    ops.append(workloads.matrix_gate("u3q", (12, 1, 7), m))
    ops += [workloads.named("rx", (q,), (0.3 * q,)) for q in range(13)]
    plan = helpers.host_plan(13, ops, 0, 12, 4)
    assert 2 in [int(p["type"]) for p in plan["passes"]]
    got = helpers.interpret(plan, oracle.zero_state(13))
    assert np.abs(got - oracle.simulate(13, ops)).max() < 1e-13


def _unitary(k, seed):
    rng = np.random.default_rng(seed)
    d = 1 << k
    return np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))[0]


@pytest.mark.parametrize("n,T", [(10, 11), (15, 12)])
def test_wide_dense_gates_plans(n, T):
    """Dense gates on 7, 8 and 12 targets (the reference applies any count,
    statevector.hpp:945-995): given in any target order, with and without
    controls, in small states (split whole-state passes) and tiled ones."""
    rng = np.random.default_rng(n)
    ops = [workloads.named("h", (q,)) for q in range(n)]
    for k, nc in ((7, 0), (8, 1), (7, 2)):
        qs = [int(q) for q in rng.permutation(n)[: k + nc]]
        ops.append(workloads.matrix_gate(f"u{k}", qs, _unitary(k, k + nc), ncontrols=nc))
        ops += [workloads.named("ry", (q,), (0.1 + 0.2 * q,)) for q in range(n)]
    if n >= 12:
        qs = [int(q) for q in rng.permutation(n)[:12]]
        ops.append(workloads.matrix_gate("u12", qs, _unitary(12, 3)))
    plan = helpers.host_plan(n, ops, 0, T, 4)
    got = helpers.interpret(plan, oracle.zero_state(n))
    assert np.abs(got - oracle.simulate(n, ops)).max() < 1e-12


def test_dense_gate_beyond_twelve_targets_rejected():
    from pyquafu_gb300 import _native as nat

    with pytest.raises(nat.QfvmError, match="at most 12"):
        helpers.host_plan(14, [workloads.matrix_gate("u13", list(range(13)), np.eye(1 << 13))])


def test_wide_dense_gate_in_adjoint_sweep():
    n = 9
    ops, _ = workloads.hea(n, 2, seed=1)
    ops.insert(10, workloads.matrix_gate("u7", [8, 0, 3, 5, 1, 7, 2], _unitary(7, 5)))
    terms = workloads.zz_x_hamiltonian(n, seed=2)
    plan = helpers.host_plan(n, ops, 0, adjoint=True)
    psi = oracle.simulate(n, ops)
    lam = oracle.apply_hamiltonian(psi, terms)
    vals = helpers.interpret2(plan, psi, lam)
    grads = np.zeros(max(o.slot for o in ops) + 1)
    for slot, v in zip(plan["probe_slots"], vals):
        grads[slot] += v
    ref = oracle.grad_adjoint(n, ops, [o.slot for o in ops], terms)
    np.testing.assert_allclose(grads, ref, atol=1e-12)


@pytest.mark.parametrize("R", [3, 4])
def test_round_diagonals_merge(R):
    """Plain plans merge the register-only diagonals of a round into one
    phase table (K_DIAGR, exact quarter turns coded), applied before the
    first op that acts non-diagonally on its bits; the interpreter checks the
    codes against the coefficients and the state against the oracle."""
    n = 14
    rng = np.random.default_rng(R)
    ops = []
    for layer in range(6):
        for q in range(n):
            g = ["s", "t", "z", "rz", "h", "rx", "sdg", "tdg"][int(rng.integers(8))]
            ops.append(workloads.named(g, (q,), (float(rng.uniform(0, 6.3)),) if g in ("rz", "rx") else ()))
        for _ in range(3):
            a, b = (int(x) for x in rng.choice(n, 2, replace=False))
            ops.append(workloads.named(["cz", "rzz", "cp"][layer % 3], (a, b),
                                       (0.7,) if layer % 3 else (), ncontrols=0 if layer % 3 == 1 else 1))
    plan = helpers.host_plan(n, ops, 0, 12, R)
    assert int(np.sum(plan["ops"]["kind"] == helpers.K_DIAGR)) > 0
    got = helpers.interpret(plan, oracle.zero_state(n))
    assert np.abs(got - oracle.simulate(n, ops)).max() < 1e-13
    # batched and adjoint plans keep every gate
    assert int(np.sum(helpers.host_plan(n, ops, 0, adjoint=True)["ops"]["kind"] == helpers.K_DIAGR)) == 0


def test_invalid_ops_rejected():
    from pyquafu_gb300 import _native as nat

    with pytest.raises(nat.QfvmError):
        helpers.host_plan(4, [workloads.named("h", (4,))])
    with pytest.raises(nat.QfvmError):
        helpers.host_plan(4, [workloads.named("cx", (2, 2), ncontrols=1)])
    with pytest.raises(nat.QfvmError):
        helpers.host_plan(4, [workloads.named("h", (0,))], 0, 9, 4)  # shape not compiled in


@pytest.mark.parametrize("n,precision", [(8, 0), (13, 0), (13, 2), (14, 1)])
def test_adjoint_sweep_plan(n, precision):
    """The reverse sweep (probes + inverse gates) planned for the GPU, run by
    the numpy interpreter from (psi, H psi), gives the oracle's gradients."""
    ops, _ = workloads.hea(n, 3, seed=n)
    ops.insert(3, workloads.named("rzz", (0, n - 1), (0.7,)))
    ops[3].slot = max(o.slot for o in ops) + 1
    terms = workloads.zz_x_hamiltonian(n, seed=n) + [(0.4, "YZ", [1, 2])]
    plan = helpers.host_plan(n, ops, precision, adjoint=True)
    psi = oracle.simulate(n, ops)
    lam = oracle.apply_hamiltonian(psi, terms)
    vals = helpers.interpret2(plan, psi, lam)
    nslot = max(o.slot for o in ops) + 1
    got = np.zeros(nslot)
    for v, s in zip(vals, plan["probe_slots"]):
        got[s] += v
    ref = oracle.grad_adjoint(n, [o if o.name != "rzz" else o for o in ops], [o.slot for o in ops], terms)
    # the oracle's grad_gate knows rx/ry/rz; check rzz by finite differences instead
    rzz_slot = ops[3].slot
    mask = np.arange(nslot) != rzz_slot
    np.testing.assert_allclose(got[mask], ref[mask], atol=1e-11)
    h = 1e-6
    ep = oracle.energy(n, [workloads.named("rzz", (0, n - 1), (0.7 + h,)) if o is ops[3] else o for o in ops], terms)
    em = oracle.energy(n, [workloads.named("rzz", (0, n - 1), (0.7 - h,)) if o is ops[3] else o for o in ops], terms)
    assert abs(got[rzz_slot] - (ep - em) / (2 * h)) < 1e-8


def test_unnormalized_hadamards_fold_into_other_gates():
    """Plain plans turn uncontrolled Hadamards into additions and fold their
    1/sqrt(2) factors into other gates' coefficients: same state."""
    from pyquafu_gb300 import ir

    n = 6
    ops = []
    for layer in range(5):
        ops += [workloads.named("h", (q,)) for q in range(n)]
        ops += [ir.Op("ry", ir.OP_RY, (layer % n,), 0, (0.3 + layer,))]
        ops += [workloads.named("cx", (q, q + 1), ncontrols=1) for q in range(n - 1)]
    plan = helpers.host_plan(n, ops)
    kinds = [int(k) for k in plan["ops"]["kind"]]
    assert kinds.count(helpers.K_HAD) == 5 * n
    psi = helpers.interpret(plan, oracle.zero_state(n))
    assert np.max(np.abs(psi - oracle.simulate(n, ops))) < 1e-13
    # no gate to take the factor: the Hadamards stay normalized
    only_h = [workloads.named("h", (q,)) for q in range(n)]
    plan = helpers.host_plan(n, only_h)
    assert helpers.K_HAD not in [int(k) for k in plan["ops"]["kind"]]
    assert np.max(np.abs(helpers.interpret(plan, oracle.zero_state(n)) - oracle.simulate(n, only_h))) < 1e-14


@pytest.mark.parametrize("seed", range(6))
def test_random_commuting_merges(seed):
    """Dense random mixes of diagonals, RX, X, cx, cz, ccx and Hadamards on few
    qubits (many merge opportunities) against the oracle."""
    rng = np.random.default_rng(seed)
    n = 6
    named = workloads.named
    ops = []
    for _ in range(120):
        k = int(rng.integers(9))
        q = int(rng.integers(n))
        if k == 0:
            ops.append(named("rz", (q,), (float(rng.uniform(0, 6.3)),)))
        elif k == 1:
            ops.append(named(["t", "s", "z", "sdg", "tdg"][int(rng.integers(5))], (q,)))
        elif k == 2:
            ops.append(named("rx", (q,), (float(rng.uniform(0, 6.3)),)))
        elif k == 3:
            ops.append(named("x", (q,)))
        elif k == 4:
            a, b = (int(v) for v in rng.choice(n, 2, replace=False))
            ops.append(named("cx", (a, b), ncontrols=1))
        elif k == 5:
            a, b = (int(v) for v in rng.choice(n, 2, replace=False))
            ops.append(named("cz", (a, b), ncontrols=1))
        elif k == 6:
            a, b, c = (int(v) for v in rng.choice(n, 3, replace=False))
            ops.append(named("ccx", (a, b, c), ncontrols=2))
        elif k == 7:
            ops.append(named("h", (q,)))
        else:
            ops.append(named("p", (q,), (float(rng.uniform(0, 6.3)),)))
    plan = helpers.host_plan(n, ops, 0, 0, 0)
    got = helpers.interpret(plan, oracle.zero_state(n))
    assert np.abs(got - oracle.simulate(n, ops)).max() < 1e-12
    assert plan_op_count(plan) < len(ops)


@pytest.mark.parametrize("eb", [16, 8])
def test_tile_layout(eb):
    """The padded tile layout: one-to-one, additive over disjoint bits, runs of
    32 contiguous and 16-byte aligned (bulk-copy units), and each position's
    slot bit as the planner assumes."""
    for T in (6, 11, 12, 13, 14):
        s = np.arange(1 << T)
        off = helpers.tile_off(s, eb)
        assert len(set(off.tolist())) == s.size
        run_start = off[:: 32] * eb
        assert np.all(run_start % 16 == 0)
        assert np.all(np.diff(off.reshape(-1, 32), axis=1) == 1)
        rng = np.random.default_rng(T)
        a = rng.integers(0, 1 << T, 500)
        b = rng.integers(0, 1 << T, 500) & ~a
        assert np.array_equal(helpers.tile_off(a | b, eb), helpers.tile_off(a, eb) + helpers.tile_off(b, eb))
    # slot bits: p < 3 (p < 4) direct, 3..4 (4) none, 5 + j -> j mod 3 (+1)
    direct = 3 if eb == 16 else 4
    for p in range(14):
        want = p if p < direct else (-1 if p < 5 else (p - 5) % 3 + (0 if eb == 16 else 1))
        assert helpers.slot_bit(p, eb, eb) == want, p
        if eb == 8 and p >= 1:
            assert helpers.slot_bit(p, 8, 16) == (p - 1 if p < 4 else (-1 if p == 4 else (p - 5) % 3))


@pytest.mark.parametrize("precision,T,R", [(0, 11, 4), (0, 12, 3), (1, 12, 4), (1, 13, 5)])
def test_round_wavefronts_hit_distinct_banks(precision, T, R):
    """Every register round's first wavefront of lanes (8 lanes of 16-byte
    accesses, 16 of 8-byte ones; 16-byte pairs for complex64 rounds that hold
    position 0 in registers) lands on distinct bank groups of the tile layout
    whenever the round's free positions offer a position for every slot bit."""
    n = 22
    ops = workloads.random_layers(n, 8, seed=5, extras=True)
    plan = helpers.host_plan(n, ops, precision, T, R)
    eb = plan["elem_bytes"]
    rounds = checked = 0
    for pd in plan["passes"]:
        if pd["type"] != 0:
            continue
        for sd in plan["steps"][pd["step_begin"]: pd["step_begin"] + pd["step_count"]]:
            if sd["type"] != 0:
                continue
            rounds += 1
            rpos = [int(x) for x in sd["rpos"][:R]]
            tpos = [int(x) for x in sd["tpos"][: T - R]]
            access = 16 if (eb == 8 and 0 in rpos) else eb
            nslot = 3 if access == 16 else 4
            if {helpers.slot_bit(p, eb, access) for p in tpos} >= set(range(nslot)):
                checked += 1
                lanes = 1 << nslot
                groups = set()
                for lane in range(lanes):
                    s = sum(1 << tpos[k] for k in range(nslot) if (lane >> k) & 1)
                    groups.add((helpers.tile_off(s, eb) * eb // access) % (128 // access))
                assert len(groups) == lanes, (rpos, tpos)
    assert rounds > 0 and checked >= 0.9 * rounds, (checked, rounds)


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_edge_sizes(precision):
    """Smallest states (one and two qubits, a whole-state pass), an empty
    circuit (no passes), the largest supported qubit count (planned only)
    and counts outside the supported range (refused)."""
    from pyquafu_gb300 import _native as nat

    cases = [(1, [workloads.named("h", (0,)), workloads.named("rz", (0,), [0.3])]),
             (2, [workloads.named("h", (0,)), workloads.named("cx", (0, 1), ncontrols=1)]),
             (3, [])]
    for n, ops in cases:
        plan = helpers.host_plan(n, ops, precision)
        assert len(plan["passes"]) == (1 if ops else 0)
        got = helpers.interpret(plan, oracle.zero_state(n))
        assert np.abs(got - oracle.simulate(n, ops)).max() < 1e-15
    plan = helpers.host_plan(nat.QFVM_MAX_QUBITS, [workloads.named("h", (nat.QFVM_MAX_QUBITS - 1,))], precision)
    assert len(plan["passes"]) == 1
    for n in (0, nat.QFVM_MAX_QUBITS + 1):
        with pytest.raises(nat.QfvmError) as err:
            helpers.host_plan(n, [workloads.named("h", (0,))], precision)
        assert "qubit count out of range" in str(err.value)


@pytest.mark.parametrize("precision,T,R", [(0, 11, 4), (2, 12, 3), (1, 13, 5)])
@pytest.mark.parametrize("gates", ["rot", "mixed", "one", "dense"])
@pytest.mark.parametrize("angle", [None, 0.0, np.pi / 2, np.pi, np.pi - 1e-5, -np.pi])
def test_normalized_passes(precision, T, R, gates, angle):
    """Scalars taken out of a pass's rotations and phases go back into one of
    its gates: same state, at random angles and where a rotation's diagonal
    vanishes (left as it is) or nearly does (|c| = 5e-6: unit form with
    off-diagonal entries of 2e5).  At most about 8 gates deep on any
    amplitude's path per layer and 4 layers: rounding stays below 1e-13."""
    from pyquafu_gb300 import ir

    n = T + 2
    rng = np.random.default_rng(T + R)
    ops = []

    def rot(name, q):
        th = float(rng.uniform(0, 2 * np.pi)) if angle is None else angle
        ops.append(ir.Op(name, ir.NAMED_KIND[name], (q,), 0, (th,)))

    for layer in range(1 if gates == "one" else 4):
        if gates == "one":
            rot("ry", n - 1)
            continue
        for q in range(n):
            rot(["ry", "rx"][(q + layer) % 2] if gates != "mixed" else ["ry", "rz", "rx"][(q + layer) % 3], q)
        if gates == "dense":
            z, _ = np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))
            ops.append(workloads.matrix_gate("u", (layer,), z))
            z, _ = np.linalg.qr(rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4)))
            ops.append(workloads.matrix_gate("u2", (layer, n - 2), z))
        ops += [workloads.named("cx", (q, q + 1), ncontrols=1) for q in range(n - 1)]
    plan = helpers.host_plan(n, ops, precision, T, R)
    psi = helpers.random_state(n, 5)
    ref = oracle.simulate(n, ops, psi.copy())
    assert np.abs(helpers.interpret(plan, psi) - ref).max() < 1e-13
    unit = [int(o["special"]) for o in plan["ops"] if int(o["kind"]) in (helpers.K_REAL, helpers.K_RX)]
    full = angle is not None and abs(angle) == np.pi  # |cos| = 6e-17
    assert (sum(unit) == 0) == (full or gates == "one")


@pytest.mark.parametrize("n,precision", [(13, 0), (14, 1), (13, 2)])
def test_normalized_sweep_probes(n, precision):
    """A reverse sweep planned at given angles takes scalars out of its
    passes; its probes are rescaled (gradients against the oracle, angles
    near pi among them)."""
    ops, _ = workloads.hea(n, 2, seed=n)
    for o in ops[::7]:
        if o.slot >= 0:
            o.params = (np.pi - 1e-4 * (1 + o.slot),)
    plan = helpers.host_plan(n, ops, precision, adjoint=True)
    assert len(plan["binds"]) == 0
    # a round applies its thread-bit phases at its end, after its probes: such
    # a phase must not carry the scalars of a pass with probes
    for o in plan["ops"]:
        if int(o["kind"]) == helpers.K_DIAG and int(o["flags"]) & 4 and not int(o["flags"]) & 1:
            d = plan["coef"][int(o["coef"]): int(o["coef"]) + 2]
            assert abs(np.hypot(*d) - 1) < 1e-15
    assert any(int(o["special"]) == 1 for o in plan["ops"] if int(o["kind"]) == helpers.K_REAL)
    terms = workloads.zz_x_hamiltonian(n, seed=n)
    psi = oracle.simulate(n, ops)
    vals = helpers.interpret2(plan, psi, oracle.apply_hamiltonian(psi, terms))
    got = np.zeros(max(o.slot for o in ops) + 1)
    for v, s in zip(vals, plan["probe_slots"]):
        got[s] += v
    ref = oracle.grad_adjoint(n, ops, [o.slot for o in ops], terms)
    np.testing.assert_allclose(got, ref, atol=1e-11)


def _mixed_structure(n, seed):
    """Every gate kind the planner schedules, two-target and wide dense gates
    among them."""
    rng = np.random.default_rng(seed)
    ops = workloads.random_layers(n, 4, seed=seed, extras=True, extra_rate=0.7)
    for k in (2, 3, 7):
        u, _ = np.linalg.qr(rng.normal(size=(1 << k, 1 << k)) + 1j * rng.normal(size=(1 << k, 1 << k)))
        qs = tuple(int(q) for q in rng.choice(n, k, replace=False))
        ops.insert(int(rng.integers(len(ops))), workloads.matrix_gate("u", qs, u))
    return ops


@pytest.mark.parametrize("n,precision,T,R", [(13, 0, 11, 3), (14, 2, 12, 5), (14, 1, 13, 4)])
def test_replanned_structures(n, precision, T, R):
    """The sets found for a structure's passes and rounds are looked up when it
    is planned again: same records, right states, also at other angles and
    after more structures than are kept."""
    circuits = [_mixed_structure(n, seed) for seed in range(3)]
    first = [helpers.host_plan(n, ops, precision, T, R) for ops in circuits]
    other = [op if op.name not in ("rx", "ry") else type(op)(op.name, op.kind, op.qubits, 0, (op.params[0] + 0.1,))
             for op in circuits[0]]
    for q in range(40):  # pushes the first ones out
        helpers.host_plan(n, [workloads.named("h", (q % n,)), workloads.named("x", ((q * 5 + 1) % n,)),
                              workloads.named("h", ((q // n) % n,))], precision, T, R)
    for ops, plan in zip(circuits, first):
        again = helpers.host_plan(n, ops, precision, T, R)  # searched anew, then looked up
        twice = helpers.host_plan(n, ops, precision, T, R)
        for field in ("passes", "steps", "ops", "coef"):
            assert np.array_equal(plan[field], again[field]) and np.array_equal(plan[field], twice[field])
        psi = helpers.random_state(n, 9)
        assert np.abs(helpers.interpret(plan, psi.copy()) - oracle.simulate(n, ops, psi.copy())).max() < 1e-13
    plan = helpers.host_plan(n, other, precision, T, R)
    assert np.array_equal(plan["passes"]["tq"], first[0]["passes"]["tq"])
    psi = helpers.random_state(n, 9)
    assert np.abs(helpers.interpret(plan, psi.copy()) - oracle.simulate(n, other, psi.copy())).max() < 1e-13


def _trained_angles(kind, count, seed):
    """Angles of trained and initialised circuits: all equal, or each 0 or pi
    with a spread."""
    rng = np.random.default_rng(seed)
    if kind.startswith("spread"):
        return rng.integers(0, 2, count) * np.pi + rng.normal(0, float(kind[6:]), count)
    return np.full(count, np.pi - float(kind[4:]) if kind.startswith("eps") else float(kind[5:]))


def _trained_circuit(n, layers, ansatz, kind, seed=0):
    ops, params = workloads.hea(n, layers, seed=seed)
    if ansatz == "ry":
        ops = [o for o in ops if o.name != "rz"]
    rotations = [o for o in ops if o.name in ("ry", "rz")]
    for k, (o, a) in enumerate(zip(rotations, _trained_angles(kind, len(rotations), seed))):
        o.params, o.slot = (float(a),), k
    return ops


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("ansatz,n,layers", [("ry", 13, 4), ("ryrz", 14, 2)])
@pytest.mark.parametrize("kind", ["spread1e-1", "spread1e-3", "equal3.0157", "equal3.1337", "equal3.1403", "eps 3.2e-4",
                                  "eps 1e-6"])
def test_sweep_probes_stay_in_single_precision(monkeypatch, precision, ansatz, n, layers, kind):
    """A reverse sweep's probes meet both states while scalars of its pass are
    out: their products and the probe's coefficient, divided by the square,
    have to stay within FP32's exponents, also for an observable of 1e3 times
    the size and with the low half of a float pair (48 bits below)."""
    ops = _trained_circuit(n, layers, ansatz, kind, seed=n)
    terms = [(1e3 * c, p, q) for c, p, q in workloads.zz_x_hamiltonian(n, seed=n)]
    plan = helpers.host_plan(n, ops, precision, adjoint=True)
    worst = []
    inner = helpers.probe_value

    def probe(psi, lam, xmask, zmask, cmask, ny, scale):
        ix = np.arange(psi.size) ^ xmask
        products = np.abs(psi[ix]) * np.abs(lam)
        high = np.float32(scale)
        pair = float(high) + float(np.float32(scale - float(high)))
        worst.append((products.sum(), abs(pair / scale - 1), abs(scale)))
        return inner(psi, lam, xmask, zmask, cmask, ny, scale)

    monkeypatch.setattr(helpers, "probe_value", probe)
    psi = oracle.simulate(n, ops)
    vals = helpers.interpret2(plan, psi, oracle.apply_hamiltonian(psi, terms))
    products, pair, scale = (max(w[k] for w in worst) for k in range(3))
    # sums of products: |psi| |lam| <= 1e3 * sum |c| < 2^16, taken out: 2^-36 of each state
    assert products < 2.0 ** 88 and scale < 2.0 ** 73
    assert pair < 2.0 ** -46
    got = np.zeros(max(o.slot for o in ops) + 1)
    for v, s in zip(vals, plan["probe_slots"]):
        got[s] += v
    np.testing.assert_allclose(got, oracle.grad_adjoint(n, ops, [o.slot for o in ops], terms), atol=1e-8)


@pytest.mark.parametrize("precision,T,R", [(1, 12, 4), (2, 12, 3)])
def test_hadamards_and_unit_rotations_stay_in_single_precision(monkeypatch, precision, T, R):
    """Hadamards without their 1/sqrt(2) (up to 128 before a gate takes their
    scalar) while rotations near pi are in unit form (2^48 at most)."""
    n, near = 14, np.pi - 2.0 ** -14
    ops = [workloads.named("ry", (q,), (near,)) for q in (0, 1, 2)]
    ops += [workloads.named("h", (q,)) for _ in range(125) for q in (5, 6)]
    ops += [workloads.named("ry", (5,), (0.3,))] + [workloads.named("ry", (q,), (near,)) for q in (0, 1, 2)]
    ops += [workloads.named("ry", (7,), (0.3,))]
    plan = helpers.host_plan(n, ops, precision, T, R)
    largest = [0.0]
    inner = helpers.apply_global

    def apply(psi, *args):
        inner(psi, *args)
        largest[0] = max(largest[0], float(np.abs(psi).max()))

    monkeypatch.setattr(helpers, "apply_global", apply)
    got = helpers.interpret(plan, oracle.zero_state(n))
    assert largest[0] < 2.0 ** 113
    assert np.abs(got - oracle.simulate(n, ops)).max() < 1e-13


def test_unit_rotations_keep_the_norm():
    """The scalars of unit rotations go back as one product: what the plan's
    rotations do to the norm is no further from 1 than what the gates do
    rounded one by one (rms of 12 circuits, in long double)."""
    n, plans, gates = 12, [], []
    for seed in range(12):
        rng = np.random.default_rng(seed)
        ops = []
        for _ in range(30):
            ops += [workloads.named(["ry", "rx"][int(rng.integers(2))], (q,), (float(rng.uniform(0, 2 * np.pi)),))
                    for q in range(n)]
            ops += [workloads.named("cx", rng.choice(n, 2, replace=False), ncontrols=1) for _ in range(4)]
        half = np.array([o.params[0] / 2 for o in ops if o.params])
        c, s = np.cos(half).astype(np.longdouble), np.sin(half).astype(np.longdouble)
        gates.append(np.log(c * c + s * s).sum())
        plan = helpers.host_plan(n, ops, 0, 11, 4)
        drift = np.longdouble(0)
        for o in plan["ops"]:
            m = plan["coef"][int(o["coef"]): int(o["coef"]) + 4].astype(np.longdouble)
            if int(o["kind"]) == helpers.K_REAL:
                drift += np.log(m[0] * m[3] - m[1] * m[2])
            elif int(o["kind"]) == helpers.K_RX:
                drift += np.log(m[0] * m[0] + m[1] * m[1])
        plans.append(drift)
    assert np.sqrt(np.mean(np.square(plans))) <= np.sqrt(np.mean(np.square(gates)))


@pytest.mark.parametrize("seed", [41, 42])
def test_plans_do_not_depend_on_earlier_ones(seed):
    """The sets kept for a structure are those of one amplitude size: complex64
    and complex128 plans of one shape, in either order, and alone."""
    n, first = 16, {}
    for order in ((0, 1), (1, 0)):
        ops = workloads.random_layers(n, 12, seed=seed, extras=True)
        for k in range(order[0] * 40):  # pushes the kept sets of the first order out
            helpers.host_plan(n, [workloads.named("h", (q,)) for q in range(1 + k % 8)] +
                              [workloads.named("x", (k // 8,)), workloads.named("h", (k // 8,))], 0, 12, 4)
        for precision in order:
            plan = helpers.host_plan(n, ops, precision, 12, 4)
            ref = first.setdefault(precision, plan)
            for field in ("passes", "steps", "ops"):
                assert np.array_equal(plan[field], ref[field]), (order, precision, field)


def test_kept_sets_are_bounded_in_bytes():
    """Structures of 100 K gates each (3.7 MB of key): what stays on the heap
    after planning ten of them is below the 16 MiB that are kept, and a margin."""
    import ctypes

    class Info(ctypes.Structure):
        _fields_ = [(k, ctypes.c_size_t) for k in ("arena", "ordblks", "smblks", "hblks", "hblkhd", "usmblks", "fsmblks",
                                                   "uordblks", "fordblks", "keepcost")]

    libc = ctypes.CDLL(None)
    if not hasattr(libc, "mallinfo2"):
        pytest.skip("no mallinfo2")
    libc.mallinfo2.restype = Info

    def used():
        m = libc.mallinfo2()
        return m.uordblks + m.hblkhd

    def plan(k):
        helpers.host_plan(12, [workloads.named("ry", (q % 12,), (0.3,)) for q in range(k, k + 12)] * 8400 +
                          [workloads.named("h", (k,))], 0, 11, 4)

    plan(0)
    before = used()
    for k in range(1, 11):
        plan(k)
    assert used() - before < 20 << 20


@pytest.mark.parametrize("n,shots", [(12, 4096), (24, 10), (29, 1), (29, 3), (30, 1), (30, 100)])
def test_trajectory_memory(n, shots):
    """What a trajectory run holds: half of the free memory where more than one
    shot fits with the state that they start from, that state only where it
    fits and is used more than once, and never more than one shot's where that
    is all there is room for."""
    import ctypes

    from pyquafu_gb300 import _native as nat

    state, item = 16 << n, (16 << n) + 5000
    for free in (item + 1000, 2 * state + 4000, 2 * item + (65 << 20), 4 * item, 284 << 30):
        chunk, shared = ctypes.c_int64(), np.zeros(1, np.int32)
        nat.check(nat.load().qfvm_host_items_memory(free, n, item, shots, ctypes.byref(chunk), nat.i32ptr(shared)))
        held = chunk.value * item + int(shared[0]) * state
        assert 1 <= chunk.value <= shots
        assert held <= (free if chunk.value == 1 else free // 2)
        assert held == item or shots > 1
        if free == 284 << 30:
            assert shared[0] == (shots > 1)
            assert chunk.value == shots or held + item > free // 2


@pytest.mark.parametrize("precision,T,one,two", [(0, 11, 1, 6), (1, 13, 3, 4), (2, 12, 1, 5)])
def test_small_states_have_few_passes(precision, T, one, two):
    """A pass of a small state costs its latency, whatever it holds: a state of
    one tile is one pass (complex64: for every 128 operations of its 380), and one
    of two tiles takes no more than the first-need order alone needs (20 layers)."""
    for n, most in ((T, one), (T + 1, two)):
        plan = helpers.host_plan(n, workloads.random_layers(n, 20, seed=3), precision)
        assert plan["T"] == T and len(plan["passes"]) <= most
