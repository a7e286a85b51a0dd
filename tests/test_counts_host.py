"""Counting of sampled indices and the packed op records (host only): the
vectorised forms against the per-shot and per-gate ones."""

import numpy as np
import pytest

from pyquafu_gb300 import ir, qfvm, workloads


@pytest.mark.parametrize("measures", [[(0, 0)], [(3, 0), (0, 1), (5, 2)], [(q, 11 - q) for q in range(12)],
                                      [(1, 0), (2, 0), (3, 1)], [(q % 34, q) for q in range(64)]])
def test_counts_match_bitstrings(measures):
    """Same counts in the same (first shot) order as the shots' strings:
    permuted, partial and repeated classical bits, registers beyond 63 bits."""
    idx = np.random.default_rng(len(measures)).integers(0, 1 << 34, 300).astype(np.uint64)
    idx[::3] = idx[0]
    strings = qfvm._count(qfvm._bitstrings(idx, measures))
    assert list(qfvm._count_strings(idx, measures).items()) == list(strings.items())
    assert list(qfvm._count_values(idx, measures).items()) == [(int(s, 2), c) for s, c in strings.items()]


def test_counts_refuse_a_bit_outside_the_string():
    for f in (qfvm._count_values, qfvm._count_strings):
        with pytest.raises(qfvm.QfvmError):
            f(np.zeros(3, np.uint64), [(0, 0), (1, 2)])


def test_pack_records():
    ops = workloads.random_layers(9, 2, seed=1, extras=True, extra_rate=1.0)
    ops.append(workloads.matrix_gate("u2", (2, 4), np.arange(16).reshape(4, 4)))
    ops.append(ir.Op("ry", ir.OP_RY, (3,), 0, (0.25,), slot=7))
    ops.append(ir.Op("id", ir.OP_NOP, (0,)))
    arr, pool = ir.pack(ops)
    gates = [o for o in ops if o.kind != ir.OP_NOP]
    assert len(arr) == len(gates)
    for r, o in zip(arr, gates):
        assert (r["kind"], r["ncontrols"], r["nqubits"], r["slot"], r["gen"]) == (o.kind, o.ncontrols, len(o.qubits),
                                                                                o.slot, o.gen)
        assert tuple(r["qubits"]) == o.qubits + (0,) * (16 - len(o.qubits))
        assert tuple(r["params"]) == o.params + (0.0,) * (4 - len(o.params))
        if o.matrix is None:
            assert r["mat_offset"] == -1 and r["mat_dim"] == 0
        else:
            m = np.asarray(o.matrix, dtype=np.complex128)
            assert r["mat_dim"] == m.shape[0]
            assert np.array_equal(pool[r["mat_offset"]: r["mat_offset"] + m.size], m.ravel())
    with pytest.raises(ValueError):
        ir.pack([ir.Op("x", ir.OP_X, range(17))])


@pytest.mark.parametrize("form", [list, np.array])
def test_pack_takes_fields_set_later(form):
    """A record's qubits and params may have been set to another sequence."""
    op = ir.Op("rzz", ir.OP_RZZ, (0, 1), 0, (0.5,))
    ref, _ = ir.pack([op])
    op.qubits, op.params = form([0, 1]), form([0.5])
    assert np.array_equal(ir.pack([op])[0], ref)
