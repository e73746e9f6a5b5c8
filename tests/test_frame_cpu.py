"""CPU tests of framed sweep programs: planned for the interpreting kernels
and applied on the host, they must give the oracle's state to 1e-12 per
amplitude (a few hundred operations at 1e-16 each), for every kind of gate
that has a framed form, at every tile width; gates that have none must be
refused."""
import numpy as np
import pytest

import oracle
from dgquest_b200 import circuits as C
from dgquest_b200 import ir

FRAMED = [C.H, C.X, C.Y, C.Z, C.S, C.T, C.RX, C.RY, C.RZ, C.PHASE, C.CNOT, C.CZ, C.CPHASE, C.CRZ, C.SQX, C.SQY, C.SQW,
          C.COMPACT, C.UNITARY]


def framed(n, w, ops):
    t, tm, cm, o = ir.ops_to_ir(ops, n)
    a = np.zeros(1 << n, dtype=np.complex128)
    a[0] = 1.0
    return ir.frame_apply_host(n, w, t, tm, cm, o, a)


@pytest.mark.parametrize("n,w", [(9, 9), (10, 9), (12, 9), (11, 10), (12, 11), (12, 12), (14, 12)])
@pytest.mark.parametrize("kind", ["random", "ghzqft", "hea", "grid", "mixed", "clifford"])
def test_framed_sweeps_match_oracle(n, w, kind):
    seed = 17 * n + w
    ops = {"random": lambda: C.random_layers(n, 8, seed),
           "ghzqft": lambda: C.ghz_qft(n, swaps=False),
           "hea": lambda: C.hea(n, 6, seed),
           "grid": lambda: C.grid_sqrt(2, n // 2, 8, seed),
           # several linear gates between rotations, on all kinds of bits
           "mixed": lambda: C.mixed_ops(n, 300, seed, kinds=FRAMED),
           "clifford": lambda: C.mixed_ops(n, 300, seed, kinds=[C.H, C.X, C.Y, C.Z, C.S, C.CNOT, C.CZ, C.CNOT, C.RX])}[kind]()
    got, sweeps = framed(n, w, ops)
    assert sweeps >= 1
    ref = oracle.run(n, ops)[0]
    assert np.abs(got - ref).max() <= 1e-12
    assert abs(np.vdot(got, got).real - 1.0) <= 1e-12


@pytest.mark.parametrize("kind", [C.CRX, C.CRY, C.CUNITARY, C.CCOMPACT, C.CY])
def test_gates_without_a_framed_form_are_refused(kind):
    ops = np.concatenate([C.hea(10, 1, 3), C.mixed_ops(10, 3, 5, kinds=[kind])])
    got, sweeps = framed(10, 10, ops)
    assert sweeps == 0 and got[0] == 1.0 and not got[1:].any()


def multi_controlled(n, seed, rounds=6):
    """Rotations and CNOT, then phases and sign flips on 3 qubits and more:
    (IR arrays, the oracle's state)."""
    gen = np.random.default_rng(seed)
    o = oracle.Oracle(n)
    parts = []
    for r in range(rounds):
        ops = C.mixed_ops(n, 25, seed + r, kinds=[C.H, C.RX, C.RY, C.RZ, C.CNOT, C.CNOT, C.X, C.UNITARY])
        parts.append(ir.ops_to_ir(ops, n))
        o.apply(ops)
        for _ in range(4):
            qubits = gen.choice(n, gen.integers(3, min(n, 7) + 1), replace=False)
            mask = sum(1 << int(q) for q in qubits)
            kind = [ir.OP_Z, ir.OP_PHASE, ir.OP_S][gen.integers(3)]
            angle = gen.uniform(-3, 3)
            parts.append((np.array([kind], dtype=np.int32), np.array([0], dtype=np.uint64),
                          np.array([mask], dtype=np.uint64), np.array([[angle] + 7 * [0.0]])))
            a = o.amps()
            a[(np.arange(1 << n) & mask) == mask] *= {ir.OP_Z: -1, ir.OP_S: 1j}.get(kind, np.exp(1j * angle))
            o.set_amps(a)
    want = o.amps()
    o.close()
    return [np.concatenate(x) for x in zip(*parts)], want


@pytest.mark.parametrize("n,w", [(9, 9), (12, 9), (11, 10), (13, 11), (12, 12), (14, 12)])
@pytest.mark.parametrize("seed", range(4))
def test_phases_on_many_qubits_are_framed(n, w, seed):
    arrays, want = multi_controlled(n, 100 * n + seed)
    a = np.zeros(1 << n, dtype=np.complex128)
    a[0] = 1.0
    got, sweeps = ir.frame_apply_host(n, w, *arrays, a)
    assert sweeps >= 1
    assert np.abs(got - want).max() <= 1e-12


@pytest.mark.parametrize("entry", [2, 4, 6])
def test_matrices_off_unitarity_beyond_rounding_run_as_given(entry):
    # a general 2x2 is framed as a unitary, so one that is not to rounding
    # (within what the API accepts) has no framed form
    u = C.random_unitary(np.random.default_rng(3), 2).ravel()
    p = np.stack([u.real, u.imag], -1).ravel()
    assert framed(9, 9, C.OpList().add(C.UNITARY, 3, p=p).array())[1] == 1
    p[entry:entry + 2] *= 1 + 1e-14
    assert framed(9, 9, C.OpList().add(C.UNITARY, 3, p=p).array())[1] == 0
