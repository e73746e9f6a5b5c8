"""Framed sweep programs on the GPU (csrc/frame.h, the interpreting kernels):
every framed gate kind at every tile width in both precisions, with CNOT, CZ
and Pauli gates between rotations on tile, thread and CTA bits, a collapse
between two parts, and batches that are framed or not, against the oracle.

Bound: the same factors as the gate-by-gate product, so 1e-12 per amplitude
in complex128. In complex64 each of G gates rounds its products and sums at
most 4 times, 2^-24 of the state each: 4 G 2^-24 in the 2-norm of the
difference, with no normalisation, so a wrong overall factor shows."""
import numpy as np
import pytest

import oracle
from dgquest_b200 import circuits as C

pytestmark = pytest.mark.gpu

FRAMED = [C.H, C.X, C.Y, C.Z, C.S, C.T, C.RX, C.RY, C.RZ, C.PHASE, C.CNOT, C.CNOT, C.CZ, C.CPHASE, C.CRZ, C.SQX, C.SQY,
          C.SQW, C.COMPACT, C.UNITARY, C.SWAP]


def check(amps, ref, single, gates=0):
    if single:
        assert gates and np.linalg.norm(amps - ref) <= 4 * gates * 2.0 ** -24
    else:
        assert np.abs(amps - ref).max() <= 1e-12


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("n,width", [(2, 9), (5, 9), (9, 9), (10, 9), (13, 9), (12, 10), (13, 11), (12, 12), (15, 12)])
def test_framed_sweeps_match_oracle(quest, env, n, width, single):
    Q = quest
    ops = np.concatenate([C.mixed_ops(n, 250, 31 * n + width, kinds=FRAMED), C.hea(n, 4, n)])
    q = Q.dgq_createQuregF32(n, env) if single else Q.createQureg(n, env)
    try:
        Q.dgq_setTileBits(q, width)
        Q.dgq_setDenseFusion(q, 0)
        C.replay(q, ops)
        amps = Q.state_vector(q)
    finally:
        Q.destroyQureg(q, env)
    check(amps, oracle.run(n, ops)[0], single, len(ops))


def test_collapse_between_framed_sweeps(quest, env):
    Q, n = quest, 14
    b = C.OpList()
    for t in (3, 12):
        b.add(C.MEASURE, t)
    ops = np.concatenate([C.mixed_ops(n, 150, 5, kinds=FRAMED), b.array(), C.mixed_ops(n, 150, 6, kinds=FRAMED)])
    q = Q.createQureg(n, env)
    try:
        Q.seed([77])
        outcomes = C.replay(q, ops)
        amps = Q.state_vector(q)
    finally:
        Q.destroyQureg(q, env)
    ref = oracle.run(n, ops, seed_keys=[77])
    assert list(outcomes) == list(ref[2])
    check(amps, ref[0], False)


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("unframed", [False, True])
def test_batches_with_and_without_a_framed_form(quest, env, unframed, single):
    Q = quest
    sizes = [9, 10, 12, 13, 14]
    lists = [C.mixed_ops(n, 200, 40 + n, kinds=FRAMED) for n in sizes]
    if unframed:
        lists[2] = np.concatenate([lists[2], C.mixed_ops(sizes[2], 5, 9, kinds=[C.CRX])])
    regs = [(Q.dgq_createQuregF32 if single else Q.createQureg)(n, env) for n in sizes]
    try:
        for q, ops in zip(regs, lists):
            C.replay(q, ops)
        b = Q.Batch(regs, config={"tileBits": 12})
        b.launch()
        b.wait()
        states = [Q.state_vector(q) for q in regs]
        b.close()
    finally:
        for q in regs:
            Q.destroyQureg(q, env)
    for n, ops, a in zip(sizes, lists, states):
        check(a, oracle.run(n, ops)[0], single, len(ops))


@pytest.mark.parametrize("unframed", [False, True])
def test_a_phase_longer_than_a_program(quest, env, unframed):
    # 1050 gates on 4 qubits: one register phase, cut into two programs; the
    # same register in a batch
    Q, n = quest, 4
    b = C.OpList()
    for _ in range(150):
        for t in range(n):
            b.add(C.H, t)
        for t in range(n - 1):
            b.add(C.CZ, t, t + 1)
    if unframed:
        b.add(C.CRX, 0, 1, p=(0.3,))
    ops = b.array()
    ref = oracle.run(n, ops)[0]
    for batched in (False, True):
        q = Q.createQureg(n, env)
        try:
            Q.dgq_setTileBits(q, 9)
            Q.dgq_setDenseFusion(q, 0)
            C.replay(q, ops)
            if batched:
                batch = Q.Batch([q], config={"tileBits": 12})
                batch.launch()
                batch.wait()
            amps = Q.state_vector(q)
            if batched:
                batch.close()
        finally:
            Q.destroyQureg(q, env)
        check(amps, ref, False)


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("n,width", [(6, 9), (10, 9), (13, 11), (14, 12)])
def test_phases_on_many_qubits(quest, env, n, width, single):
    # phases and sign flips on 3..6 qubits among rotations and CNOT, by itself
    # and in a batch with a register that has none
    Q, gen = quest, np.random.default_rng(n)
    o = oracle.Oracle(n)
    regs = [(Q.dgq_createQuregF32 if single else Q.createQureg)(n, env) for _ in range(3)]
    try:
        for q in regs:
            Q.dgq_setTileBits(q, width)
            Q.dgq_setDenseFusion(q, 0)
        for r in range(5):
            ops = C.mixed_ops(n, 20, 7 * n + r, kinds=[C.H, C.RX, C.RY, C.RZ, C.CNOT, C.CNOT, C.X, C.UNITARY])
            o.apply(ops)
            for q in regs:
                Q.apply_circuit(q, ops)
            for _ in range(3):
                k = int(gen.integers(3, 7))
                qubits = gen.choice(n, k, replace=False).tolist()
                flip, angle = bool(gen.integers(2)), float(gen.uniform(-3, 3))
                a = o.amps()
                mask = sum(1 << t for t in qubits)
                a[(np.arange(1 << n) & mask) == mask] *= -1 if flip else np.exp(1j * angle)
                o.set_amps(a)
                for q in regs[:2]:
                    if flip:
                        Q.multiControlledPhaseFlip(q, Q.int_array(qubits), k)
                    else:
                        Q.multiControlledPhaseShift(q, Q.int_array(qubits), k, angle)
        want = o.amps()
        o.close()
        gates = 5 * (20 + 3)
        check(Q.state_vector(regs[0]), want, single, gates)
        b = Q.Batch(regs[1:], config={"tileBits": width})
        b.launch()
        b.wait()
        check(Q.state_vector(regs[1]), want, single, gates)
        b.close()
    finally:
        for q in regs:
            Q.destroyQureg(q, env)
