"""Unitaries and channels of 2..4 targets in specialised sweeps
(csrc/jit_prelude.cuh jDenseAt): any register bits, in phases shared with
other gates, the zero entries of channels left out; one kernel for all
matrices on the same targets.

Bound: an amplitude is a sum of at most 2 x 16 products per gate; 1e-12 over
the 40 gates of a circuit, as for every gate of the register phases. In
complex64 each gate rounds its 32 products and sums once, 32 x 2^-24 of an
amplitude bound of 1, and the circuit has 18 such gates and 168 others: a
state error of 18 x 32 x 2^-24 + 168 x 4 x 2^-24 at most."""
import numpy as np
import pytest

import oracle
from dgquest_b200 import circuits as C

pytestmark = pytest.mark.gpu


def matrices(gen, k):
    """Full, diagonal, permutation, block and nearly-identity unitaries."""
    d = 1 << k
    yield C.random_unitary(gen, d)
    yield np.diag(np.exp(1j * gen.uniform(-3, 3, d)))
    yield np.eye(d, dtype=complex)[gen.permutation(d)]
    u = np.eye(d, dtype=complex)
    u[d - 2:, d - 2:] = C.random_unitary(gen, 2)
    yield u
    yield np.kron(C.random_unitary(gen, 2), np.eye(d // 2))
    yield 1j * np.eye(d, dtype=complex)


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("n,width", [(10, 9), (12, 12), (14, 11)])
def test_small_unitaries_match_oracle(quest, env, n, width, single):
    Q = quest
    gen = np.random.default_rng(n)
    o = oracle.Oracle(n)
    bits = Q.dgq_setSpecialisationMinBits(9)
    q = (Q.dgq_createQuregF32 if single else Q.createQureg)(n, env)
    try:
        Q.dgq_setTileBits(q, width)
        Q.dgq_setDenseFusion(q, 0)
        ops = C.mixed_ops(n, 60, n)
        C.replay(q, ops)
        o.apply(ops)
        for k in (2, 3, 4):
            for i, u in enumerate(matrices(gen, k)):
                targs = gen.choice(n, k, replace=False).tolist()
                if single and i % 2 == 0 and 0 not in targs:
                    targs[i % k] = 0  # no paired form: the unpaired complex64 sweep
                m = Q.matrixN(u)
                Q.multiQubitUnitary(q, Q.int_array(targs), k, m)
                Q.destroyComplexMatrixN(m)
                o.multi_qubit_unitary(targs, u)
                ops = C.mixed_ops(n, 6, 100 * k + i)
                C.replay(q, ops)
                o.apply(ops)
        got = Q.state_vector(q)
    finally:
        Q.dgq_setSpecialisationMinBits(bits)
        Q.destroyQureg(q, env)
    want = o.amps()
    o.close()
    if single:
        assert np.linalg.norm(got - want) <= (18 * 32 + 168 * 4) * 2.0 ** -24
    else:
        assert np.abs(got - want).max() <= 1e-12


@pytest.mark.parametrize("single", [False, True])
def test_one_kernel_for_every_matrix_on_the_same_targets(quest, env, single):
    # tensor products of random Paulis, permutations, diagonals: other zeros
    # each time, the kernel of the first
    Q, n, targs = quest, 11, [0, 4, 7]
    gen = np.random.default_rng(1)
    bits = Q.dgq_setSpecialisationMinBits(9)
    q = (Q.dgq_createQuregF32 if single else Q.createQureg)(n, env)
    o = oracle.Oracle(n)
    compiled = []
    try:
        Q.dgq_setDenseFusion(q, 0)
        for u in matrices(gen, 3):
            ops = C.mixed_ops(n, 8, 4, kinds=[C.H, C.T, C.CZ, C.CNOT])
            Q.apply_circuit(q, ops)
            o.apply(ops)
            m = Q.matrixN(u)
            Q.multiQubitUnitary(q, Q.int_array(targs), 3, m)
            Q.destroyComplexMatrixN(m)
            o.multi_qubit_unitary(targs, u)
            Q.dgq_planPending(q)
            compiled.append(Q.plan_stats(q).jitCompiled)
            Q.dgq_launchPlanned(q)
        got = Q.state_vector(q)
    finally:
        Q.dgq_setSpecialisationMinBits(bits)
        Q.destroyQureg(q, env)
    want = o.amps()
    o.close()
    # (the first plan also initialises the register)
    assert not any(compiled[2:])
    assert np.linalg.norm(got - want) <= ((6 * 32 + 48 * 4) * 2.0 ** -24 if single else 1e-12)


def test_one_kernel_for_every_probability(quest, env):
    Q, n = quest, 6
    bits = Q.dgq_setSpecialisationMinBits(9)
    q = Q.createDensityQureg(n, env)
    compiled = []
    try:
        # 0 and 1/2 make entries zero that others do not
        for p in (0.2, 0.37, 0.0, 0.5):
            Q.initPlusState(q)
            for t in range(n):
                Q.applyOneQubitDephaseError(q, t, p)
                Q.applyOneQubitDepolariseError(q, t, p)
                Q.applyOneQubitDampingError(q, t, p)
            Q.applyTwoQubitDephaseError(q, 0, 3, p)
            Q.applyTwoQubitDepolariseError(q, 4, 1, p)
            Q.dgq_planPending(q)
            compiled.append(Q.plan_stats(q).jitCompiled)
            Q.dgq_launchPlanned(q)
    finally:
        Q.dgq_setSpecialisationMinBits(bits)
        Q.destroyQureg(q, env)
    assert compiled[0] > 0 and not any(compiled[1:])


def test_channels_equal_the_interpreting_kernel(quest, env):
    Q, n = quest, 6
    rng = np.random.default_rng(6)
    ops = C.mixed_ops(n, 50, 6, kinds=[k for k in range(C.CY + 1) if k != C.MEASURE])
    pairs = [rng.choice(n, 2, replace=False).tolist() for _ in range(4)]

    def run(min_bits):
        bits = Q.dgq_setSpecialisationMinBits(min_bits)
        q = Q.createDensityQureg(n, env)
        try:
            for layer in range(2):
                C.replay(q, ops)
                for t in range(n):
                    Q.applyOneQubitDephaseError(q, t, 0.05)
                    Q.applyOneQubitDepolariseError(q, t, 0.1 * t / n)
                    Q.applyOneQubitDampingError(q, t, 1.0 if t == 3 and layer else 0.2)
                for a, b in pairs:
                    Q.applyTwoQubitDephaseError(q, a, b, 0.1)
                    Q.applyTwoQubitDepolariseError(q, a, b, 0.2)
            return Q.density_matrix(q)
        finally:
            Q.dgq_setSpecialisationMinBits(bits)
            Q.destroyQureg(q, env)

    assert np.abs(run(9) - run(40)).max() <= 1e-13
