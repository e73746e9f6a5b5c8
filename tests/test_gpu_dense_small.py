"""Unitaries and channels of 2..4 targets in specialised sweeps
(csrc/jit_prelude.cuh jDenseAt): any register bits, in phases shared with
other gates, with zero entries and identity rows left out.

Bound: an amplitude is a sum of at most 2 x 16 products per gate; 1e-12 over
the 40 gates of a circuit, as for every gate of the register phases."""
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


@pytest.mark.parametrize("n,width", [(10, 9), (12, 12), (14, 11)])
def test_small_unitaries_match_oracle(quest, env, n, width):
    Q = quest
    gen = np.random.default_rng(n)
    o = oracle.Oracle(n)
    bits = Q.dgq_setSpecialisationMinBits(9)
    q = Q.createQureg(n, env)
    try:
        Q.dgq_setTileBits(q, width)
        Q.dgq_setDenseFusion(q, 0)
        ops = C.mixed_ops(n, 60, n)
        C.replay(q, ops)
        o.apply(ops)
        for k in (2, 3, 4):
            for i, u in enumerate(matrices(gen, k)):
                targs = gen.choice(n, k, replace=False).tolist()
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
    assert np.abs(got - want).max() <= 1e-12


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
