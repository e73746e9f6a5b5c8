"""Specialised sweeps move diagonal gates between the phases of a sweep and
into the next sweep (csrc/planner.cpp placeDiagonals): circuits whose
diagonal gates meet Rx, Ry, H, CNOT, dense and controlled gates on the same
qubits, in both precisions and several tile widths, against the oracle; and
phases that collect more gates than one program holds.

Bound: the moved gates are the same factors in another order, so the
register-phase tolerances hold: 1e-12 per amplitude, fidelity 1 - 1e-6."""
import numpy as np
import pytest

import oracle
from dgquest_b200 import circuits as C

pytestmark = pytest.mark.gpu


def diagonal_mix(n, count, seed):
    kinds = [C.RX, C.RY, C.H, C.CNOT, C.CRX, C.UNITARY, C.RZ, C.RZ, C.Z, C.S, C.T, C.PHASE, C.CZ, C.CZ, C.CPHASE,
             C.CPHASE, C.CRZ, C.SWAP]
    return C.mixed_ops(n, count, seed, kinds=kinds)


@pytest.mark.parametrize("n,width,single", [
    (12, 9, False), (12, 12, False), (13, 10, False), (15, 11, False), (16, 0, False), (12, 0, True), (13, 10, True),
    (16, 0, True),
])
def test_moved_diagonals_match_oracle(quest, env, n, width, single):
    Q = quest
    circuits = [diagonal_mix(n, 300, 17 * n + width), C.random_layers(n, 6, n), C.ghz_qft(n), C.hea(n, 3, n)]
    ops = np.concatenate(circuits)
    bits = Q.dgq_setSpecialisationMinBits(9)
    q = Q.dgq_createQuregF32(n, env) if single else Q.createQureg(n, env)
    try:
        Q.dgq_setTileBits(q, width)
        Q.dgq_setDenseFusion(q, 0)
        C.replay(q, ops)
        amps, st = Q.state_vector(q), Q.plan_stats(q)
        assert st.jitCompiled + st.jitReused > 0 and st.phases > 1
    finally:
        Q.dgq_setSpecialisationMinBits(bits)
        Q.destroyQureg(q, env)
    ref = oracle.run(n, ops)[0]
    if single:
        assert abs(np.vdot(ref, amps)) ** 2 / np.vdot(amps, amps).real >= 1 - 1e-6
    else:
        assert np.abs(amps - ref).max() <= 1e-12


def test_more_diagonals_than_a_program_holds(quest, env):
    """900 distinct controlled phases between two layers: more than one
    program's ops and coefficients."""
    Q, n = quest, 16
    rng = np.random.default_rng(3)
    b = C.OpList()
    for q in range(n):
        b.add(C.H, q)
    pairs = [(i, j) for i in range(n) for j in range(i)]
    for k in range(900):
        i, j = pairs[k % len(pairs)]
        # a T between repeats of a pair keeps the planner from merging them
        b.add(C.CPHASE, i, j, p=(rng.uniform(-3, 3),))
        if k % len(pairs) == 0:
            for q in range(n):
                b.add(C.PHASE, q, p=(rng.uniform(-3, 3),))
    for q in range(n):
        b.add(C.RX, q, p=(rng.uniform(-3, 3),))
    ops = b.array()
    bits = Q.dgq_setSpecialisationMinBits(9)
    q = Q.createQureg(n, env)
    try:
        Q.dgq_setDenseFusion(q, 0)
        C.replay(q, ops)
        amps = Q.state_vector(q)
    finally:
        Q.dgq_setSpecialisationMinBits(bits)
        Q.destroyQureg(q, env)
    assert np.abs(amps - oracle.run(n, ops)[0]).max() <= 1e-12
