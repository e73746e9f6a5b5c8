"""complex64 sweeps whose rotations, Hadamards or unitaries leave a long
product of factors to one multiply: the product must stay a normal float
(csrc/planner.h kMaxScalarBitsF32), in every form that runs the sweep.

Bound: each of G gates rounds its two products and a sum once, at most
4 x 2^-24 of the norm, so the state is off by at most 4 G 2^-24 (2-norm); the
scale itself is checked by comparing amplitudes, with no normalisation."""
import ctypes
import math
from ctypes import POINTER as P

import numpy as np
import pytest

import oracle
from dgquest_b200 import circuits as C
from dgquest_b200 import ir
from dgquest_b200 import quest as Quest


def deep(n, layers, kind):
    gen = np.random.default_rng(n + layers)
    b = C.OpList()
    for _ in range(layers):
        for q in range(n):
            if kind == "h":
                b.add(C.H, q)
            else:
                # entries of equal size: the least factor a unitary can leave
                t, p, r = gen.uniform(-math.pi, math.pi, 3)
                u = np.array([[1, np.exp(1j * t)], [-np.exp(1j * p), np.exp(1j * (t + p))]]) * np.exp(1j * r) / math.sqrt(2)
                b.add(C.UNITARY, q, p=np.stack([u.real, u.imag], -1).ravel())
        for q in range(n - 1):
            b.add(C.CZ, q, q + 1)
    return b.array()


# layers such that one sweep's gates would leave less than a float holds
CASES = [(4, 90, "h"), (4, 75, "u"), (10, 60, "h"), (10, 40, "u"), (12, 60, "h")]


@pytest.mark.parametrize("n,layers,kind", CASES)
@pytest.mark.parametrize("precision", [1, 3])
def test_sweeps_end_before_their_scalar_leaves_the_float_range(n, layers, kind, precision):
    ops = deep(n, layers, kind)
    t, tm, cm, o = ir.ops_to_ir(ops, n)
    buf = ctypes.create_string_buffer(1 << 20)
    sweeps = Quest.dgq_sweepSource(n, max(n, 9), len(t), t.ctypes.data_as(P(ctypes.c_int32)),
                                   tm.ctypes.data_as(P(ctypes.c_uint64)), cm.ctypes.data_as(P(ctypes.c_uint64)),
                                   o.ctypes.data_as(P(ctypes.c_double)), 0, precision, buf, len(buf))
    # every gate leaves 2^-1/2, a sweep no less than 2^-80
    assert sweeps >= n * layers * 0.5 / 80.0


def close_to(amps, ref, gates):
    assert np.linalg.norm(amps - ref) <= 4 * gates * 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("specialised", [False, True])
@pytest.mark.parametrize("n,layers,kind", CASES)
def test_deep_complex64_circuits_keep_their_scale(quest, env, n, layers, kind, specialised):
    Q, ops = quest, deep(n, layers, kind)
    bits = Q.dgq_setSpecialisationMinBits(9 if specialised else 40)
    q = Q.dgq_createQuregF32(n, env)
    try:
        Q.dgq_setDenseFusion(q, 0)
        C.replay(q, ops)
        amps = Q.state_vector(q)
    finally:
        Q.dgq_setSpecialisationMinBits(bits)
        Q.destroyQureg(q, env)
    close_to(amps, oracle.run(n, ops)[0], len(ops))


@pytest.mark.gpu
@pytest.mark.parametrize("framed", [True, False])
def test_deep_complex64_batches_keep_their_scale(quest, env, framed):
    Q = quest
    lists = [deep(*case) for case in CASES]
    if not framed:
        # a controlled rotation by nothing: no framed form
        lists[2] = np.concatenate([lists[2], C.OpList().add(C.CRX, 0, 1, p=(0.0,)).array()])
    regs = [Q.dgq_createQuregF32(n, env) for n, _, _ in CASES]
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
    for (n, _, _), ops, amps in zip(CASES, lists, states):
        close_to(amps, oracle.run(n, ops)[0], len(ops))
