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
