"""CPU test of the keys under which loaded sweep kernels are found: sweeps
with the same key must have the same generated source, over circuits of all
gate kinds, widths and precisions, and over angles and tile placements."""
import ctypes
from ctypes import POINTER as P

import numpy as np

from dgquest_b200 import circuits as C
from dgquest_b200 import ir
from dgquest_b200 import quest as Q

NO_SWAP = [C.H, C.X, C.Y, C.Z, C.S, C.T, C.RX, C.RY, C.RZ, C.PHASE, C.CNOT, C.CZ, C.CPHASE, C.CRX, C.CRY, C.CRZ,
           C.COMPACT, C.CCOMPACT, C.UNITARY, C.CUNITARY, C.SQX, C.SQY, C.SQW, C.CY]


def keyed_sources(ops, n, w, precision):
    t, tm, cm, o = ir.ops_to_ir(ops, n)
    buf = ctypes.create_string_buffer(1 << 20)
    key = ctypes.c_uint64(0)
    args = (n, w, len(t), t.ctypes.data_as(P(ctypes.c_int32)), tm.ctypes.data_as(P(ctypes.c_uint64)),
            cm.ctypes.data_as(P(ctypes.c_uint64)), o.ctypes.data_as(P(ctypes.c_double)))
    count = Q.dgq_sweepSource(*args, 0, precision, buf, len(buf))
    for s in range(count):
        Q.dgq_sweepSourceKey(*args, s, precision, buf, len(buf), ctypes.byref(key))
        yield key.value, buf.value


def test_equal_keys_mean_equal_sources():
    seen, hits = {}, 0
    for w, precision in [(9, 2), (12, 2), (13, 1), (11, 1), (12, 3)]:
        for n in (14, 17, 20):
            for seed in range(4):
                lists = [C.random_layers(n, 3, seed), C.hea(n, 3, seed), C.ghz_qft(n, swaps=False),
                         C.grid_sqrt(2, n // 2, 4, seed), C.mixed_ops(n, 60, seed, kinds=NO_SWAP)]
                for ops in lists:
                    for key, source in keyed_sources(ops, n, w, precision):
                        hits += key in seen
                        assert seen.setdefault(key, source) == source
    # other angles, and other sizes with the same tile structure, share keys
    assert hits > 50 and len(np.unique([hash(s) for s in seen.values()])) > 50
