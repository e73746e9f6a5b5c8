"""Dense 5..7-qubit sweeps on the FP64 matrix instruction (csrc/dense.cu) at
the edges of its tiles: 4, 8 and 16 columns (fewer than a warp's 16), a full
tile, several tiles; low, high and mixed targets; both state precisions.

Bound: an output is a sum of 2 x 2^K products in FP64, so its error is at
most (2 x 2^K + 2) 2^-53 times the norm of the state (1). complex64 adds the
rounding of the output and of the closing renormalisation's factor."""
import numpy as np
import pytest

from dense_ref import apply_multi
from dgquest_b200 import circuits as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("n,targs", [
    (9, [3, 0, 8, 5, 1]), (9, [0, 1, 2, 3, 4, 5]), (9, [8, 7, 6, 5, 4, 3, 2]), (9, [4, 0, 7, 2, 8, 1, 5]),
    (11, [10, 0, 9, 1, 8, 2, 7]), (12, [11, 3, 7, 0, 5]), (12, [0, 1, 2, 3, 4, 5, 6]), (13, [12, 0, 6, 1, 11, 7]),
    (15, [14, 13, 12, 11, 10, 9, 8]), (15, [2, 1, 0, 14, 13]),
])
def test_dense_sweep_edges(quest, env, n, targs, single):
    Q = quest
    gen = np.random.default_rng(100 * n + len(targs))
    k = len(targs)
    u = C.random_unitary(gen, 1 << k)
    x = gen.standard_normal(1 << n) + 1j * gen.standard_normal(1 << n)
    x /= np.linalg.norm(x)
    if single:
        x = x.astype(np.complex64).astype(np.complex128)
    q = Q.dgq_createQuregF32(n, env) if single else Q.createQureg(n, env)
    tensor = Q.dgq_setTensorCores(0)
    try:
        Q.init_from_amps(q, x)
        m = Q.matrixN(u)
        Q.multiQubitUnitary(q, Q.int_array(targs), k, m)
        Q.destroyComplexMatrixN(m)
        got = Q.state_vector(q)
    finally:
        Q.dgq_setTensorCores(tensor)
        Q.destroyQureg(q, env)
    want = x.copy()
    apply_multi(want, n, targs, u)
    bound = (2 * 2 ** k + 2) * 2.0 ** -53
    if single:
        bound += 4 * 2.0 ** -24 * np.abs(want).max()
    assert np.abs(got - want).max() <= bound


@pytest.mark.parametrize("single", [False, True])
def test_wide_unitaries_keep_the_tile_form(quest, env, single):
    """The gates between wide unitaries are priced as tile sweeps, so one
    layer of rotations is not fused into extra dense sweeps; the chosen plan
    equals the forced tile form."""
    Q, n = quest, 22
    gen = np.random.default_rng(22)
    first = C.random_layers(n, 1, 5)
    wide = [(gen.choice(n, k, replace=False).tolist(), C.random_unitary(gen, 1 << k)) for k in (6, 5, 7, 6)]

    def run(form):
        q = Q.dgq_createQuregF32(n, env) if single else Q.createQureg(n, env)
        Q.dgq_setDenseFusion(q, form)
        C.replay(q, first)
        for targs, u in wide:
            m = Q.matrixN(u)
            Q.multiQubitUnitary(q, Q.int_array(targs), len(targs), m)
            Q.destroyComplexMatrixN(m)
        amps = Q.state_vector(q)
        st = Q.plan_stats(q)
        Q.destroyQureg(q, env)
        return amps, st

    amps, st = run(-1)
    assert st.formAuto == 1 and st.formK == 0 and st.denseBlocks == 0
    assert 0.0 < st.predictedTileMs < 1e3
    want, _ = run(0)
    # the two plans may differ in their tile width: rounding of the first layer only
    assert np.linalg.norm(amps - want) <= (1e-5 if single else 1e-13)
