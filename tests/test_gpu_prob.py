"""The all-qubit probability pass (csrc/kernels.cu probKernel) at the edges of
its shapes: registers narrower than one unit (2^12 loads), one unit, several
CTAs, several units per CTA, with address bit 0 free (16-byte loads of two
complex64 amplitudes) and collapsed.

Bound: a probability is a sum of at most 2^18 non-negative terms added over
at most 16 + 64 + 20 + 4096 / 256 levels in FP64, 2^-53 each (2e-14); a
collapse divides by a probability of at least 0.05."""
import numpy as np
import pytest


pytestmark = pytest.mark.gpu
TOL = 1e-12


def zero_sums(p, n):
    return np.array([p.reshape(-1, 2, 1 << q)[:, 0].sum() for q in range(n)])


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("n,collapse", [
    (1, []), (4, [1]), (9, []), (11, [0]), (12, []), (13, []), (13, [0]), (14, [0, 13]), (17, [3, 0, 9]), (18, []),
    (18, [17]),
])
def test_probabilities_match_numpy(quest, env, n, collapse, single):
    Q = quest
    gen = np.random.default_rng(7 * n + len(collapse))
    x = gen.standard_normal(1 << n) + 1j * gen.standard_normal(1 << n)
    x /= np.linalg.norm(x)
    if single:
        x = x.astype(np.complex64).astype(np.complex128)
    p = np.abs(x) ** 2
    q = Q.dgq_createQuregF32(n, env) if single else Q.createQureg(n, env)
    try:
        Q.init_from_amps(q, x)
        scale = 1.0
        assert np.abs(Q.prob_all_zero(q) - zero_sums(p, n)).max() <= TOL
        for k, b in enumerate(collapse):
            zero = zero_sums(p, n)[b] * scale
            prob = Q.collapseToOutcome(q, b, k % 2)
            assert abs(prob - (1.0 - zero if k % 2 else zero)) <= TOL
            p = p.reshape(-1, 2, 1 << b).copy()
            p[:, 1 - k % 2] = 0.0
            p = p.reshape(-1)
            scale /= prob
            assert np.abs(Q.prob_all_zero(q) - zero_sums(p, n) * scale).max() <= TOL
        assert abs(Q.calcTotalProb(q) - p.sum() * scale) <= TOL
    finally:
        Q.destroyQureg(q, env)
