"""The exchange of address-bit pairs in HBM (csrc/kernels.cu swapBitsKernel):
swapGate relabels and dgq_getDeviceState undoes them, so the buffer then holds
the amplitudes in logical order. Values move and are not computed, so they
must be equal. Sizes: below one run, one tile, several tiles; pairs inside the
run bits, across them, above them, and none of the low bits."""
import numpy as np
import pytest

import oracle
from dgquest_b200 import circuits as C

pytestmark = pytest.mark.gpu


def swaps(n, kind):
    if kind == "reverse":
        return [(i, n - 1 - i) for i in range(n // 2)]
    if kind == "ends":
        return [(0, n - 1)]
    if kind == "high":
        return [(n - 1, n - 2)] + ([(n - 3, n - 5)] if n > 12 else [])
    if kind == "low":
        return [(0, 1), (2, min(4, n - 1))] if n > 2 else [(0, 1)]
    rng = np.random.default_rng(n)
    # overlapping swaps: cycles, which take several passes
    return [tuple(rng.choice(n, 2, replace=False).tolist()) for _ in range(2 * n)]


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("kind", ["reverse", "ends", "high", "low", "random"])
@pytest.mark.parametrize("n", [2, 5, 9, 10, 11, 13, 16, 18])
def test_buffer_in_logical_order(quest, env, n, kind, single):
    import torch
    Q = quest
    b = C.OpList()
    for x, y in swaps(n, kind):
        b.add(C.SWAP, int(x), int(y))
    ops = np.concatenate([C.random_layers(n, 2, n), b.array()])
    q = Q.dgq_createQuregF32(n, env) if single else Q.createQureg(n, env)
    try:
        C.replay(q, ops)
        before = Q.state_vector(q)  # through the map, nothing moved
        address = Q.dgq_getDeviceState(q, None)
        view = type("View", (), {"__cuda_array_interface__": {
            "shape": (1 << n, 2), "strides": None, "version": 2, "typestr": "<f4" if single else "<f8",
            "data": (address, False)}})()
        raw = torch.as_tensor(view, device="cuda").cpu().numpy().astype(np.float64)
    finally:
        Q.destroyQureg(q, env)
    buffer = raw[:, 0] + 1j * raw[:, 1]
    assert np.array_equal(buffer, before)
    assert np.abs(buffer - oracle.run(n, ops)[0]).max() <= (1e-6 if single else 1e-12)
