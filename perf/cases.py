"""The performance cases of this library: what its users have it do.

A pass is a whole call sequence through the public API (`dgquest_b200.quest`):
initialise a register, record a circuit, run it, read P(q = 0) of every qubit
and hand out the final state in device memory. Cases name a workload of
`dgquest_b200.circuits` (or dense unitaries, a noisy density matrix, a batch)
with its qubit count, depth and precision; the circuit's random choices
(gates, angles, targets, hidden strings, matrices) come from the seed.
"""
import math
import random

import numpy as np
import torch

from dgquest_b200 import circuits as C
from dgquest_b200 import quest as Q

# ------------------------------------------------------------------ the cases
_LISTED = [
    # one step of a small variational loop: host work and launches count
    {"name": "ansatz_n10_c128", "kind": "circuit", "form": "ansatz", "n": 10, "depth": 4, "single": False},
    # Fourier transform of a mid-size register, which stays in L2
    {"name": "ghz_qft_n21_c128", "kind": "circuit", "form": "ghz_qft", "n": 21, "depth": 1, "single": False},
    # a variational step on a complex64 register of odd width
    {"name": "ansatz_n23_c64", "kind": "circuit", "form": "ansatz", "n": 23, "depth": 8, "single": True},
    # random circuit sampling: the circuit, then 1024 shots
    {"name": "random_n25_shots_c128", "kind": "circuit", "form": "random", "n": 25, "depth": 20, "single": False,
     "shots": 1024},
    # the headline circuit at its full size
    {"name": "random_n30_c128", "kind": "circuit", "form": "random", "n": 30, "depth": 20, "single": False},
    # the same in the single-precision form, at an odd width
    {"name": "random_n29_c64", "kind": "circuit", "form": "random", "n": 29, "depth": 20, "single": True},
    # square-root gates on a grid with CZ patterns
    {"name": "grid_4x7_c128", "kind": "circuit", "form": "grid", "n": 28, "rows": 4, "depth": 16, "single": False},
    # Bernstein-Vazirani, the hidden bits measured one after the other
    {"name": "bv_measure_n27_c128", "kind": "circuit", "form": "bv", "n": 27, "depth": 1, "single": False},
    # dense unitaries on 6 qubits, in both precisions
    {"name": "dense6_n26_c128", "kind": "dense", "n": 26, "k": 6, "blocks": 4, "single": False},
    {"name": "dense6_n29_c64", "kind": "dense", "n": 29, "k": 6, "blocks": 4, "single": True},
    # a noisy circuit on a density matrix (2^24 elements)
    {"name": "density_n12", "kind": "density", "n": 12, "depth": 2, "single": False},
    # many small ansatz registers in one launch
    {"name": "batch48_c128", "kind": "batch", "count": 48, "low": 10, "high": 20, "sizes": 4, "single": False},
]


def listed():
    return [dict(c) for c in _LISTED]


def draw(rng):
    what = rng.choice(["circuit"] * 6 + ["dense"] * 2 + ["density", "batch"])
    single = rng.random() < 0.4
    if what == "circuit":
        form = rng.choice(["ansatz", "random", "random", "ghz_qft", "grid", "bv"])
        n = rng.randint(10, 29)
        case = {"kind": "circuit", "form": form, "n": n, "depth": rng.randint(2, 20), "single": single}
        if form in ("ghz_qft", "bv"):
            case["depth"] = 1
        if form == "grid":
            case["rows"] = rng.choice([r for r in (2, 3, 4, 5) if n // r >= 2])
            case["n"] = case["rows"] * (n // case["rows"])
        # shots are drawn from sums of all probabilities: reproducible in 64 bits
        if form in ("ansatz", "random") and not single and rng.random() < 0.4:
            case["shots"] = int(2 ** rng.uniform(4, 12))
        return case
    if what == "dense":
        k = rng.choice([5, 6, 7])
        # a case costs 2^(n + k) or so: up to 2^27 amplitudes in double precision
        n = rng.randint(14, 29 if single else 33 - k)
        return {"kind": "dense", "n": n, "k": k, "blocks": rng.randint(1, 4), "single": single}
    if what == "density":
        return {"kind": "density", "n": rng.randint(6, 13), "depth": rng.randint(1, 3), "single": False}
    low = rng.randint(10, 14)
    return {"kind": "batch", "count": rng.randint(8, 60), "low": low, "high": rng.randint(low, 20),
            "sizes": rng.randint(0, 1 << 20), "single": single}


# ------------------------------------------------------------------ the inputs
def _ops(case, seed):
    """The circuit of a "circuit" case as an op list."""
    n, form = case["n"], case["form"]
    if form == "ansatz":
        return C.hea(n, case["depth"], seed)
    if form == "random":
        return C.random_layers(n, case["depth"], seed)
    if form == "grid":
        return C.grid_sqrt(case["rows"], n // case["rows"], case["depth"], seed)
    if form == "ghz_qft":
        rng = random.Random(seed)
        first = C.OpList()
        for q in range(n):
            first.add(C.RY, q, p=(2.0 * math.pi * rng.random(),))
        return np.concatenate([first.array(), C.ghz_qft(n)])
    measures = C.OpList()
    for q in range(n - 1):
        measures.add(C.MEASURE, q)
    return np.concatenate([C.bernstein_vazirani(n, seed, measure=False), measures.array()])


def _dense_inputs(case, seed):
    """First layer, and per block the targets and the unitary."""
    rng = np.random.default_rng(seed)
    first = C.random_layers(case["n"], 1, seed & 0xFFFFFFFF)
    return first, [(rng.choice(case["n"], case["k"], replace=False).tolist(), C.random_unitary(rng, 1 << case["k"]))
                   for _ in range(case["blocks"])]


def _density_inputs(case, seed):
    """Per layer: an ansatz layer, then one channel per qubit and one two-qubit channel."""
    rng = random.Random(seed)
    n, layers = case["n"], []
    for d in range(case["depth"]):
        noise = [(rng.choice(["dephase", "depolarise", "damping"]), (q,), rng.uniform(0.01, 0.1)) for q in range(n)]
        noise.append((rng.choice(["dephase2", "depolarise2"]), tuple(rng.sample(range(n), 2)), rng.uniform(0.01, 0.1)))
        layers.append((C.hea(n, 1, (seed + d) & 0xFFFFFFFF), noise))
    return layers


def _batch_inputs(case, seed):
    """Per register its qubits and its ansatz; sizes belong to the case, angles to the seed."""
    rng = random.Random(case["sizes"])
    out = []
    for i in range(case["count"]):
        n, depth = rng.randint(case["low"], case["high"]), rng.randint(4, 32)
        out.append((n, C.hea(n, depth, (seed + 1009 * i) & 0xFFFFFFFF)))
    return out


_env = None


class Register:
    """A register, destroyed with its last user, and its state as a device array (2^n x 2 reals)."""

    def __init__(self, n, single, density=False):
        global _env
        if _env is None:
            _env = Q.createQuESTEnv()
        make = Q.createDensityQureg if density else Q.dgq_createQuregF32 if single else Q.createQureg
        self.q = make(n, _env)
        self.address = Q.dgq_getDeviceState(self.q, None)
        self.__cuda_array_interface__ = {"shape": (1 << (2 * n if density else n), 2), "strides": None, "version": 2,
                                         "typestr": "<f4" if single else "<f8", "data": (self.address, False)}

    def __del__(self):
        Q.destroyQureg(self.q, _env)


def _view(register):
    return torch.as_tensor(register, device="cuda")


class Plan:
    """A batch plan, destroyed before its registers."""

    def __init__(self, registers):
        self.registers = registers
        self.batch = Q.Batch([r.q for r in registers])

    def __del__(self):
        if hasattr(self, "batch"):
            self.batch.close()


_CHANNELS = {"dephase": "applyOneQubitDephaseError", "depolarise": "applyOneQubitDepolariseError",
             "damping": "applyOneQubitDampingError", "dephase2": "applyTwoQubitDephaseError",
             "depolarise2": "applyTwoQubitDepolariseError"}


def prepare(case, seed):
    torch.cuda.init()
    if case["kind"] == "batch":
        registers = []
        for n, ops in _batch_inputs(case, seed):
            r = Register(n, case["single"])
            Q.initZeroState(r.q)
            Q.apply_circuit(r.q, ops)
            registers.append(r)
        return {"case": case, "plan": Plan(registers), "views": [_view(r) for r in registers]}
    r = Register(case["n"], case["single"], case["kind"] == "density")
    state = {"case": case, "register": r, "view": _view(r), "seed": seed}
    if case["kind"] == "circuit":
        state["ops"] = _ops(case, seed)
    elif case["kind"] == "dense":
        state["first"], blocks = _dense_inputs(case, seed)
        state["blocks"] = [(Q.int_array(t), Q.matrixN(u)) for t, u in blocks]
    else:
        state["layers"] = _density_inputs(case, seed)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        batch = state["plan"].batch
        batch.launch()
        z = batch.expectation_z()
        for r in state["plan"].registers:
            assert Q.dgq_getDeviceState(r.q, None) == r.address
        return {"z": z, "states": state["views"]}
    r, out = state["register"], {}
    Q.initZeroState(r.q)
    if case["kind"] == "circuit":
        if case["form"] == "bv":
            Q.seed([state["seed"] & 0xFFFFFFFF])
            out["outcomes"] = np.array(Q.apply_circuit(r.q, state["ops"]), dtype=np.int64)
        else:
            Q.apply_circuit(r.q, state["ops"])
    elif case["kind"] == "dense":
        Q.apply_circuit(r.q, state["first"])
        for targets, matrix in state["blocks"]:
            Q.multiQubitUnitary(r.q, targets, case["k"], matrix)
    else:
        for ops, noise in state["layers"]:
            Q.apply_circuit(r.q, ops)
            for channel, qubits, prob in noise:
                getattr(Q, _CHANNELS[channel])(r.q, *qubits, prob)
    out["p0"] = Q.prob_all_zero(r.q)
    if case.get("shots"):
        out["shots"] = Q.sample(r.q, case["shots"], state["seed"]).astype(np.int64)
    assert Q.dgq_getDeviceState(r.q, None) == r.address
    out["state"] = state["view"]
    return out


# ------------------------------------------------------------------ what a pass cannot do without
_FLOPS = {C.H: 4, C.RX: 4, C.RY: 4, C.RZ: 3, C.SQX: 4, C.SQY: 4, C.SQW: 8, C.CPHASE: 1.5}


def _flops(ops, n):
    return sum(_FLOPS.get(int(k), 0) for k in ops["kind"]) * 2.0 ** n


def work(case):
    """The state written once (and read once by shots); the gates' own arithmetic."""
    size = 8 if case["single"] else 16
    if case["kind"] == "batch":
        regs = _batch_inputs(case, 1)
        return {"bytes": sum(size * 2.0 ** n for n, _ in regs), "flops": sum(_flops(ops, n) for n, ops in regs)}
    n = case["n"]
    if case["kind"] == "density":
        layers = _density_inputs(case, 1)
        flops = sum(2 * _flops(ops, 2 * n) + len(noise) * 2.0 ** (2 * n) * 8 * 4 for ops, noise in layers)
        return {"bytes": size * 4.0 ** n, "flops": flops}
    if case["kind"] == "dense":
        return {"bytes": size * 2.0 ** n, "flops": case["blocks"] * 8.0 * 2 ** case["k"] * 2.0 ** n}
    ops = _ops(case, 1)
    return {"bytes": size * 2.0 ** n * (2 if case.get("shots") else 1), "flops": _flops(ops, n)}


def tolerance(case):
    """About four times the largest error against 64-bit sums (complex64) or between two orders of them."""
    if case["single"]:
        return {"rel": 3.5e-6}
    return {"rel": 5e-14}


# ------------------------------------------------------------------ the same in plain torch, 64 bits
_R2 = 1.0 / math.sqrt(2.0)
_FIXED = {C.H: [[_R2, _R2], [_R2, -_R2]], C.X: [[0, 1], [1, 0]], C.SQX: [[_R2, -1j * _R2], [-1j * _R2, _R2]],
          C.SQY: [[_R2, -_R2], [_R2, _R2]], C.SQW: [[_R2, -0.5 - 0.5j], [0.5 - 0.5j, _R2]]}


def _matrix(kind, t):
    c, s = math.cos(t / 2), math.sin(t / 2)
    if kind == C.RX:
        return [[c, -1j * s], [-1j * s, c]]
    if kind == C.RY:
        return [[c, -s], [s, c]]
    if kind == C.RZ:
        return [[c - 1j * s, 0], [0, c + 1j * s]]
    return _FIXED[kind]


def _one(x, q, u):
    v = x.view(-1, 2, 1 << q)
    a, b = v[:, 0].clone(), v[:, 1].clone()
    for r in (0, 1):
        v[:, r] = a * u[r][0]
        v[:, r] += b * u[r][1]


def _two(x, a, b):
    """x by the bits a and b: element (i, j) of the answer has a = i and b = j."""
    hi, lo = max(a, b), min(a, b)
    v = x.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
    return lambda i, j: v[:, i, :, j] if hi == a else v[:, j, :, i]


def _apply(x, ops):
    for rec in ops:
        kind, a, b, t = int(rec["kind"]), int(rec["q0"]), int(rec["q1"]), float(rec["p"][0])
        if kind in (C.CZ, C.CPHASE):
            _two(x, a, b)(1, 1).mul_(-1 if kind == C.CZ else complex(math.cos(t), math.sin(t)))
        elif kind in (C.CNOT, C.SWAP):
            at = _two(x, a, b)
            v, w = (at(1, 0), at(1, 1)) if kind == C.CNOT else (at(0, 1), at(1, 0))
            kept = v.clone()
            v.copy_(w)
            w.copy_(kept)
        elif kind != C.MEASURE:
            _one(x, a, _matrix(kind, t))


def _many(x, bits, u):
    """A dense matrix on several bits, bits[0] the lowest of its index."""
    order = sorted(bits, reverse=True)
    shape, above = [], x.numel().bit_length() - 1
    for b in order:
        shape += [1 << (above - b - 1), 2]
        above = b
    shape.append(1 << above)
    v = x.view(shape)
    axes = [2 * order.index(b) + 1 for b in reversed(bits)]
    rest = [d for d in range(len(shape)) if d not in axes]
    moved = v.permute(axes + rest)
    y = torch.as_tensor(u, device=x.device) @ moved.reshape(1 << len(bits), -1)
    moved.copy_(y.view(moved.shape))


def _zero_state(bits):
    x = torch.zeros(1 << bits, dtype=torch.complex128, device="cuda")
    x[0] = 1.0
    return x


def _p0(p, n):
    return np.array([float(p.view(-1, 2, 1 << q)[:, 0].sum()) for q in range(n)])


def _channel(name, qubits, prob, n):
    """The channel's matrix on the row and column bits of its qubits."""
    pauli = [np.eye(2), np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.diag([1.0, -1.0])]
    if name == "damping":
        kraus = [np.diag([1.0, math.sqrt(1 - prob)]), np.array([[0, math.sqrt(prob)], [0, 0]])]
    elif len(qubits) == 1:
        kinds = (3,) if name == "dephase" else (1, 2, 3)
        kraus = [math.sqrt(1 - prob) * pauli[0]] + [math.sqrt(prob / len(kinds)) * pauli[i] for i in kinds]
    else:
        kinds = [(i, j) for i in range(4) for j in range(4) if i + j > 0 and (name != "dephase2" or i % 3 + j % 3 == 0)]
        kraus = [math.sqrt(1 - prob) * np.eye(4)]
        kraus += [math.sqrt(prob / len(kinds)) * np.kron(pauli[j], pauli[i]) for i, j in kinds]
    # index: row bits low, column bits high
    return [*qubits, *(q + n for q in qubits)], sum(np.kron(k.conj(), k) for k in kraus).astype(complex)


def _shots(p, case, seed):
    """The smallest index whose cumulative probability exceeds u times the total."""
    # the documented draws: MT19937 seeded with init_genrand, 53 bits each
    u = np.random.RandomState(seed & 0xFFFFFFFF).random_sample(case["shots"])
    sums = torch.cumsum(p, 0)
    want = torch.as_tensor(u, device=p.device) * sums[-1]
    return torch.searchsorted(sums, want, right=True).cpu().numpy()


def _real(x):
    return torch.view_as_real(x)


def exact(case, seed):
    if case["kind"] == "batch":
        z, states = [], []
        for n, ops in _batch_inputs(case, seed):
            x = _zero_state(n)
            _apply(x, ops)
            z.append(2.0 * _p0(x.abs() ** 2, n) - 1.0)
            states.append(_real(x))
        return {"z": np.concatenate(z), "states": states}
    n = case["n"]
    if case["kind"] == "density":
        x = _zero_state(2 * n)
        for ops, noise in _density_inputs(case, seed):
            # U rho U^dagger: the circuit on the row bits, its conjugate on the column bits
            _apply(x, ops)
            x = x.conj().resolve_conj()
            moved = ops.copy()
            moved["q0"] += n
            moved["q1"] += n
            _apply(x, moved)
            x = x.conj().resolve_conj()
            for channel, qubits, prob in noise:
                _many(x, *_channel(channel, qubits, prob, n))
        return {"p0": _p0(x.view(1 << n, 1 << n).diagonal().real.contiguous(), n), "state": _real(x)}
    if n > 28:
        return None
    x, out = _zero_state(n), {}
    if case["kind"] == "dense":
        first, blocks = _dense_inputs(case, seed)
        _apply(x, first)
        for targets, u in blocks:
            _many(x, targets, u)
    else:
        _apply(x, _ops(case, seed))
        if case["form"] == "bv":
            out["outcomes"] = np.array(C.bv_secret(n, seed), dtype=np.int64)
    p = x.abs() ** 2
    out["p0"] = _p0(p, n)
    if case.get("shots"):
        out["shots"] = _shots(p, case, seed)
    out["state"] = _real(x)
    return out
