"""The work that users of logosq_b200 have it do, through its public entry points.

Each case names a family and the sizes of one call.  The families are the ways
in which the engine is driven: circuits submitted whole (brickwork, QFT, Trotter
steps, the renormalising dense builders, circuits with noise models), energies of
Pauli sums, parameter-shift gradients of one ansatz and of many at once, shots,
the complex64 form on the tensor cores, and a training step of the warm-start
network.  Sizes are those of the repository's benchmark, configurations and
tests, and the ranges around them.
"""
import ctypes
import math

import numpy as np
import torch

from logosq_b200 import Circuit, EfficientSU2Ansatz, ParameterShift, State, abi, qft
from logosq_b200 import xyz_heisenberg
from logosq_b200._lib import call
from logosq_b200.batch import heisenberg_batch
from logosq_b200.learned import DEPTH, HIDDEN, IN_DIM, LAYERS, OUT_DIM, WarmStartMLP
from logosq_b200.noise import AmplitudeDampingNoise, PhaseDampingNoise


def listed():
    return [
        # the headline circuit (random U3 + CNOT brickwork, 20 layers) at its parity size,
        # a 4 GiB state: the largest call
        {"name": "brickwork_28q", "family": "brickwork", "n": 28, "layers": 20},
        # quantum Fourier transform of a given 20-qubit state (16 MiB, stays in L2)
        {"name": "qft_20q", "family": "qft", "n": 20, "inverse": False},
        # time evolution: Trotter steps of an XYZ chain, an odd width
        {"name": "trotter_19q", "family": "trotter", "n": 19, "steps": 10},
        # a textbook circuit made with the renormalising builders h/x/s/t/rx_matrix
        {"name": "builders_14q", "family": "builders", "n": 14, "gates": 100},
        # the smallest VQE: one gradient of a 4-qubit ansatz (latency and launches)
        {"name": "gradient_4q", "family": "gradient", "n": 4, "depth": 1},
        # one gradient of an ordinary VQE through ParameterShift
        {"name": "gradient_11q", "family": "gradient", "n": 11, "depth": 2},
        # one iteration of the warm-start data set: 256 chains of 12-16 qubits
        {"name": "batch_256_n12_16", "family": "batch", "count": 256, "n_lo": 12, "n_hi": 16},
        # energy of an XYZ chain with field in a given state
        {"name": "energy_24q", "family": "energy", "n": 24, "c64": False},
        # the complex64 form: 5-qubit blocks on the tensor cores
        {"name": "precision_26q", "family": "precision", "n": 26, "layers": 20},
        # sampling a given state
        {"name": "shots_23q", "family": "shots", "n": 23, "shots": 4096},
        # a circuit with damping models after every gate
        {"name": "noise_15q", "family": "noise", "n": 15, "layers": 2, "gamma": 0.01},
        # a training step of the warm-start network (46 -> 256 x 3 -> 128) on one batch
        {"name": "network_256", "family": "network", "batch": 256},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    family = rng.choice(["brickwork", "brickwork", "qft", "trotter", "builders", "gradient",
                         "gradient", "batch", "batch", "energy", "precision", "shots", "noise",
                         "network"])
    c = {"family": family}
    if family == "brickwork":
        c.update(n=rng.randint(6, 27), layers=_log_int(rng, 1, 20))
    elif family == "qft":
        c.update(n=rng.randint(4, 24), inverse=rng.random() < 0.5)
    elif family == "trotter":
        c.update(n=rng.randint(4, 21), steps=rng.randint(1, 10))
    elif family == "builders":
        c.update(n=rng.randint(2, 18), gates=_log_int(rng, 10, 150))
    elif family == "gradient":
        c.update(n=rng.randint(2, 12), depth=rng.randint(1, 3))
    elif family == "batch":
        lo = rng.randint(5, 13)
        c.update(count=_log_int(rng, 8, 128), n_lo=lo, n_hi=lo + rng.randint(0, 3))
    elif family == "energy":
        c.update(n=rng.randint(4, 27), c64=rng.random() < 0.25)
    elif family == "precision":
        c.update(n=rng.randint(12, 26), layers=_log_int(rng, 2, 20))
    elif family == "shots":
        c.update(n=rng.randint(4, 25), shots=_log_int(rng, 100, 20000))
    elif family == "noise":
        c.update(n=rng.randint(3, 16), layers=rng.randint(1, 2),
                 gamma=round(rng.uniform(0.002, 0.05), 4))
    else:
        c.update(batch=_log_int(rng, 16, 1024))
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
class _Buffer:
    """A state's device buffer as torch sees it.  The handle keeps owning it: a tensor
    holds this object, and this object the handle, for as long as it is used."""

    def __init__(self, state):
        self.state = state
        p = ctypes.c_void_p()
        call("lq_state_device_ptr", state.handle, ctypes.byref(p))
        kind = "<c8" if state.dtype == abi.LQ_C64 else "<c16"
        self.__cuda_array_interface__ = {"shape": (1 << state.num_qubits(),), "typestr": kind,
                                         "data": (p.value, False), "version": 3, "strides": None}


def _amplitudes(state):
    return torch.as_tensor(_Buffer(state), device="cuda")


def _gaussian(n, seed, dtype=torch.complex128):
    """A random state: complex Gaussian amplitudes, normalised."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + n)
    v = torch.randn(1 << n, dtype=torch.complex128, device=dev, generator=g)
    v /= torch.linalg.vector_norm(v)
    return v.to(dtype)


def _random_state(n, seed, c64=False):
    s = State(n, abi.LQ_C64 if c64 else abi.LQ_C128)
    call("lq_state_synchronize", s.handle)
    _amplitudes(s).copy_(_gaussian(n, seed, torch.complex64 if c64 else torch.complex128))
    torch.cuda.synchronize()
    return s


def _rng(case, seed):
    return np.random.default_rng([int(seed), case["n"] if "n" in case else 0])


def _brickwork_gates(case, seed):
    """[(name, qubits, angles)] of the U3 + CNOT brickwork."""
    n, out = case["n"], []
    ang = _rng(case, seed).uniform(0.0, 2.0 * math.pi, (case["layers"], n, 3))
    for layer in range(case["layers"]):
        out += [("u3", (q,), tuple(ang[layer, q])) for q in range(n)]
        out += [("cnot", (q, q + 1), ()) for q in range(layer % 2, n - 1, 2)]
    return out


def _trotter(case, seed):
    r = _rng(case, seed)
    return dict(jx=r.uniform(0.5, 1.0), jy=r.uniform(0.5, 1.0), jz=r.uniform(0.5, 1.0),
                external_field=r.uniform(0.1, 0.5), time_steps=case["steps"], dt=0.05)


def _neel(n):
    return sum(1 << b for b in range(0, n, 2))


def _builder_gates(case, seed):
    """Random single-qubit builders, with an entangler after every second one."""
    n, r, out = case["n"], _rng(case, seed), []
    while len(out) < case["gates"]:
        kind = ["h", "x", "s", "t", "rx_matrix", "ry_matrix"][r.integers(6)]
        q = int(r.integers(n))
        out.append((kind, (q,), (float(r.uniform(0, 2 * math.pi)),) if "_" in kind else ()))
        if n > 1 and len(out) % 3 == 2:
            a, b = (int(x) for x in r.choice(n, 2, replace=False))
            out.append((["cnot", "cz"][r.integers(2)], (a, b), ()))
    return out[:case["gates"]]


def _noise_gates(case, seed):
    n, r, out = case["n"], _rng(case, seed), []
    for _ in range(case["layers"]):
        out += [("ry", (q,), (float(r.uniform(-math.pi, math.pi)),)) for q in range(n)]
        out += [("cnot", (q, q + 1), ()) for q in range(n - 1)]
    return out


def _circuit(n, gates):
    c = Circuit(n)
    for name, qubits, angles in gates:
        getattr(c, name)(*qubits, *angles)
    return c


def _couplings(n, r):
    return (r.uniform(-1, 1, n - 1), r.uniform(-1, 1, n - 1), r.uniform(-1, 1, n - 1),
            float(r.uniform(0.05, 0.5)))


def _chains(case, seed):
    """Records as workloads.heisenberg_instances makes them, the sizes in turn."""
    r, out = np.random.default_rng([int(seed), case["count"]]), []
    for i in range(case["count"]):
        n = case["n_lo"] + (7 * i) % (case["n_hi"] - case["n_lo"] + 1)
        jx, jy, jz, h = _couplings(n, r)
        out.append({"n": n, "jx": jx, "jy": jy, "jz": jz, "h": h,
                    "theta": r.uniform(-math.pi, math.pi, 2 * n * LAYERS)})
    return out


def _network(case, seed):
    """Weights, inputs (couplings), target angles and masks of one batch, FP32."""
    r = np.random.default_rng([int(seed), case["batch"]])
    dims = [IN_DIM] + [HIDDEN] * DEPTH + [OUT_DIM]
    p = []
    for a, b in zip(dims[:-1], dims[1:]):
        p += [r.uniform(-1, 1, b * a) * math.sqrt(6.0 / a), r.uniform(-0.1, 0.1, b)]
    x = r.uniform(-1, 1, (case["batch"], IN_DIM))
    t = r.uniform(-math.pi, math.pi, (case["batch"], OUT_DIM))
    m = np.arange(OUT_DIM)[None, :] < 2 * LAYERS * r.integers(12, 17, case["batch"])[:, None]
    return tuple(np.ascontiguousarray(a, dtype=np.float32) for a in (np.concatenate(p), x, t, m))


def prepare(case, seed):
    f, s = case["family"], {"family": case["family"], "case": case}
    if f in ("brickwork", "precision"):
        s["state"] = State(case["n"], abi.LQ_C64 if f == "precision" else abi.LQ_C128)
        s["circuit"] = _circuit(case["n"], _brickwork_gates(case, seed))
        s["gates"] = s["circuit"].packed()
    elif f == "qft":
        s["input"] = _random_state(case["n"], seed)
        s["state"] = State(case["n"])
        make = qft.create_inverse_circuit if case["inverse"] else qft.create_circuit
        s["circuit"] = make(case["n"])
    elif f == "trotter":
        s["state"] = State(case["n"])
        s["circuit"] = xyz_heisenberg.create_circuit(case["n"], **_trotter(case, seed))
    elif f == "builders":
        s["state"] = State(case["n"])
        s["circuit"] = _circuit(case["n"], _builder_gates(case, seed))
    elif f == "noise":
        s["state"] = State(case["n"])
        s["circuit"] = _circuit(case["n"], _noise_gates(case, seed))
        s["circuit"].add_noise(AmplitudeDampingNoise(case["gamma"]))
        s["circuit"].add_noise(PhaseDampingNoise(0.02))
    elif f == "gradient":
        r = _rng(case, seed)
        s["ansatz"] = EfficientSU2Ansatz(case["n"], case["depth"])
        s["hamiltonian"] = xyz_heisenberg.hamiltonian(case["n"], *_couplings(case["n"], r))
        s["theta"] = r.uniform(-math.pi, math.pi, s["ansatz"].num_parameters())
        s["method"] = ParameterShift()
    elif f == "batch":
        recs = _chains(case, seed)
        s["batch"] = heisenberg_batch(recs)
        s["theta"] = np.concatenate([q["theta"] for q in recs])
        s["batch"].gradients(s["theta"])  # an optimisation loop's handle is tuned by its first call
    elif f == "energy":
        s["state"] = _random_state(case["n"], seed, case["c64"])
        s["hamiltonian"] = xyz_heisenberg.hamiltonian(case["n"],
                                                      *_couplings(case["n"], _rng(case, seed)))
    elif f == "shots":
        s["state"] = _random_state(case["n"], seed)
        s["seed"] = int(seed)
    else:
        p, s["x"], s["t"], s["m"] = _network(case, seed)
        s["net"] = WarmStartMLP()
        s["net"].set_params(p)
    if "state" in s:
        s["out"] = _amplitudes(s["state"])
        call("lq_state_synchronize", s["state"].handle)
    return s


def run(s):
    f = s["family"]
    if f == "precision":
        h, g = s["state"].handle, s["gates"]
        call("lq_state_set_basis", h, 0)
        call("lq_apply_circuit_tc", h, s["case"]["n"], abi.gate_ptr(g), len(g), None, 0, None, None)
        return s["out"]
    if f in ("brickwork", "trotter", "builders", "noise", "qft"):
        if f == "qft":
            call("lq_state_copy", s["state"].handle, s["input"].handle)
        else:
            call("lq_state_set_basis", s["state"].handle,
                 _neel(s["case"]["n"]) if f == "trotter" else 0)
        s["circuit"].execute(s["state"])
        return s["out"]
    if f == "gradient":
        return s["method"].compute_gradient(s["ansatz"], s["hamiltonian"], s["theta"])
    if f == "batch":
        energies, gradients = s["batch"].gradients(s["theta"])
        return {"energies": energies, "gradients": gradients}
    if f == "energy":
        return s["hamiltonian"].expectation(s["state"])
    if f == "shots":
        out = np.empty(s["case"]["shots"], np.uint64)
        call("lq_measure_shots", s["state"].handle, len(out), s["seed"],
             out.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)))
        return out.astype(np.int64)
    loss = s["net"].loss_grad(s["x"], s["t"], s["m"])
    return {"loss": loss, "grads": s["net"].grads()}


# ---------------------------------------------------------------------------
# Work: every input read once and every output written once, and the arithmetic
# of the gates.  Per amplitude a 2x2 unitary takes 8 operations (scaled to one
# unit entry per row, [1, t; -t*, 1]), a 4x4 rotation of two 2x2 blocks the same,
# a phase 6; a gradient takes one circuit forward and two back.
# ---------------------------------------------------------------------------
def _chain(n):
    return 2 * LAYERS * n, 11.0 * LAYERS * n * 2.0 ** n


def work(case):
    f, n = case["family"], case.get("n", 0)
    N = 2.0 ** n
    if f == "brickwork":
        return {"bytes": 16 * N, "flops": 8 * N * n * case["layers"]}
    if f == "precision":
        return {"bytes": 8 * N, "flops": 8 * N * n * case["layers"]}
    if f == "qft":
        return {"bytes": 32 * N, "flops": N * (4 * n + 6 * n)}
    if f == "trotter":
        return {"bytes": 16 * N, "flops": case["steps"] * N * (n - 1) * (4 + 4 + 6)}
    if f == "builders":
        return {"bytes": 16 * N, "flops": 4 * N * case["gates"]}
    if f == "noise":
        gates = case["layers"] * (2 * n - 1)
        return {"bytes": 16 * N, "flops": gates * N * (4 + 4 * n + 4)}
    if f == "gradient":
        p = 3 * n * case["depth"]
        return {"bytes": 16.0 * p, "flops": 3 * N * 8 * n * case["depth"] + 8 * N * p}
    if f == "batch":
        mean = [_chain(k) for k in range(case["n_lo"], case["n_hi"] + 1)]
        p, g = (case["count"] * sum(v) / len(mean) for v in zip(*mean))
        return {"bytes": 16.0 * p, "flops": 3.0 * g}
    if f == "energy":
        return {"bytes": (8 if case["c64"] else 16) * N, "flops": 8 * N * n}
    if f == "shots":
        return {"bytes": 16 * N + 8 * case["shots"], "flops": 4 * N}
    weights = IN_DIM * HIDDEN + (DEPTH - 1) * HIDDEN * HIDDEN + HIDDEN * OUT_DIM
    return {"bytes": 8.0 * weights + 4.0 * case["batch"] * (IN_DIM + 2 * OUT_DIM),
            "flops": 6.0 * case["batch"] * weights}


# ---------------------------------------------------------------------------
# The same results in 64 bits by plain torch
# ---------------------------------------------------------------------------
def _m(*rows):
    return torch.stack([torch.stack([torch.as_tensor(x, dtype=torch.complex128) for x in r])
                        for r in rows])


def _one(v, n, q, m):
    """A 2x2 matrix on qubit q (qubit 0 is the highest index bit)."""
    v = v.reshape(1 << q, 2, -1)
    a, b = v[:, 0], v[:, 1]
    return torch.stack([m[0, 0] * a + m[0, 1] * b, m[1, 0] * a + m[1, 1] * b], 1).reshape(-1)


def _cnot(v, n, c, t):
    lo, hi = min(c, t), max(c, t)
    w = v.reshape(1 << lo, 2, 1 << (hi - lo - 1), 2, -1)
    if c < t:
        return torch.stack([w[:, 0], w[:, 1].flip(2)], 1).reshape(-1)
    return torch.stack([w[:, :, :, 0], w[:, :, :, 1].flip(1)], 3).reshape(-1)


def _two_phases(v, n, a, b, ph):
    """Phase ph[i][j] where qubit a is i and qubit b is j."""
    lo, hi = min(a, b), max(a, b)
    w = v.reshape(1 << lo, 2, 1 << (hi - lo - 1), 2, -1).clone()
    for i in range(2):
        for j in range(2):
            x, y = (i, j) if a < b else (j, i)
            w[:, x, :, y] *= ph[i][j]
    return w.reshape(-1)


def _matrix(name, ang):
    e = lambda x: torch.exp(1j * torch.as_tensor(x, dtype=torch.float64))  # noqa: E731
    if name in ("rx", "rx_matrix", "ry", "ry_matrix", "rz", "u3"):
        h = torch.as_tensor(ang[0], dtype=torch.float64) / 2
        c, s = torch.cos(h) + 0j, torch.sin(h) + 0j
        if name.startswith("rx"):
            return _m((c, -1j * s), (-1j * s, c))
        if name.startswith("ry"):
            return _m((c, -s), (s, c))
        if name == "rz":
            return _m((e(-h), 0), (0, e(h)))
        return _m((c, -s * e(ang[2])), (s * e(ang[1]), c * e(ang[1] + ang[2])))
    r = math.sqrt(0.5)
    return _m(*{"h": ((r, r), (r, -r)), "x": ((0, 1), (1, 0)), "s": ((1, 0), (0, 1j)),
                "t": ((1, 0), (0, complex(math.cos(math.pi / 4), math.sin(math.pi / 4))))}[name])


def _gate(v, n, gate):
    name, q, ang = gate
    if name == "cnot":
        return _cnot(v, n, *q)
    if name == "cz":
        return _two_phases(v, n, *q, ((1, 1), (1, -1)))
    return _one(v, n, q[0], _matrix(name, ang).to(v.device))


def _zero(n, index=0):
    v = torch.zeros(1 << n, dtype=torch.complex128,
                    device="cuda" if torch.cuda.is_available() else "cpu")
    v[index] = 1
    return v


def _chain_energy(v, n, jx, jy, jz, h):
    """<v| sum_b Jx XX + Jy YY + Jz ZZ + h sum Z |v>, open chain."""
    e = 0.0
    p = v.abs() ** 2
    for b in range(n - 1):
        w = v.reshape(1 << b, 2, 2, -1)
        flip = 2 * (w[:, 0, 0].conj() * w[:, 1, 1]).real.sum()
        hop = 2 * (w[:, 0, 1].conj() * w[:, 1, 0]).real.sum()
        d = p.reshape(1 << b, 2, 2, -1).sum((0, 3))
        e = e + jx[b] * (flip + hop) + jy[b] * (hop - flip)
        e = e + jz[b] * (d[0, 0] + d[1, 1] - d[0, 1] - d[1, 0])
    for q in range(n):
        d = p.reshape(1 << q, 2, -1).sum((0, 2))
        e = e + h * (d[0] - d[1])
    return e


def _gradient(n, gates, theta, couplings):
    """Energy and its derivatives (the parameter-shift rule's value for shift pi/2)."""
    t = torch.tensor(np.asarray(theta), dtype=torch.float64, requires_grad=True)
    v = _zero(n)
    for name, q, p in gates:
        v = _cnot(v, n, *q) if name == "cnot" else _one(v, n, q[0], _matrix(name, (t[p],)).to(v.device))
    e = _chain_energy(v, n, *couplings)
    e.backward()
    return float(e.detach()), t.grad.numpy()


def exact(case, seed):
    f, n = case["family"], case.get("n", 0)
    if f in ("brickwork", "precision", "builders"):
        make = _builder_gates if f == "builders" else _brickwork_gates
        v = _zero(n)
        for g in make(case, seed):
            v = _gate(v, n, g)
        return v
    if f == "qft":
        make = torch.fft.fft if case["inverse"] else torch.fft.ifft
        return make(_gaussian(n, seed), norm="ortho")
    if f == "trotter":
        k, v = _trotter(case, seed), _zero(n, _neel(n))
        for _ in range(case["steps"]):
            # RXX and RYY rotate only |00>, |11> for ascending qubits, as the reference does
            for j, sign in ((k["jx"], -1), (k["jy"], 1)):
                c, s = math.cos(j * k["dt"]), math.sin(j * k["dt"])
                for b in range(n - 1):
                    w = v.reshape(1 << b, 2, 2, -1).clone()
                    x, y = w[:, 0, 0].clone(), w[:, 1, 1].clone()
                    w[:, 0, 0] = c * x + sign * 1j * s * y
                    w[:, 1, 1] = c * y + sign * 1j * s * x
                    v = w.reshape(-1)
            a = k["jz"] * k["dt"]
            p, m = complex(math.cos(a), -math.sin(a)), complex(math.cos(a), math.sin(a))
            for b in range(n - 1):
                v = _two_phases(v, n, b, b + 1, ((p, m), (m, p)))
            for q in range(n):
                v = _one(v, n, q, _matrix("rz", (k["external_field"] * k["dt"],)).to(v.device))
        return v
    if f == "noise":
        v, sg, s1 = _zero(n), math.sqrt(case["gamma"]), math.sqrt(1 - case["gamma"])
        sl = math.sqrt(0.98)
        for g in _noise_gates(case, seed):
            v = _gate(v, n, g)
            acc = 0
            for q in range(n):
                w = v.reshape(1 << q, 2, -1)
                acc = acc + torch.stack([w[:, 0] + sg * w[:, 1], s1 * w[:, 1]], 1).reshape(-1)
            v = acc / torch.linalg.vector_norm(acc)
            w = v.reshape(2, -1)  # index bit n-1, the last target
            v = torch.cat([w[0], sl * w[1]])
            v = v / torch.linalg.vector_norm(v)
        return v
    if f == "gradient":
        r = _rng(case, seed)
        couplings = _couplings(n, r)
        theta = r.uniform(-math.pi, math.pi, 3 * n * case["depth"])
        gates, p = [], 0
        for _ in range(case["depth"]):
            for q in range(n):
                gates += [("rz", (q,), p), ("ry", (q,), p + 1), ("rz", (q,), p + 2)]
                p += 3
            gates += [("cnot", (q, q + 1), 0) for q in range(n - 1)]
        return _gradient(n, gates, theta, couplings)[1]
    if f == "batch":
        if case["count"] * 2.0 ** (case["n_hi"] - 12) > 300:
            return None
        es, gs = [], []
        for k in _chains(case, seed):
            gates, p = [], 0
            for _ in range(LAYERS):
                for q in range(k["n"]):
                    gates += [("ry", (q,), p), ("rz", (q,), p + 1)]
                    p += 2
                gates += [("cnot", (q, q + 1), 0) for q in range(k["n"] - 1)]
            e, g = _gradient(k["n"], gates, k["theta"], (k["jx"], k["jy"], k["jz"], k["h"]))
            es.append(e)
            gs.append(g)
        return {"energies": np.array(es), "gradients": np.concatenate(gs)}
    if f == "energy":
        v = _gaussian(n, seed, torch.complex64 if case["c64"] else torch.complex128)
        return float(_chain_energy(v.to(torch.complex128), n, *_couplings(n, _rng(case, seed))))
    if f == "shots":
        return None
    p, x, t, m = (torch.tensor(a, dtype=torch.float64) for a in _network(case, seed))
    p.requires_grad_(True)
    dims, h, off = [IN_DIM] + [HIDDEN] * DEPTH + [OUT_DIM], x, 0
    for i, (a, b) in enumerate(zip(dims[:-1], dims[1:])):
        h = h @ p[off:off + a * b].reshape(b, a).T + p[off + a * b:off + a * b + b]
        off += a * b + b
        if i + 2 < len(dims):
            h = torch.nn.functional.gelu(h)
    loss = (m * (1 - torch.cos(h - t))).sum() / m.sum()
    loss.backward()
    return {"loss": float(loss.detach()), "grads": p.grad.numpy()}
