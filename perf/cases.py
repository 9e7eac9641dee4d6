"""What the library is timed on: the work its users have it do, through its public entry points.

Each listed case says below what it stands for. `draw` gives more cases of the same kinds over
the same ranges: qubit counts (the work doubles with each), depths, precisions and shot counts.
Circuits are the benchmark's (qclojure_gb300/workloads.py): layers of one random gate per qubit
and CNOTs on a random matching, a QFT, QAOA MaxCut on random 3-regular graphs.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from qclojure_gb300 import hardware, variational, workloads
from qclojure_gb300.backend import create_simulator, execute_circuit
from qclojure_gb300.state import Context
from qclojure_gb300.sweep import Sweep

# depolarizing on every gate type, asymmetric readout: the benchmark's noisy workload
_GATES_1Q = ("h", "x", "y", "z", "s", "t", "rx", "ry", "rz")


def listed() -> list[dict]:
    return [
        # the smallest work: one job of the job API (10 qubits, 20 layers, 1024 shots), with its
        # probabilities and final state on the host; latency and host work count
        {"name": "job-c128-10q", "kind": "job", "qubits": 10, "depth": 20, "shots": 1024, "precision": "c128"},
        # a circuit that runs once, below the size from which its passes get kernels of their
        # own: the interpreting executor in both precisions (the serving stream's larger jobs)
        {"name": "oneoff-c128-21q", "kind": "circuit", "qubits": 21, "depth": 30, "qft": False, "precision": "c128",
         "arithmetic": "double-float", "kernels": "auto"},
        {"name": "oneoff-c64-25q", "kind": "circuit", "qubits": 25, "depth": 12, "qft": True, "precision": "c64",
         "arithmetic": "double-float", "kernels": "auto"},
        # the arithmetic that equals the reference's simulator bit for bit
        {"name": "exact-c128-19q", "kind": "circuit", "qubits": 19, "depth": 20, "qft": False, "precision": "c128",
         "arithmetic": "exact", "kernels": "auto"},
        # the headline path: a large circuit on a resident state, its pass kernels compiled
        # beforehand; layers and a QFT, double-float complex128 and complex64
        {"name": "circuit-c128-28q", "kind": "circuit", "qubits": 28, "depth": 10, "qft": True, "precision": "c128",
         "arithmetic": "double-float", "kernels": "always"},
        {"name": "circuit-c64-29q", "kind": "circuit", "qubits": 29, "depth": 8, "qft": True, "precision": "c64",
         "arithmetic": "double-float", "kernels": "always"},
        # measurements with collapse inside a circuit (syndrome rounds, feed-forward protocols)
        {"name": "midcircuit-c128-20q", "kind": "midcircuit", "qubits": 20, "depth": 3, "rounds": 6, "measured": 3,
         "precision": "c128"},
        # a parameter sweep over sizes (QAOA MaxCut, p = 3): every circuit's energy
        {"name": "sweep-c64-12-22q", "kind": "sweep", "circuits": 64, "least": 12, "most": 22, "layers": 3,
         "precision": "c64"},
        # one step of a variational loop: new angles, the energy and the parameter-shift points
        {"name": "gradient-c128-18q", "kind": "gradient", "qubits": 18, "layers": 3, "precision": "c128"},
        # a million shots from a large resident state
        {"name": "shots-c64-30q", "kind": "shots", "qubits": 30, "shots": 1000000, "precision": "c64"},
        # the energy of a Heisenberg chain in a field (X, Y and Z terms) on a resident state
        {"name": "energy-c128-24q", "kind": "energy", "qubits": 24, "depth": 4, "precision": "c128"},
        # the noisy simulator's shot loop, with the first hundred trajectories
        {"name": "noisy-c128-10q", "kind": "noisy", "qubits": 10, "depth": 20, "shots": 20000, "p1": 0.001,
         "p2": 0.01, "precision": "c128"},
    ]


def draw(rng: random.Random) -> dict:
    kind = rng.choice(("job", "oneoff", "exact", "circuit", "midcircuit", "sweep", "gradient", "shots", "energy",
                       "noisy"))
    prec = rng.choice(("c128", "c64"))
    if kind == "job":
        return {"kind": "job", "qubits": rng.randint(5, 14), "depth": rng.randint(5, 40),
                "shots": int(math.exp(rng.uniform(math.log(100), math.log(20000)))), "precision": "c128"}
    if kind == "oneoff":
        return {"kind": "circuit", "qubits": rng.randint(13, 24 if prec == "c128" else 26),
                "depth": rng.randint(4, 30), "qft": rng.random() < 0.5, "precision": prec,
                "arithmetic": "double-float", "kernels": "auto"}
    if kind == "exact":
        return {"kind": "circuit", "qubits": rng.randint(8, 22), "depth": rng.randint(4, 30),
                "qft": rng.random() < 0.5, "precision": "c128", "arithmetic": "exact", "kernels": "auto"}
    if kind == "circuit":
        return {"kind": "circuit", "qubits": rng.randint(23, 27 if prec == "c128" else 28),
                "depth": rng.randint(3, 10), "qft": rng.random() < 0.7, "precision": prec,
                "arithmetic": "double-float", "kernels": "always"}
    if kind == "midcircuit":
        return {"kind": "midcircuit", "qubits": rng.randint(12, 23), "depth": rng.randint(1, 4),
                "rounds": rng.randint(2, 8), "measured": rng.randint(1, 5), "precision": prec}
    if kind == "sweep":
        least = rng.choice((12, 14))
        return {"kind": "sweep", "circuits": rng.randint(8, 64), "least": least,
                "most": rng.choice((least, 16, 18, 20)), "layers": rng.randint(1, 4), "precision": prec}
    if kind == "gradient":
        return {"kind": "gradient", "qubits": 2 * rng.randint(6, 10), "layers": rng.randint(1, 4), "precision": prec}
    if kind == "shots":
        return {"kind": "shots", "qubits": rng.randint(12, 29),
                "shots": int(math.exp(rng.uniform(math.log(1000), math.log(1000000)))), "precision": prec}
    if kind == "energy":
        return {"kind": "energy", "qubits": rng.randint(12, 24), "depth": rng.randint(2, 5), "precision": prec}
    return {"kind": "noisy", "qubits": rng.randint(4, 11), "depth": rng.randint(4, 20),
            "shots": int(math.exp(rng.uniform(math.log(1000), math.log(20000)))),
            "p1": 10 ** rng.uniform(-3.5, -1.7), "p2": 10 ** rng.uniform(-2.5, -1.3), "precision": "c128"}


# ---- circuits ----------------------------------------------------------------------------
def _circuit(case: dict, seed: int) -> dict:
    n = case["qubits"]
    c = workloads.layered_circuit(n, case["depth"], seed)
    if case.get("qft"):
        c["operations"] = c["operations"] + workloads.qft_ops(n)
    return c


def _midcircuit(case: dict, seed: int) -> dict:
    n, rng = case["qubits"], random.Random(seed)
    ops: list = []
    for r in range(case["rounds"]):
        ops += workloads.layered_circuit(n, case["depth"], 1000 * seed + r)["operations"]
        ops.append({"operation-type": "measure",
                    "operation-params": {"measurement-qubits": rng.sample(range(n), case["measured"])}})
    return {"num-qubits": n, "operations": ops}


def _heisenberg(n: int) -> list[tuple[float, str]]:
    terms = []
    for p, j in (("X", 1.0), ("Y", 1.0), ("Z", 0.5)):
        for q in range(n - 1):
            terms.append((j, "I" * q + p + p + "I" * (n - q - 2)))
    return terms + [(0.3, "I" * q + "Z" + "I" * (n - q - 1)) for q in range(n)]


def _sweep_circuits(case: dict, seed: int) -> list[dict]:
    sizes = range(case["least"], case["most"] + 1, 2)
    rng = np.random.default_rng(seed)
    ns = [sizes[i % len(sizes)] for i in range(case["circuits"])]
    return [workloads.qaoa_maxcut(n, case["layers"], int(rng.integers(1 << 30))) for n in ns]


def _gradient_inputs(case: dict, seed: int):
    rng = np.random.default_rng(seed)
    edges = workloads.random_3_regular_graph(case["qubits"], rng)
    params = [float(x) for x in rng.uniform(0.1, math.pi / 2, 2 * case["layers"])]
    return edges, params


def _maxcut(n: int, edges) -> list[dict]:
    ham = []
    for a, b in edges:
        ham.append({"coefficient": 0.5, "pauli-string": "I" * n})
        ham.append({"coefficient": -0.5,
                    "pauli-string": "".join("Z" if q in (a, b) else "I" for q in range(n))})
    return ham


def _random_state(n: int, precision: str, seed: int) -> torch.Tensor:
    """Gaussian amplitudes, normalised: what a deep random circuit leaves (Porter-Thomas)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    real = torch.float32 if precision == "c64" else torch.float64
    x = torch.randn((1 << n) * 2, dtype=real, device="cuda", generator=g)
    norm2 = sum(float(c.double().square().sum()) for c in x.split(1 << 26))
    x /= math.sqrt(norm2)
    return torch.view_as_complex(x.view(-1, 2))


class _DeviceArray:
    """A state's amplitude array, for torch; a tensor made of it keeps the state alive."""

    def __init__(self, state, owner):
        self.owner = owner
        ptr, _ = state.device_ptr()
        self.__cuda_array_interface__ = {"shape": (1 << state.n,), "data": (ptr, False), "version": 3,
                                         "typestr": "<c16" if state.precision == "c128" else "<c8"}


class _Owner:
    """Closes what it was given, last first, when nothing refers to it any more."""

    def __init__(self):
        self.owned: list = []

    def __del__(self):
        for x in reversed(self.owned):
            x.close()


class _Held:
    """What a user's program keeps between calls."""

    def __init__(self, case: dict, **kw):
        self.case = case
        self.owner = _Owner()
        self.__dict__.update(kw)

    def own(self, x):
        self.owner.owned.append(x)
        return x


def _held_state(case: dict, **context) -> _Held:
    h = _Held(case)
    ctx = h.own(Context(**context))
    h.state = h.own(ctx.state(case["qubits"], case["precision"]))
    h.array = torch.as_tensor(_DeviceArray(h.state, h.owner), device="cuda")
    return h


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind == "job":
        h = _Held(case, circuit=_circuit(case, seed), seed=seed)
        h.sim = h.own(create_simulator({"precision": case["precision"]}))
        return h
    if kind == "circuit":
        h = _held_state(case, arithmetic=case["arithmetic"], pass_kernels=case["kernels"])
        h.circuit, h.seed = _circuit(case, seed), seed
        if case["kernels"] == "always":
            h.state.prepare(h.circuit)
        return h
    if kind == "midcircuit":
        h = _held_state(case)
        h.circuit, h.seed = _midcircuit(case, seed), seed
        return h
    if kind == "sweep":
        h = _Held(case)
        ctx = h.own(Context())
        circuits = _sweep_circuits(case, seed)
        h.hamiltonians = [c["hamiltonian"] for c in circuits]
        h.sweep = h.own(Sweep(ctx, circuits, case["precision"]))
        return h
    if kind == "gradient":
        n = case["qubits"]
        edges, h_params = _gradient_inputs(case, seed)
        h = _Held(case, params=h_params)
        ctx = h.own(Context())
        h.objective = h.own(variational.BatchedObjective(
            ctx, _maxcut(n, edges), lambda p: variational.qaoa_maxcut_circuit(n, edges, p), case["precision"]))
        # the loop's first step makes the sweep; the timed step gives it other angles
        h.objective.energies([[0.3] * len(h_params)] * (2 * len(h_params) + 1))
        return h
    if kind == "shots":
        h = _held_state(case)
        h.seed = seed
        h.array.copy_(_random_state(case["qubits"], case["precision"], seed))
        torch.cuda.synchronize()
        return h
    if kind == "energy":
        h = _held_state(case)
        h.terms = _heisenberg(case["qubits"])
        h.state.set_basis(0)
        h.state.apply(_circuit(case, seed))
        return h
    h = _Held(case, circuit=_circuit(case, seed), seed=seed)
    h.ctx = h.own(Context())
    one = {"noise-type": "depolarizing", "noise-strength": case["p1"]}
    h.noise = {"gate-noise": dict({g: one for g in _GATES_1Q},
                                  cnot={"noise-type": "depolarizing", "noise-strength": case["p2"]}),
               "readout-error": {"prob-0-to-1": 0.01, "prob-1-to-0": 0.02}}
    return h


def run(h):
    case = h.case
    kind = case["kind"]
    if kind == "job":
        res = execute_circuit(h.sim, h.circuit, {"result-specs": {"measurements": {"shots": case["shots"]},
                                                                  "probabilities": {}, "state-vector": True},
                                                 "seed": h.seed})
        r = res["results"]
        out = {"shots": np.array(r["measurement-results"]["measurement-outcomes"], dtype=np.int64),
               "probabilities": r["probability-results"]["all-probabilities"],
               "state": np.asarray(r["state-vector-result"]["state-vector"])}
        h.sim.free_job(res["job-id"])
        return out
    if kind in ("circuit", "midcircuit"):
        h.state.set_basis(0)
        h.state.apply(h.circuit, seed=h.seed)
        return h.array
    if kind == "sweep":
        return h.sweep.run(h.hamiltonians)[0]
    if kind == "gradient":
        e, g = variational._energy_and_gradient(h.objective, h.params, {})
        return {"energy": np.float64(e), "gradient": g}
    if kind == "shots":
        return h.state.sample(case["shots"], h.seed).view(np.int64)
    if kind == "energy":
        return np.float64(h.state.hamiltonian(h.terms))
    res = hardware.run_trajectories(h.ctx, h.circuit, h.noise, case["shots"], seed=h.seed)
    return {"shots": res["outcomes"].view(np.int64), "trajectories": res["trajectories"],
            "last": res["final_state"]}


def _gate_flops(ops: list, n: int) -> float:
    """Real operations on the amplitudes: a full 2x2 on every pair, a phase on the amplitudes it
    touches; permutations none. A global factor may be left to the end."""
    per = 0.0
    for op in ops:
        t = op["operation-type"]
        if t in ("h", "rx", "ry"):
            per += 4.0  # with its diagonal factored out: one product and one sum per real
        elif t in ("s", "t", "z", "rz"):
            per += 3.0
        elif t == "rydberg-cphase":
            per += 1.5
        elif t == "rzz":
            per += 3.0
    return per * (1 << n)


def work(case: dict) -> dict:
    kind, size = case["kind"], 16 if case["precision"] == "c128" else 8
    if kind == "sweep":
        circuits = _sweep_circuits(case, 0)
        # |0...0> is made and every energy needs each final amplitude once
        return {"bytes": float(sum(size << c["num-qubits"] for c in circuits)),
                "flops": sum(_gate_flops(c["operations"], c["num-qubits"]) for c in circuits)}
    n = case["qubits"]
    state = float(size << n)
    if kind == "job":
        return {"bytes": state + (8 << n) + 8 * case["shots"], "flops": _gate_flops(_circuit(case, 0)["operations"], n)}
    if kind == "circuit":
        return {"bytes": state, "flops": _gate_flops(_circuit(case, 0)["operations"], n)}
    if kind == "midcircuit":
        return {"bytes": state, "flops": _gate_flops(_midcircuit(case, 0)["operations"], n)
                + 3.0 * case["rounds"] * (1 << n)}
    if kind == "gradient":
        edges, params = _gradient_inputs(case, 0)
        count = 2 * len(params) + 1
        ops = variational.qaoa_maxcut_circuit(n, edges, params)["operations"]
        return {"bytes": count * state, "flops": count * _gate_flops(ops, n)}
    if kind == "shots":
        return {"bytes": state + 8.0 * case["shots"], "flops": 3.0 * (1 << n)}
    if kind == "energy":
        return {"bytes": state, "flops": 4.0 * len(_heisenberg(n)) * (1 << n)}
    return {"bytes": state * 100 + 8.0 * case["shots"],
            "flops": 100 * _gate_flops(_circuit(case, 0)["operations"], n)}


# ---- the same in 64 bits, plain torch ----------------------------------------------------
_R = 1 / math.sqrt(2)


def _apply_1q(s: torch.Tensor, n: int, q: int, m) -> None:
    v = s.view(1 << q, 2, -1)
    a, b = v[:, 0], v[:, 1]
    if m[0][1] == 0 and m[1][0] == 0:
        if m[0][0] != 1:
            a.mul_(m[0][0])
        if m[1][1] != 1:
            b.mul_(m[1][1])
        return
    x = a * m[0][0]
    x.add_(b, alpha=m[0][1])
    b.mul_(m[1][1])
    b.add_(a, alpha=m[1][0])
    a.copy_(x)


def _pair(s: torch.Tensor, n: int, a: int, b: int) -> torch.Tensor:
    """A view with the bits of qubits a < b as dimensions 1 and 3."""
    return s.view(1 << a, 2, 1 << (b - a - 1), 2, -1)


def _exact_ops(s: torch.Tensor, n: int, ops: list) -> None:
    for op in ops:
        t, p = op["operation-type"], op["operation-params"]
        th = p.get("angle", 0.0)
        c, i = math.cos(th / 2), math.sin(th / 2)
        if t in ("cnot", "rydberg-cphase", "swap", "rzz"):
            a, b = ((p["control"], p["target"]) if t in ("cnot", "rydberg-cphase") else (p["qubit1"], p["qubit2"]))
            v = _pair(s, n, min(a, b), max(a, b))
            if t == "rydberg-cphase":
                v[:, 1, :, 1].mul_(complex(math.cos(th), math.sin(th)))
            elif t == "rzz":
                for x in (0, 1):
                    v[:, x, :, x].mul_(complex(c, -i))
                    v[:, x, :, 1 - x].mul_(complex(c, i))
            else:
                x, y = ((v[:, 0, :, 1], v[:, 1, :, 0]) if t == "swap" else
                        (v[:, 1, :, 0], v[:, 1, :, 1]) if a < b else (v[:, 0, :, 1], v[:, 1, :, 1]))
                z = x.clone()
                x.copy_(y)
                y.copy_(z)
            continue
        m = {"h": [[_R, _R], [_R, -_R]], "x": [[0, 1], [1, 0]], "y": [[0, -1j], [1j, 0]], "z": [[1, 0], [0, -1]],
             "s": [[1, 0], [0, 1j]], "t": [[1, 0], [0, complex(_R, _R)]], "rx": [[c, -1j * i], [-1j * i, c]],
             "ry": [[c, -i], [i, c]], "rz": [[complex(c, -i), 0], [0, complex(c, i)]]}[t]
        _apply_1q(s, n, p["target"], m)


def _exact_state(n: int, ops: list) -> torch.Tensor:
    s = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    s[0] = 1
    _exact_ops(s, n, ops)
    return s


def _exact_cut(c: dict, n: int, edges) -> float:
    p = _exact_state(n, c["operations"]).abs().square_()
    e = 0.0
    for a, b in edges:
        v = _pair(p, n, min(a, b), max(a, b))
        e += float(v[:, 0, :, 1].sum() + v[:, 1, :, 0].sum())
    return e


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "job":
        s = _exact_state(case["qubits"], _circuit(case, seed)["operations"])
        return {"shots": None, "probabilities": s.abs().square(), "state": s}
    if kind == "circuit":
        return _exact_state(case["qubits"], _circuit(case, seed)["operations"])
    if kind == "sweep":
        cs = _sweep_circuits(case, seed)
        return torch.tensor([_exact_cut(c, c["num-qubits"], c["edges"]) for c in cs], dtype=torch.float64)
    if kind == "gradient":
        n = case["qubits"]
        edges, params = _gradient_inputs(case, seed)
        shift = variational.DEFAULT_SHIFT
        pts = [params]
        for k in range(len(params)):
            for d in (shift, -shift):
                pts.append(params[:k] + [params[k] + d] + params[k + 1:])
        e = [_exact_cut(variational.qaoa_maxcut_circuit(n, edges, p), n, edges) for p in pts]
        g = [(e[1 + 2 * k] - e[2 + 2 * k]) / (2 * math.sin(shift)) for k in range(len(params))]
        return {"energy": np.float64(e[0]), "gradient": torch.tensor(g, dtype=torch.float64)}
    if kind == "energy":
        n = case["qubits"]
        s = _exact_state(n, _circuit(case, seed)["operations"])
        e = 0.0
        for coef, text in _heisenberg(n):
            t = s.clone()
            for q, ch in enumerate(text):
                if ch != "I":
                    _exact_ops(t, n, [{"operation-type": ch.lower(), "operation-params": {"target": q}}])
            e += coef * float(torch.vdot(s, t).real)
        return np.float64(e)
    return None  # outcomes are whole numbers; measured and noisy states depend on the library's draws
