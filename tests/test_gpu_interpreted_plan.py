"""The interpreter's planned passes (permutations in layout changes, phase runs) against the
oracle: states of less than one warp per tile, of one tile, and with tile bits that control
permutations and phases; circuits of permutations only, of phases only, with permutations at the
end, and QFTs with swaps. Tolerances are the contracts: 1e-12 and 2e-5 per amplitude.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _op(t, **p):
    return {"operation-type": t, "operation-params": p}


def _some(n, count, gates, rng):
    out = []
    for _ in range(count):
        a, b, c = (int(x) for x in rng.choice(n, 3, replace=False))
        ang = float(rng.uniform(0, 2 * math.pi))
        out.append({"x": _op("x", target=a), "y": _op("y", target=a), "z": _op("z", target=a), "s": _op("s", target=a),
                    "t": _op("t", target=a), "h": _op("h", target=a), "rx": _op("rx", target=a, angle=ang),
                    "ry": _op("ry", target=a, angle=ang), "rz": _op("rz", target=a, angle=ang),
                    "cnot": _op("cnot", control=a, target=b), "cz": _op("cz", control=a, target=b),
                    "cphase": _op("rydberg-cphase", control=a, target=b, angle=ang),
                    "swap": _op("swap", qubit1=a, qubit2=b), "iswap": _op("iswap", qubit1=a, qubit2=b),
                    "toffoli": _op("toffoli", control1=a, control2=b, target=c),
                    "fredkin": _op("fredkin", control=a, target1=b, target2=c),
                    "rzz": _op("rzz", qubit1=a, qubit2=b, angle=ang)}[gates[rng.integers(len(gates))]])
    return out


_PERM = ["x", "cnot", "cnot", "swap"]
_PHASE = ["z", "s", "t", "rz", "cz", "cphase"]
_ALL = _PERM + _PHASE + ["y", "h", "rx", "ry", "iswap", "toffoli", "fredkin", "rzz"]


@pytest.mark.parametrize("precision,tol", [("c128", 1e-12), ("c64", 2e-5)])
@pytest.mark.parametrize("n", [5, 6, 8, 11, 12, 13, 14, 17])
def test_interpreted_plans(oracle, n, precision, tol):
    from qclojure_gb300 import workloads
    from qclojure_gb300.state import Context

    rng = np.random.default_rng(700 + n)
    sv = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    sv /= np.linalg.norm(sv)
    circuits = [_some(n, 25, _PERM, rng), _some(n, 40, _PHASE, rng),
                _some(n, 30, _ALL, rng) + _some(n, 10, _PERM, rng), _some(n, 400, _ALL, rng),
                workloads.qft_ops(n) + _some(n, 5, _PERM + _PHASE, rng)]
    with Context(pass_kernels="off", arithmetic="double-float") as ctx, ctx.state(n, precision) as st:
        for ops in circuits:
            c = {"num-qubits": n, "operations": ops}
            st.upload(sv)
            _, kinds = st.profile(c)
            assert np.all(kinds == 1)
            assert np.max(np.abs(st.download() - oracle.run(c, sv))) <= tol


@pytest.mark.parametrize("precision,tol", [("c128", 1e-12), ("c64", 2e-5)])
@pytest.mark.parametrize("n", [5, 9, 12])
def test_small_jobs(oracle, n, precision, tol):
    """The same plans in the job kernels, which hold the whole state in one tile."""
    from qclojure_gb300.backend import create_simulator, execute_circuit

    rng = np.random.default_rng(900 + n)
    c = {"num-qubits": n, "operations": _some(n, 200, _ALL, rng) + _some(n, 6, _PERM, rng)}
    for loop in ("on", "off"):
        sim = create_simulator({"precision": precision, "small-job-loop": loop})
        try:
            r = execute_circuit(sim, c, {"result-specs": {"state-vector": True}})["results"]
            sv = np.asarray(r["state-vector-result"]["state-vector"])
            assert np.max(np.abs(sv - oracle.run(c))) <= tol
        finally:
            sim.close()


def test_complex64_plans_of_large_states():
    """complex64 is planned from 25 qubits on, two tiles per dispatch: phases over thread and tile
    bits, permutations, gates, against the same circuit in complex128. Tolerance: two roundings
    of 2^-24 per operation."""
    from qclojure_gb300 import workloads
    from qclojure_gb300.state import Context

    n = 25
    rng = np.random.default_rng(25)
    ops = _some(n, 60, _PHASE, rng) + [_op("h", target=q) for q in range(n)] + _some(n, 150, _ALL, rng)
    ops += workloads.qft_ops(n) + _some(n, 10, _PERM, rng)
    c = {"num-qubits": n, "operations": ops}
    got = []
    with Context(pass_kernels="off", arithmetic="double-float") as ctx:
        for precision in ("c64", "c128"):
            with ctx.state(n, precision) as st:
                st.apply(c)
                got.append(st.download())
    assert np.linalg.norm(got[0] - got[1]) <= len(ops) * 2 * 2.0**-24
