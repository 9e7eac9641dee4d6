"""Specialised double-float and complex64 passes: one gate between the conversions from and to
IEEE doubles (every gate form of the generator on its own, where a packed product meets the
store's sum directly), and tile shapes at the edges of their range, against the oracle.
Tolerances are the contracts of the two precisions: 1e-12 and 2e-5 per amplitude.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_GATES = ["h", "x", "y", "z", "s", "s-dag", "t", "t-dag", ("rx", 0.7), ("rx", 2.9), ("ry", 0.7), ("ry", 2.9),
          ("rz", 0.7), ("phase", 0.7), ("phase", np.pi / 4), ("global-ry", 0.3)]


def _random(n, seed):
    rng = np.random.default_rng(seed)
    sv = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return sv / np.linalg.norm(sv)


@pytest.mark.parametrize("gate", _GATES)
def test_one_gate_between_conversions(oracle, gate):
    from qclojure_gb300.state import Context

    n = 12
    name, angle = gate if isinstance(gate, tuple) else (gate, None)
    sv = _random(n, 5)
    with Context(pass_kernels="always", arithmetic="double-float") as ctx, ctx.state(n) as st:
        for q in (0, 5, 11):
            p = {"target": q} if angle is None else {"target": q, "angle": angle}
            c = {"num-qubits": n, "operations": [{"operation-type": name, "operation-params": p}]}
            st.upload(sv)
            st.apply(c)
            assert np.max(np.abs(st.download() - oracle.run(c, sv))) <= 1e-12, (gate, q)


@pytest.mark.parametrize("n,precision,shape", [
    (10, "c128", (10, 3, 2, 4)), (11, "c128", (10, 3, 2, 4)), (13, "c128", (10, 3, 1, 4)), (13, "c128", (12, 3, 2, 1)),
    (22, "c128", None), (11, "c64", (10, 4, 2, 8)), (13, "c64", (13, 4, 2, 1)), (14, "c64", (11, 3, 2, 4)),
    (22, "c64", None)])
def test_shapes_and_defaults(oracle, n, precision, shape):
    from qclojure_gb300 import workloads
    from qclojure_gb300.state import Context

    c = workloads.layered_circuit(n, 3, seed=40 + n)
    c = {"num-qubits": n, "operations": c["operations"] + workloads.qft_ops(n)}
    with Context(pass_kernels="always", arithmetic="double-float") as ctx:
        if shape:
            ctx.set_tuning(n, precision, *shape)
        with ctx.state(n, precision) as st:
            ms, kinds = st.profile(c)
            assert len(ms) > 0 and np.all(kinds == 3)
            got = st.download()
    assert np.max(np.abs(got - oracle.run(c))) <= (1e-12 if precision == "c128" else 2e-5)


@pytest.mark.parametrize("n,precision,shape", [
    (10, "c128", (10, 3, 2, 4)), (13, "c128", (10, 3, 2, 4)), (14, "c128", (12, 3, 2, 1)), (12, "c64", (12, 4, 2, 2)),
    (14, "c64", (11, 4, 2, 4)), (13, "c64", (10, 3, 2, 8))])
def test_index_permutations(oracle, n, precision, shape):
    """X, CNOT, SWAP, Toffoli and controlled swaps between gates that need registers: maps of
    layout changes with local and tile controls, at the start and the end of a pass, bit 0 of
    8-byte amplitudes among the targets, and passes of permutations only."""
    from qclojure_gb300.state import Context

    rng = np.random.default_rng(n)
    op = lambda t, **p: {"operation-type": t, "operation-params": p}

    def some(count, gates):
        ops = []
        for _ in range(count):
            a, b, c = (int(x) for x in rng.choice(n, 3, replace=False))
            g = gates[rng.integers(len(gates))]
            ops.append({"x": lambda: op("x", target=a), "y": lambda: op("y", target=a),
                        "cnot": lambda: op("cnot", control=a, target=b),
                        "swap": lambda: op("swap", qubit1=a, qubit2=b),
                        "iswap": lambda: op("iswap", qubit1=a, qubit2=b),
                        "toffoli": lambda: op("toffoli", control1=a, control2=b, target=c),
                        "fredkin": lambda: op("fredkin", control=a, target1=b, target2=c),
                        "h": lambda: op("h", target=a), "t": lambda: op("t", target=a),
                        "ry": lambda: op("ry", target=a, angle=float(rng.uniform(0, 6)))}[g]())
        return ops

    perms = ["x", "cnot", "cnot", "cnot", "swap"]
    sv = _random(n, 100 + n)
    with Context(pass_kernels="always", arithmetic="double-float") as ctx:
        ctx.set_tuning(n, precision, *shape)
        for ops in (some(30, perms), some(8, perms) + some(40, perms + ["h", "t", "ry", "y"]) + some(8, perms),
                    some(60, perms + ["toffoli", "fredkin", "iswap", "h"])):
            c = {"num-qubits": n, "operations": ops}
            with ctx.state(n, precision) as st:
                st.upload(sv)
                st.apply(c)
                got = st.download()
            assert np.max(np.abs(got - oracle.run(c, sv))) <= (1e-12 if precision == "c128" else 2e-5)
