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
