"""Explicit 2x2 gates [[0, a], [b, 0]] of entries that differ in size, unitary or not, against the
oracle within the contract (1e-12, 2e-5) of the largest amplitude.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("c128", 1e-12), ("c64", 2e-5)])
@pytest.mark.parametrize("a,b", [(1.0, 1e-60), (1e-60, 1.0), (1e-45j, 1e-45), (1.0, 1e-25), (0.0, 1e-30), (3.0, 0.5j), (-1j, 1j), (0.6 + 0.8j, -1)])
def test_antidiagonal_gates(oracle, a, b, precision, tol):
    from qclojure_gb300.state import Context

    n = 6
    ops = [{"operation-type": "h", "operation-params": {"target": q}} for q in range(n)]
    ops.append({"operation-type": "t", "operation-params": {"target": 3}})
    ops.append({"operation-type": "u", "operation-params": {"target": 2, "matrix": [[0, a], [b, 0]]}})
    ops.append({"operation-type": "s", "operation-params": {"target": 2}})
    c = {"num-qubits": n, "operations": ops}
    want = oracle.run(c)
    for fusion in ("tiled", "plain"):
        with Context(arithmetic="double-float") as ctx, ctx.state(n, precision) as st:
            st.apply(c, fusion=fusion)
            got = st.download()
        assert np.max(np.abs(got - want)) <= tol * max(1.0, np.max(np.abs(want)))
