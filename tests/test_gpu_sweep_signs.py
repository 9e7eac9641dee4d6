"""A complex128 sweep whose members' rotation angles lie on both sides of zero runs as specialised
kernels (the sign of a sine is a value, not a structure), before and after an update that moves
them across; a complex64 one stays interpreted. Energies equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("c128", 1e-10), ("c64", 2e-4)])
def test_angles_of_both_signs_share_kernels(oracle, precision, tol):
    from qclojure_gb300 import variational, workloads
    from qclojure_gb300.state import Context
    from qclojure_gb300.sweep import Sweep

    n = 12
    edges = workloads.random_3_regular_graph(n, np.random.default_rng(3))
    ham = [{"coefficient": -0.5, "pauli-string": "".join("Z" if q in e else "I" for q in range(n))} for e in edges]

    def circuits(shift):
        return [variational.qaoa_maxcut_circuit(n, edges, [0.4 + shift, s * 0.3 + shift, -0.7, s * 1.1])
                for s in (1, -1, 0.5)]

    with Context() as ctx, Sweep(ctx, circuits(0.0), precision) as sw:
        for shift in (0.0, -1.0, 0.25):
            cs = circuits(shift)
            sw.update(cs)
            got, stats = sw.run([ham] * len(cs))
            assert stats["groups"] == 1
            assert stats["specialised"] == (1 if precision == "c128" else 0)
            for e, c in zip(got, cs):
                ref = oracle.run(c)
                want = sum(t["coefficient"] * oracle.pauli_expectation(ref, t["pauli-string"]) for t in ham)
                assert abs(e - want) <= tol
