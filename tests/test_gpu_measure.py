"""Measurement with collapse on the device: one outcome and many, repeated qubits, the highest and
lowest bits, states smaller than a chunk of the sums and with several chunks per outcome. The
outcome equals the integer rule on the oracle's draw (the first outcome whose cumulative
floor(p 2^62) exceeds floor(draw T / 2^64)); the state is the projection within 1e-12
(complex128) or 2e-5 (complex64).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("c128", 1e-12), ("c64", 2e-5)])
@pytest.mark.parametrize("n,qubits", [
    (1, [0]), (2, [1, 0]), (5, [4]), (9, [8, 0, 3]), (13, [0]), (13, [12, 0, 7, 3]), (14, [2, 5, 2]), (14, [3, 1, 3, 0, 1]),
    (15, list(range(11))), (17, [16, 15, 0, 1, 2]), (17, [6])])
def test_measure(oracle, n, qubits, precision, tol):
    from qclojure_gb300.state import Context

    rng = np.random.default_rng(10 * n + len(qubits))
    sv = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    sv[rng.random(1 << n) < 0.2] = 0
    sv[-1] += 1
    sv /= np.linalg.norm(sv)
    with Context() as ctx, ctx.state(n, precision) as st:
        for seed in (1, 2, 3):
            st.upload(sv)
            held = st.download()
            p = held.real * held.real + held.imag * held.imag
            outcome = np.zeros(1 << n, np.int64)
            for k, q in enumerate(qubits):
                outcome |= ((np.arange(1 << n) >> (n - 1 - q)) & 1) << k
            sums: dict[int, int] = {}
            for o, x in zip(outcome.tolist(), p.tolist()):
                sums[o] = sums.get(o, 0) + int(x * 2.0 ** 62)
            u, c = (oracle.lib().or_draw64(seed, 0, 1) * sum(sums.values())) >> 64, 0
            for o in sorted(sums):
                c += sums[o]
                if c > u:
                    break
            got, prob = st.measure(qubits, seed)
            keep = outcome == o
            assert got == o and abs(prob - p[keep].sum()) <= tol
            want = np.where(keep, held / np.sqrt(p[keep].sum()), 0)
            assert np.max(np.abs(st.download() - want)) <= tol


def test_measurements_inside_a_circuit(oracle):
    from qclojure_gb300 import workloads
    from qclojure_gb300.state import Context

    n, ops = 13, []
    for r, qs in enumerate(([0], [12, 3], [5, 5, 1])):
        ops += workloads.layered_circuit(n, 2, 50 + r)["operations"]
        ops.append({"operation-type": "measure", "operation-params": {"measurement-qubits": qs}})
    c = {"num-qubits": n, "operations": ops}
    for arithmetic in ("exact", "double-float"):
        with Context(arithmetic=arithmetic) as ctx, ctx.state(n) as st:
            st.apply(c, seed=9)
            assert np.max(np.abs(st.download() - oracle.run(c, seed=9))) <= 1e-12
