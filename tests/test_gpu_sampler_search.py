"""Shot sampling where its search and scan change shape: states smaller than a chunk, one block,
a few blocks, and more blocks than one step of the scan takes; one shot, a warp's worth and one
more, and enough shots for batches. Outcomes are integers and equal the oracle's.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rule(oracle, sv, shots, seed):
    """The oracle's rule on its own draws (its sampler refuses the norm of a complex64 state):
    the first i whose cumulative floor(p 2^62) exceeds floor(draw T / 2^64)."""
    p = sv.real * sv.real + sv.imag * sv.imag
    cum, T = [], 0
    for x in p.tolist():
        T += int(x * 2.0 ** 62)
        cum.append(T)
    cum = np.array(cum, np.uint64)
    draws = [oracle.lib().or_draw64(seed, j, 0) for j in range(shots)]
    u = np.array([(d * T) >> 64 for d in draws], np.uint64)
    return np.searchsorted(cum, u, side="right").astype(np.uint64)


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("n,shots", [(1, 33), (4, 1000), (5, 1), (6, 32), (12, 2000), (13, 20000), (14, 33), (18, 50000),
                                     (19, 20001)])
def test_outcomes_equal_the_oracle(oracle, n, shots, precision):
    from qclojure_gb300.state import Context

    rng = np.random.default_rng(n)
    sv = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    sv[rng.random(1 << n) < 0.3] = 0  # zeros, so that cumulative sums repeat
    sv[0] += 1
    sv /= np.linalg.norm(sv)
    with Context() as ctx, ctx.state(n, precision) as st:
        st.upload(sv)
        got, held = st.sample(shots, 7), st.download()
    assert np.array_equal(got, _rule(oracle, held, shots, 7))
    if precision == "c128":
        assert np.array_equal(got, oracle.sample(held, shots, 7))


def test_many_blocks_and_batches():
    """A uniform state's outcome is the top bits of the draw, so 28 and 20 qubits agree on 20."""
    from qclojure_gb300.state import Context

    got = []
    with Context() as ctx:
        for n in (20, 28):
            with ctx.state(n, "c64") as st:
                st.apply({"num-qubits": n, "operations": [{"operation-type": "h", "operation-params": {"target": q}}
                                                          for q in range(n)]})
                assert st.norm2() == 1.0  # amplitudes are the power of two exactly
                got.append(st.sample(100_001, 3))
    assert np.array_equal(got[1] >> np.uint64(8), got[0])


@pytest.mark.parametrize("precision,tol", [("c128", 1e-12), ("c64", 2e-5)])
def test_sweep_energies_over_chunk_counts(precision, tol):
    """Diagonal energies with four coefficients at 1, 2, 32 and 64 chunks per state."""
    from qclojure_gb300 import workloads
    from qclojure_gb300.state import Context
    from qclojure_gb300.sweep import Sweep

    ns = [12, 13, 17, 18]
    circuits = [workloads.layered_circuit(n, 3, n) for n in ns]
    terms = []
    for n in ns:
        z = lambda *qs: "".join("Z" if q in qs else "I" for q in range(n))  # noqa: E731,B023
        terms.append([{"coefficient": 0.5, "pauli-string": z()}, {"coefficient": -0.25, "pauli-string": z(0, n - 1)},
                      {"coefficient": 1.5, "pauli-string": z(1)}, {"coefficient": 2.0, "pauli-string": z(2, 3, 4)},
                      {"coefficient": -0.25, "pauli-string": z(5, 6)}])
    with Context() as ctx, Sweep(ctx, circuits, precision) as sw:
        got, _ = sw.run(terms)
        for c, n in enumerate(ns):
            p = np.abs(sw.state(c)) ** 2
            i, want = np.arange(1 << n), 0.0
            for t in terms[c]:
                sign = np.ones(1 << n)
                for q, ch in enumerate(t["pauli-string"]):
                    if ch == "Z":
                        sign *= 1 - 2 * ((i >> (n - 1 - q)) & 1)
                want += t["coefficient"] * float(np.dot(sign, p))
            assert abs(got[c] - want) <= tol * 5


def test_same_draws_over_every_depth_of_the_block_search():
    """Uniform states of 1, 32, 64, 1024, 2048, 4096, 8192 and 2^18 blocks: one to three packed
    levels of the search and none, one or two steps below them. T = 2^62 for each, so shot k
    picks the same leading index bits for all of them."""
    from qclojure_gb300.state import Context

    want = None
    with Context() as ctx:
        for n in (13, 18, 19, 23, 24, 25, 26, 31):
            with ctx.state(n, "c64") as st:
                st.apply({"num-qubits": n, "operations": [{"operation-type": "h", "operation-params": {"target": q}}
                                                          for q in range(n)]})
                got = st.sample(3001, 9) >> np.uint64(n - 13)
            want = got if want is None else want
            assert np.array_equal(got, want)


def test_complex64_sums_over_the_fixed_point_range():
    """Chunk sums of complex64 parts from 2^-149 to just below 2^-10 (whole warps stay on the
    fixed-point path): around 2^-18 and 2^-41, where its terms vanish, powers of two, zeros;
    then chunks with a part at 2^-10, a NaN and an infinity. Integers: no tolerance."""
    from qclojure_gb300.state import Context

    rng = np.random.default_rng(5)
    N = 1 << 16
    v = np.exp2(rng.uniform(-46, -10, (N, 2))).astype(np.float32)
    v[:8192] = np.exp2(-18.0) * (1 + rng.integers(-40, 41, (8192, 2)) * 2.0**-24)
    v[8192:16384] = np.exp2(-41.0) * (1 + rng.integers(-40, 41, (8192, 2)) * 2.0**-24)
    v[16384:24576] = np.exp2(rng.integers(-149, -10, (8192, 2)).astype(np.float64))
    v[24576:28672, 0] = 0
    v = np.minimum(v, np.nextafter(np.float32(2.0**-10), np.float32(0)))
    v *= rng.choice([np.float32(-1), np.float32(1)], (N, 2))
    v[40000, 1] = 2.0**-10
    a = v.view(np.complex64).ravel()
    with Context() as ctx, ctx.state(16, "c64") as st:
        for special in (None, np.nan, np.inf):
            if special is not None:
                a = a.copy()
                a[50000] = special
            st.upload(a.astype(np.complex128))
            got, total = st.sample_sums()
            with np.errstate(invalid="ignore", over="ignore"):
                w = st.download().astype(np.complex128)
                p = w.real * w.real + w.imag * w.imag
                q = [0 if x != x else min(int(x * 2.0**62) if x < 4 else 2**64 - 1, 2**64 - 1) for x in p]
            want = [sum(q[c:c + 32]) % 2**64 for c in range(0, N, 32)]
            assert got.tolist() == want
            assert total == sum(want) % 2**64
