"""Sums on the device that lose nothing but their values' own roundings.

Pauli strings of states with real integer amplitudes (times a power of two): every value is exact, so
the result may differ from the exact sum by its own rounding (2^-52, with the final addition's) and
by what a compensated sum leaves, below 2^-80 of the sum of magnitudes; the terms of most strings
cancel. Sizes cover one value per tile and less, a tile's edge and several tiles; strings alone, in
pairs and in larger groups. Outcome probabilities equal the correctly rounded sums of the rounded
probabilities, and the state after a measurement their scaling, bit for bit.
"""
import math
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bits", [("c128", 26), ("c64", 24)])
@pytest.mark.parametrize("n", [2, 5, 9, 12, 13, 15])
def test_strings_that_cancel(n, precision, bits):
    from qclojure_gb300.state import Context

    rng = np.random.default_rng(40 + n)
    N = 1 << n
    a = np.exp2(rng.uniform(0, bits - 0.01, N)).astype(np.int64) * rng.choice([-1, 1], N)
    a[N // 2:] = a[:N // 2][::-1] + rng.integers(-1, 1, N // 2)  # nearly the same on i and its complement
    scale = 0.5 ** (bits + n // 2)
    pad = lambda q, s: "I" * q + s + "I" * (n - q - len(s))
    strings = [pad(q, "Z") for q in range(n)] + [pad(q, s) for q in range(n - 1) for s in ("XX", "YY", "ZZ")]
    strings += [pad(q, "XZ") for q in range(n - 1)] + ["Z" * n, "X" * n]
    i, obj = np.arange(N), a.astype(object)
    with Context() as ctx, ctx.state(n, precision) as st:
        st.upload(a * scale + 0j)
        for t in strings:
            x = sum(1 << (n - 1 - q) for q, ch in enumerate(t) if ch in "XY")
            sign = np.ones(N, np.int64) * (-1) ** (t.count("Y") // 2)
            for q, ch in enumerate(t):
                if ch in "YZ":
                    sign = sign * (1 - 2 * ((i >> (n - 1 - q)) & 1))
            v = obj * obj[i ^ x] * sign
            unit = Fraction(scale) ** 2
            want, size = unit * int(v.sum()), unit * int(np.abs(v).sum())
            tol = abs(want) / 2**52 + size / 2**80
            others = [(1.0, s) for s in strings if s != t]
            alone = st.pauli_expectation(t)
            among = st.hamiltonian([(1.0, t)] + [(0.0, s) for _, s in others])
            for got in (alone, among):
                assert abs(Fraction(got) - want) <= tol, (t, got, float(want))


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("n,qubits", [(3, [1]), (11, [10, 2]), (13, [0]), (15, [7, 14, 3])])
def test_measured_probabilities(n, qubits, precision):
    from qclojure_gb300.state import Context

    rng = np.random.default_rng(60 + n)
    real = np.float32 if precision == "c64" else np.float64
    with Context() as ctx, ctx.state(n, precision) as st:
        for seed in range(1, 17):
            sv = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
            if n > 8 and seed % 2:  # few amplitudes, all in one thread's groups
                sv[np.arange(1 << n) % 256 != 5] = 0
            sv /= np.linalg.norm(sv)
            st.upload(sv)
            held = st.download()
            p = held.real * held.real + held.imag * held.imag
            got, prob = st.measure(qubits, seed)
            keep = np.ones(1 << n, bool)
            for k, q in enumerate(qubits):
                keep &= ((np.arange(1 << n) >> (n - 1 - q)) & 1) == (got >> k) & 1
            assert prob == math.fsum(p[keep])
            f = real(1.0 / math.sqrt(prob))
            after = st.download()
            for part in ("real", "imag"):
                want = np.where(keep, getattr(held, part).astype(real) * f, real(0))
                assert np.array_equal(getattr(after, part), want)
