"""Expectations of many Pauli strings in one launch against numpy on the same amplitudes.

Sizes cover one value per tile and less (1-5 qubits), the tile's edges (11-13) and several
tiles; string sets cover one and two strings per group (with equal and differing sign patterns
in registers), the transform (three and more), and groups of more than 256 strings. Tolerance:
the reductions' contract of 1e-12 on a unit state.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _apply(sv, n, text):
    i = np.arange(sv.size)
    x = sum(1 << (n - 1 - q) for q, ch in enumerate(text) if ch in "XY")
    z = sum(1 << (n - 1 - q) for q, ch in enumerate(text) if ch in "YZ")
    sign = np.ones(sv.size)
    for b in range(n):
        if z >> b & 1:
            sign = sign * (1 - 2 * ((i >> b) & 1))
    return ((-1j) ** (text.count("Y") % 4)) * sign * sv[i ^ x]


def _strings(n, kind, rng):
    if kind == "chain":  # XX and YY share a group; Z and ZZ the transform
        out = [p if n == 1 else "I" * q + p + p + "I" * (n - q - 2) for p in "XYZ" for q in range(max(1, n - 1))]
        return out + ["I" * q + "Z" + "I" * (n - q - 1) for q in range(n)]
    if kind == "any":
        return ["".join("IXYZ"[k] for k in rng.integers(0, 4, n)) for _ in range(24)] + ["I" * n, "Y" * n, "X" * n]
    if kind == "many-z":  # more strings than one group holds
        return ["".join("IZ"[k] for k in rng.integers(0, 2, n)) for _ in range(300)]
    x = rng.integers(0, 2, n)  # one x mask, Re and Im parts, three to nine strings each
    x[rng.integers(0, n)] = 1
    return ["".join(("XY" if b else "IZ")[k] for b, k in zip(x, rng.integers(0, 2, n))) for _ in range(12)]


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("kind", ["chain", "any", "many-z", "one-x"])
@pytest.mark.parametrize("n", [1, 2, 5, 9, 12, 13, 14, 17])
def test_pauli_strings(n, kind, precision):
    from qclojure_gb300.state import Context

    rng = np.random.default_rng(1000 * n + len(kind))
    sv = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    sv /= np.linalg.norm(sv)
    strings = _strings(n, kind, rng)
    coefs = rng.uniform(-1, 1, len(strings))
    with Context() as ctx, ctx.state(n, precision) as st:
        st.upload(sv)
        sv = st.download()  # complex64: what the device holds
        want = np.array([np.vdot(sv, _apply(sv, n, t)).real for t in strings])
        energy = st.hamiltonian(list(zip(coefs.tolist(), strings)))
        assert abs(energy - float(np.dot(coefs, want))) <= 1e-12 * len(strings)
        for k in range(0, len(strings), max(1, len(strings) // 6)):
            assert abs(st.pauli_expectation(strings[k]) - want[k]) <= 1e-12, strings[k]
