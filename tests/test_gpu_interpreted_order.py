"""Interpreted complex64 circuits keep their order of operations at every size: plans move
permutations only, so no rounding depends on the number of qubits.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _op(t, **p):
    return {"operation-type": t, "operation-params": p}


def _mixed(n, idle, count, rng, factors):
    """Gates, phases and permutations, then a transform with its swaps, on the n low bits of
    n + idle. A qubit is its bit from the top, but swap and iswap count from the bottom. factors:
    with gates whose diagonal entry is taken out and applied once, as a factor of the state."""
    out = []

    def turn(a, b):
        ang = float(rng.uniform(0, 2 * math.pi))
        if factors:
            return [_op("h", target=a), _op("rx", target=a, angle=ang), _op("ry", target=a, angle=ang)]
        return [_op("cry", control=b, target=a, angle=ang), _op("crx", control=b, target=a, angle=ang),
                _op("cry", control=b, target=a, angle=-ang)]

    for _ in range(count):
        u, v, w = (int(x) for x in rng.choice(n, 3, replace=False))
        a, b, c = u + idle, v + idle, w + idle
        ang = float(rng.uniform(0, 2 * math.pi))
        some = turn(a, b) + [_op("x", target=a), _op("s", target=a), _op("t", target=a),
                             _op("cnot", control=a, target=b), _op("cnot", control=b, target=a),
                             _op("cz", control=a, target=b), _op("rydberg-cphase", control=a, target=b, angle=ang),
                             _op("swap", qubit1=u, qubit2=v), _op("iswap", qubit1=u, qubit2=v),
                             _op("toffoli", control1=a, control2=b, target=c)]
        if factors:
            some += [_op("y", target=a), _op("rz", target=a, angle=ang), _op("rzz", qubit1=a, qubit2=b, angle=ang)]
        out.append(some[rng.integers(len(some))])
    for i in range(n):
        out.append(turn(i + idle, (i + 1) % n + idle)[0])
        for j in range(i + 1, n):
            out.append(_op("rydberg-cphase", control=j + idle, target=i + idle, angle=math.pi / (1 << (j - i))))
    return out + [_op("swap", qubit1=i, qubit2=n - 1 - i) for i in range(n // 2)]


def _random(n, rng):
    sv = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return (sv / np.linalg.norm(sv)).astype(np.complex64)


@pytest.mark.parametrize("n", [11, 12, 15, 24])
def test_an_idle_qubit_changes_no_bit(n):
    """n qubits, and the same circuit beside an idle highest qubit: the same amplitudes. (Without
    factors: passes that an idle qubit leaves open may take the factor of the state earlier.)"""
    from qclojure_gb300.state import Context

    sv = _random(n, np.random.default_rng(n))
    got = []
    with Context(pass_kernels="off", arithmetic="double-float") as ctx:
        for idle in (0, 1):
            ops = _mixed(n, idle, 150, np.random.default_rng(n), False)
            with ctx.state(n + idle, "c64") as st:
                st.upload(np.concatenate([sv, np.zeros_like(sv)]) if idle else sv)
                st.apply({"num-qubits": n + idle, "operations": ops})
                got.append(st.download())
    assert np.array_equal(got[1][: 1 << n], got[0])
    assert not np.any(got[1][1 << n:])


@pytest.mark.parametrize("n", [13, 19, 25])
def test_every_amplitude_of_a_random_state(n):
    """Against the exact arithmetic, which plans nothing. Two roundings of 2^-24 per operation, of
    amplitudes below 8 * 2^(-n/2) (2^25 Gaussian ones stay below 5): a wrong phase or place of any
    amplitude of ordinary size is a thousand times that."""
    from qclojure_gb300.state import Context

    rng = np.random.default_rng(n)
    sv = _random(n, rng)
    ops = _mixed(n, 0, 150, rng, True)
    c = {"num-qubits": n, "operations": ops}
    got = []
    for precision, arithmetic in (("c64", "double-float"), ("c128", "exact")):
        with Context(pass_kernels="off", arithmetic=arithmetic) as ctx, ctx.state(n, precision) as st:
            st.upload(sv)
            st.apply(c)
            got.append(st.download())
    assert np.max(np.abs(got[0] - got[1])) <= len(ops) * 2 * 2.0**-24 * 8 * 2.0 ** (-n / 2)
