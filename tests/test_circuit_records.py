"""EncodedCircuit's packed records against encode_operation's structures, byte for byte, for
every gate name a program can use and for operands that take the general path."""
import pytest

from qclojure_gb300 import circuit as qc

_NAMES = sorted(set(qc.GATE_ALIASES) | set(qc.GATE_ALIASES.values()) | qc._SINGLE | qc._ROT | qc._GLOBAL | {
    "cnot", "cz", "crx", "cry", "crz", "swap", "iswap", "toffoli", "fredkin", "rydberg-cz", "rydberg-cphase",
    "rydberg-blockade", "rzz", "u", "measure", "controlled", "i", "cy"})
_FULL = {"target": 3, "control": 1, "qubit1": 0, "qubit2": 4, "control1": 1, "control2": 2, "target1": 0, "target2": 4,
         "qubit-indices": [0, 2], "measurement-qubits": [4, 1], "matrix": [[0, 1], [1, 0]], "control-qubits": [0],
         "target-gate": "x", "target-qubits": [1]}


def _by_structs(op):
    try:
        return b"".join(bytes(s) for s in qc.encode_operation(op)), None
    except Exception as e:  # noqa: BLE001
        return None, (type(e), str(e))


@pytest.mark.parametrize("name", _NAMES)
def test_records_equal_structs(name):
    for change in ({}, {"angle": 0.25}, {"angle": 2}, {"angle": None}, {"target": None}, {"target": 255},
                   {"target": 256}, {"target": -1}, {"target": True}, {"target": 1.0}, {"control": "a"},
                   {"qubit2": None}, {"angle": "x"}):
        op = {"operation-type": name, "operation-params": {**_FULL, "angle": 1.5, **change}}
        for o in (op, {"operation-type": name}, {"operation-type": name, "operation-params": None}):
            want, error = _by_structs(o)
            c = {"num-qubits": 5, "operations": [o, {"operation-type": "h", "operation-params": {"target": 2}}]}
            if error:
                with pytest.raises(error[0]) as e:
                    qc.encode(c)
                assert str(e.value) == error[1]
            else:
                enc = qc.encode(c)
                got = bytes(enc.array)
                assert got[:len(want)] == want and enc.count == len(want) // 120 + 1
