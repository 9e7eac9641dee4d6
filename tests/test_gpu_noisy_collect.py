"""Final states of noisy runs, collected a batch (65536 shots) at a time: a whole batch of one-qubit
states, and five qubits across a batch's end, against the oracle. Tolerances are the contracts:
1e-12 and 2e-5 per amplitude.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NOISE = {"gate-noise": {"h": {"noise-type": "depolarizing", "noise-strength": 0.3},
                        "cnot": {"noise-type": "depolarizing", "noise-strength": 0.2}}}


@pytest.mark.parametrize("n,shots", [(1, 65536), (5, 65539)])
def test_a_batch_of_final_states(oracle, n, shots):
    from qclojure_gb300.hardware import run_trajectories
    from qclojure_gb300.state import Context

    ops = [{"operation-type": "h", "operation-params": {"target": 0}}]
    ops += [{"operation-type": "cnot", "operation-params": {"control": q, "target": q + 1}} for q in range(n - 1)]
    c = {"num-qubits": n, "operations": ops}
    _, states = oracle.noisy_shots(c, NOISE, shots, seed=31)
    with Context() as ctx:
        for precision, tol in (("c128", 1e-12), ("c64", 2e-5)):
            run = run_trajectories(ctx, c, NOISE, shots, seed=31, precision=precision, max_trajectories=shots)
            assert run["trajectories"].shape == states.shape
            assert np.max(np.abs(run["trajectories"] - states)) <= tol
            assert np.max(np.abs(run["final_state"] - states[-1])) <= tol
