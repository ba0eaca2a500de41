"""Circuits that take smaller tiles than others on a large state: gates on seven, and
on eight, of the qubits above the lowest three, and one-qubit gates on all qubits,
against tiles of 11 bits and one pass per gate."""

import numpy as np
import pytest

import qforte_b200 as qb
from qforte_b200.device import gates_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("low_bits", [3, 6])
@pytest.mark.parametrize("high", [1, 7, 8, 0])
def test_few_qubits_of_a_large_state(cuda, high, low_bits):
    n = 23
    rng = np.random.default_rng(high)
    qubits = [0, 2] + [int(q) for q in rng.choice(np.arange(3, n), high, replace=False)]
    circ = qb.Circuit()
    for k in range(40 if high else 0):
        if k % 3:
            circ.add(qb.gate(("H", "T", "Rx", "Ry")[int(rng.integers(4))],
                             *([qubits[int(rng.integers(len(qubits)))]] * 2), float(rng.uniform(0, 6))))
        else:
            t, c = (int(q) for q in rng.choice(qubits, 2, replace=False))
            circ.add(qb.gate(("cX", "cRz", "SWAP", "cZ")[int(rng.integers(4))], t, c, float(rng.uniform(0, 6))))
    for k in range(0 if high else 60):  # one-qubit gates on all of them
        circ.add(qb.gate(("H", "T", "Rx", "Ry")[k % 4], k % n, k % n, float(rng.uniform(0, 6))))
    out = []
    for tile in (0, 11, -1):
        gates_config(tile, low_bits)
        try:
            qc = qb.Computer(n)
            spread = qb.Circuit()
            for q in range(n):
                spread.add(qb.gate("Ry", q, q, 0.3 + 0.1 * q))
            qc.apply_circuit(spread)
            qc.apply_circuit(circ)
            out.append(qc.get_coeff_array().copy())
        finally:
            gates_config()
    # some eighty 64-bit gates on amplitudes below 1
    assert np.max(np.abs(out[0] - out[2])) < 1e-13 and np.max(np.abs(out[1] - out[2])) < 1e-13
