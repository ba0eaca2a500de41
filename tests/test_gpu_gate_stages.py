"""Gate runs whose phases hold more ops than a CTA stages, runs of many phases,
and more windows than one planning group, against the oracle: tiles of 5 to 12
bits, the default tiles on both sides of the fused form's line."""

import math

import numpy as np
import pytest

import qforte_b200 as qb
from oracle import oracle as O
from qforte_b200.device import gate_plan, gates_config

pytestmark = pytest.mark.gpu

ONE = ("H", "X", "Y", "Z", "S", "T", "Rx", "Ry", "Rz")
TWO = ("cX", "cZ", "SWAP", "cR", "cV")


def _circuit(n, ngates, hot, seed):
    """Random gates, nine of ten one-qubit ones on the first `hot` qubits."""
    rng = np.random.default_rng(seed)
    circ, ora = qb.Circuit(), []
    for _ in range(ngates):
        if rng.random() < 0.7:
            k = ONE[rng.integers(len(ONE))]
            t = c = int(rng.integers(hot if rng.random() < 0.9 else n))
        else:
            k = TWO[rng.integers(len(TWO))]
            t, c = (int(v) for v in rng.choice(n, 2, replace=False))
        p = float(rng.uniform(0, 4 * math.pi))
        circ.add(qb.gate(k, t, c, p))
        ora.append(O.make_gate(k, t, c, p))
    return circ, ora


@pytest.mark.parametrize("n,ngates,hot,tile,low", [
    (4, 150, 2, 0, 3), (5, 200, 2, 5, 3), (9, 250, 3, 9, 3), (11, 200, 3, 0, 3), (12, 300, 12, 0, 3),
    (12, 200, 4, 12, 6), (14, 400, 14, 0, 3), (14, 400, 14, 8, 3), (19, 120, 19, 0, 3), (20, 250, 20, 0, 3),
])
def test_runs_match_oracle(cuda, n, ngates, hot, tile, low):
    circ, ora = _circuit(n, ngates, hot, n + ngates)
    rng = np.random.default_rng(n)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi /= np.linalg.norm(psi)
    gates_config(tile, low)
    try:
        if n == 14 and tile == 8:
            assert gate_plan(circ.gates(), n)[0] > 12  # more than the first groups of windows
        qc = qb.Computer(n)
        qc.set_coeff_vec(psi)
        qc.apply_circuit(circ)
        got = qc.get_coeff_array()
    finally:
        gates_config()
    st = O.State(n, psi.copy())
    st.apply_gates(ora)
    # a few hundred 64-bit gates on amplitudes below 1
    assert np.max(np.abs(got - st.psi)) < 1e-12
