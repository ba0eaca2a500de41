"""The fused tile form is no less exact than its gates one by one, also where
layers repeat and with them the rounding of the products: transverse-field layers
with cX-Rz-cX couplings against extended precision."""

import numpy as np
import pytest

import qforte_b200 as qb
from qforte_b200.device import gates_config

pytestmark = pytest.mark.gpu


def _layers(n, layers, a, b):
    gates = []
    for _ in range(layers):
        gates += [("Rx", q, q, a) for q in range(n)]
        for q in range(n - 1):
            gates += [("cX", q + 1, q, 0.0), ("Rz", q + 1, q + 1, b), ("cX", q + 1, q, 0.0)]
    return gates


def _exact(psi, n, gates):
    """numpy in long double, from the gates' matrices as the framework rounds them."""
    v = psi.astype(np.clongdouble)
    for name, t, c, p in gates:
        m = np.array(qb.gate(name, t, c, p).matrix())
        x = v.reshape(1 << (n - 1 - t), 2, 1 << t)
        if t == c:
            y = np.stack([m[0, 0] * x[:, 0] + m[0, 1] * x[:, 1], m[1, 0] * x[:, 0] + m[1, 1] * x[:, 1]], axis=1)
            v = y.reshape(-1)
        else:  # cX
            j = np.arange(1 << n)
            v = v[np.where(j >> c & 1, j ^ (1 << t), j)]
    return v


@pytest.mark.parametrize("n", [13, 15])
def test_fused_layers_round_no_more_than_gates(cuda, n):
    draws, layers = 10, 10
    rng = np.random.default_rng(n)
    err = {True: 0.0, False: 0.0}
    for _ in range(draws):
        gates = _layers(n, layers, float(rng.uniform(0, 3)), float(rng.uniform(0, 3)))
        circ = qb.Circuit()
        for g in gates:
            circ.add(qb.gate(*g))
        psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        psi /= np.linalg.norm(psi)
        want = _exact(psi, n, gates)
        for fused in (True, False):
            gates_config(0, 3, 0, 0, fused)
            try:
                qc = qb.Computer(n)
                qc.set_coeff_vec(psi)
                qc.apply_circuit(circ)
                got = qc.get_coeff_array()
            finally:
                gates_config()
            err[fused] += float(np.linalg.norm((got - want).astype(complex))) / draws
    print(n, err)
    # a fused product is rounded once where its gates are rounded one by one; the
    # mean of ten draws spreads by about a fifth
    assert err[True] < 1.25 * err[False], err
