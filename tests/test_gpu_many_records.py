"""Programs of many steps whose patterns differ in their coefficients: each takes a
record of its own in the shared-memory kernels, and where the records outgrow
shared memory the evaluator takes its states to global memory."""

import types

import numpy as np
import pytest

import qforte_b200 as qb
from qforte_b200.device import DeviceProg
from qforte_b200.ucc import DUCC, Evaluator, evaluator_config

pytestmark = pytest.mark.gpu


def _program(steps, seed):
    """Hops between orbitals of one spin whose sign is that of (1 + Z_r + Z_s - Z_r
    Z_s) / 2 on two qubits of the other: one rotation angle, from coefficients that
    agree between the occupations of r and s to their rounding (4e-14) only."""
    rng = np.random.default_rng(seed)
    x, z, c, par = [], [], [], []
    for k in range(steps):
        spin = int(rng.integers(2))
        p, q = (2 * int(v) + spin for v in rng.choice(4, 2, replace=False))
        r, s = (2 * int(v) + 1 - spin for v in rng.choice(4, 2, replace=False))
        g = float(rng.uniform(0.5, 1.5))
        for zp, sign in ((1 << p, 1.0), (1 << q, -1.0)):
            for zz, f in ((0, 0.5), (1 << r, 0.5 + 2e-14), (1 << s, 0.5), (1 << r | 1 << s, -0.5)):
                x.append(1 << p | 1 << q)
                z.append(zp ^ zz)
                c.append(0.5 * sign * f * g)
                par.append(k)
    return DeviceProg(x, z, c, par, steps)


@pytest.mark.parametrize("mode", [True, "complex"])
@pytest.mark.parametrize("steps", [40, 1600])
def test_records_of_many_coefficients(cuda, mode, steps):
    mol = qb.random_molecule(4, 4, seed=11)
    pool = qb.SQOpPool()
    pool.set_orb_spaces(mol.hf_reference)
    pool.fill_pool("SD")
    eng = DUCC(mol.hamiltonian, pool, [0], mol.hf_reference)
    dp = _program(steps, steps)
    problem = types.SimpleNamespace(fwd=dp, grad_prog=dp, unrot_prog=dp, H=eng.H, nqubit=8,
                                    ref_index=eng.ref_index, nparam=steps)
    P = np.random.default_rng(1).uniform(-0.2, 0.2, (3, steps))

    def run(m):
        evaluator_config(m)
        try:
            ev = Evaluator(problem, 3)
        finally:
            evaluator_config(True)
        return (ev.path,) + ev.eval(P, True)

    path, E, G = run(mode)
    ref, E0, G0 = run(False)
    assert ref < 2
    # 1,600 complex steps of two coefficients and more: 3,686 records of 80 bytes
    assert path == (3 if mode == "complex" and steps == 1600 else 2)
    # 64-bit rounding of up to 1,600 rotations
    assert np.max(np.abs(E - E0)) < 1e-10 and np.max(np.abs(G - G0)) < 1e-10
