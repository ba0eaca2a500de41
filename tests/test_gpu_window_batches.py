"""Energies of more parameter sets than a window launch's grid holds (global-memory
sector path), against the same sets in a small batch."""

import numpy as np
import pytest

import qforte_b200 as qb
from qforte_b200.ucc import DUCC, evaluator_config

pytestmark = pytest.mark.gpu


def test_window_launches_of_many_sets(cuda):
    mol = qb.random_molecule(4, 4, seed=11)
    pool = qb.SQOpPool()
    pool.set_orb_spaces(mol.hf_reference)
    pool.fill_pool("SD")
    tops = list(range(len(pool)))
    B = 8 * 65535 + 9  # eight sets a block, one launch's grid and a few more
    rng = np.random.default_rng(0)
    few = rng.uniform(-0.3, 0.3, (16, len(tops)))
    P = np.ascontiguousarray(few[np.arange(B) % 16])
    evaluator_config("global")
    try:
        eng = DUCC(mol.hamiltonian, pool, tops, mol.hf_reference)
        ev, small = eng.evaluator(B), eng.evaluator(16)
    finally:
        evaluator_config(True)
    assert ev.path == 3 and small.path == 3
    E, _ = ev.eval(P, False)
    E0, _ = small.eval(few, True)
    # the same rotations in the same order
    assert np.max(np.abs(E - E0[np.arange(B) % 16])) < 1e-12
