"""Windows of program steps on blocks of a sector (the global-memory sector
path) against the full-space evaluator: energies, gradients and residuals for
windows of one and several warps a slot, slot groups that the batch does not
fill, single steps between windows, separate inner products and un-rotations (the
ansatz program un-applied, as for spin-adapted pools), real and complex states."""

import numpy as np
import pytest

import qforte_b200 as qb
from qforte_b200.ucc import DUCC, evaluator_config

pytestmark = pytest.mark.gpu


def _problem(norb, nel, pool_type, nops):
    mol = qb.random_molecule(norb, nel, 11)
    pool = qb.SQOpPool()
    pool.set_orb_spaces(mol.hf_reference)
    pool.fill_pool(pool_type)
    tops = list(range(len(pool)))
    if nops:
        tops = [int(v) for v in np.random.default_rng(norb + nops).choice(len(pool), nops, False)]
    return mol, pool, tops


def _on(mode, mol, pool, tops, P, residuals):
    evaluator_config(mode)
    try:
        eng = DUCC(mol.hamiltonian, pool, tops, mol.hf_reference,
                   "sa_SD" if residuals is None else None)
        out = eng.energy_grad(P)
        path = eng.evaluator(len(P)).path
        return out + ((eng.residuals(P)[1],) if residuals else ()), path
    finally:
        evaluator_config(True)


# residuals None: un-rotation by the ansatz program
@pytest.mark.parametrize("norb,nel,pool_type,nops,B,mode,residuals", [
    (2, 2, "SD", 0, 1, "global", True),
    (4, 3, "SD", 0, 5, "global", False),
    (5, 5, "SD", 0, 3, "global", True),
    (5, 4, "GSD", 9, 2, "global", False),
    (6, 6, "SD", 0, 4, "global", None),
    (6, 7, "SD", 0, 33, "global", True),
    (6, 6, "SD", 0, 3, "global-complex", True),
    (8, 8, "SD", 0, 9, "global", True),
])
def test_windows_match_full_space(cuda, norb, nel, pool_type, nops, B, mode, residuals):
    mol, pool, tops = _problem(norb, nel, pool_type, nops)
    P = np.random.default_rng(B).uniform(-0.3, 0.3, (B, len(tops)))
    got, path = _on(mode, mol, pool, tops, P, residuals)
    want, _ = _on(False, mol, pool, tops, P, residuals)
    assert path == 3
    # 64-bit rounding of a few hundred rotations and of sums of ~1e4 terms
    assert np.max(np.abs(got[0] - want[0])) < 1e-10
    assert np.max(np.abs(got[1] - want[1])) < 1e-10
    if residuals:
        assert np.max(np.abs(got[2] - want[2])) < 1e-10


def test_windows_are_reproducible(cuda):
    """Partial sums are added in a fixed order: equal runs give equal bits."""
    mol, pool, tops = _problem(6, 6, "SD", 0)
    P = np.random.default_rng(2).uniform(-0.3, 0.3, (4, len(tops)))
    evaluator_config("global")
    try:
        eng = DUCC(mol.hamiltonian, pool, tops, mol.hf_reference)
        a, b = eng.energy_grad(P), eng.energy_grad(P)
    finally:
        evaluator_config(True)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
