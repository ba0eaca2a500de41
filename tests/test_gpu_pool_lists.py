"""ADAPT pool gradients of one state in the global-memory sector (rows shared by
the patterns of one alpha list) against the full-space evaluator: odd and
off-filling electron counts, one-electron strings (single-entry lists), real and
complex storage, and the batched form of the same evaluators."""

import numpy as np
import pytest

import qforte_b200 as qb
from qforte_b200.ucc import DUCC, evaluator_config

pytestmark = pytest.mark.gpu


def _gradients(mode, problem, P):
    mol, pool, tops = problem
    evaluator_config(mode)
    try:
        eng = DUCC(mol.hamiltonian, pool, tops, mol.hf_reference)
        g = eng.pool_gradients(P)
        ev = eng.evaluator(np.atleast_2d(P).shape[0])
        return g, ev.path, getattr(ev, "_pool_prog", None) is not None
    finally:
        evaluator_config(True)


@pytest.mark.parametrize("norb,nel,pool_type,mode", [
    (2, 2, "GSD", "global"), (3, 3, "GSD", "global"), (4, 2, "GSD", "global"), (4, 5, "GSD", "global"),
    (5, 5, "GSD", "global-complex"), (6, 6, "GSD", "global"), (6, 7, "SD", "global"),
])
def test_pool_lists_match_full_space(cuda, norb, nel, pool_type, mode):
    mol = qb.random_molecule(norb, nel, 11)
    pool = qb.SQOpPool()
    pool.set_orb_spaces(mol.hf_reference)
    pool.fill_pool(pool_type)
    rng = np.random.default_rng(norb + nel)
    tops = [int(v) for v in rng.choice(len(pool), min(6, len(pool)), False)]
    P = rng.uniform(-0.4, 0.4, (2, len(tops)))
    problem = (mol, pool, tops)
    got, path, native = _gradients(mode, problem, P[0])
    assert path == 3 and native
    want, _, _ = _gradients(False, problem, P[0])
    # 64-bit rounding of sums of at most a few thousand products
    assert np.max(np.abs(got - want)) < 1e-11
    both, _, _ = _gradients(mode, problem, P)
    assert np.max(np.abs(both[0] - got)) < 1e-11
