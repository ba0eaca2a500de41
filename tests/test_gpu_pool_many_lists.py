"""ADAPT pool gradients of sectors with few electrons, whose alpha lists of one or two
strings meet thousands of short beta lists: the global-memory path against the
shared-memory one."""

import numpy as np
import pytest

import qforte_b200 as qb
from qforte_b200.ucc import DUCC, evaluator_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,nel,mode", [(8, 4, "global"), (9, 3, "global"), (11, 4, "global"),
                                           (8, 3, "global-complex")])
def test_short_lists_match_shared_memory(cuda, norb, nel, mode):
    mol = qb.random_molecule(norb, nel, 11)
    pool = qb.SQOpPool()
    pool.set_orb_spaces(mol.hf_reference)
    pool.fill_pool("GSD")
    tops = [int(v) for v in np.random.default_rng(norb).choice(len(pool), 6, False)]
    x = np.random.default_rng(nel).uniform(-0.3, 0.3, len(tops))
    got = []
    for m in (mode, True):
        evaluator_config(m)
        try:
            eng = DUCC(mol.hamiltonian, pool, tops, mol.hf_reference)
            got.append(np.asarray(eng.pool_gradients(x)))
            assert eng.evaluator(1).path == (3 if m == mode else 2)
        finally:
            evaluator_config(True)
    assert got[0].shape == got[1].shape and np.max(np.abs(got[1])) > 1e-3
    # sums of some thousand products of amplitudes of unit vectors
    assert np.max(np.abs(got[0] - got[1])) < 1e-11
