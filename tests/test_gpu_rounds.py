"""Rounds of the shared-memory sector path (forward program, sweep with its
gradient, residuals, packed problems) against the full-space evaluator: blocks
of one and many warps, records of several rounds and of several patterns, round
counts of every remainder modulo four, real and complex states, batches on both
sides of the two-sets-per-CTA line, packed launches larger than one group."""

import numpy as np
import pytest

import qforte_b200 as qb
from qforte_b200.ucc import DUCC, Pack, evaluator_config

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


def _on(mode, problem, P, separate):
    mol, pool, tops = problem
    evaluator_config(mode)
    try:
        eng = DUCC(mol.hamiltonian, pool, tops, mol.hf_reference, "sa_SD" if separate else None)
        out = eng.energy_grad(P)
        return out + ((eng.residuals(P)[1],) if not separate else ())
    finally:
        evaluator_config(True)


# separate: inner products and un-rotations are separate records
@pytest.mark.parametrize("norb,nel,pool_type,nops,B,mode,separate", [
    (2, 2, "SD", 0, 1, True, False),
    (3, 3, "SD", 0, 2, True, False),
    (4, 3, "SD", 0, 5, True, True),
    (5, 5, "GSD", 5, 3, True, True),
    (5, 4, "GSD", 6, 1, True, True),
    (5, 4, "GSD", 7, 2, "complex", True),
    (6, 6, "SD", 0, 3, "complex", False),
    (6, 7, "SD", 0, 4, "one-set", False),
    (4, 4, "SD", 0, 301, True, False),
    (8, 8, "SD", 0, 150, True, False),
])
def test_rounds_match_full_space(cuda, norb, nel, pool_type, nops, B, mode, separate):
    problem = _problem(norb, nel, pool_type, nops)
    P = np.random.default_rng(B).uniform(-0.3, 0.3, (B, len(problem[2])))
    got = _on(mode, problem, P, separate)
    rows = [0, B // 2, B - 1]
    want = _on(False, problem, P[rows], separate)
    # 64-bit rounding of a few hundred rotations and of sums of ~1e4 terms
    for g, w in zip(got, want):
        assert np.max(np.abs(np.asarray(g)[rows] - w)) < 1e-10


def test_packed_groups_match_single_evaluations(cuda):
    """More items than a group of launches takes, of problems of different
    block sizes, some without gradient."""
    duccs = []
    for norb, nel in ((2, 2), (4, 4), (6, 6)):
        mol, pool, tops = _problem(norb, nel, "SD", 0)
        duccs.append(DUCC(mol.hamiltonian, pool, tops, mol.hf_reference))
    n, rng = 1030, np.random.default_rng(3)
    members, grads = np.arange(n) % 3, (np.arange(n) % 4 != 2).astype(np.int32)
    params = [rng.uniform(-0.3, 0.3, duccs[m].nparam) for m in members]
    e, g = Pack(duccs, capacity=n).run(members, params, grads)
    for m, d in enumerate(duccs):
        at = np.flatnonzero(members == m)
        E, G = d.energy_grad(np.stack([params[i] for i in at]))
        assert np.max(np.abs(e[at] - E)) < 1e-10
        for k, i in enumerate(at):
            assert (g[i] is None) == (not grads[i])
            if grads[i]:
                assert np.max(np.abs(g[i] - G[k])) < 1e-10
