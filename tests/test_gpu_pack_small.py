"""Packs of small problems only, which go out in one launch: against their own
evaluators, bit for bit the results of the same items in a pack with a larger
problem, one item and more items than the launch of complex states takes, and a
problem number that is no member's."""

import numpy as np
import pytest

import qforte_b200 as qb
from qforte_b200.ucc import DUCC, Pack, evaluator_config

pytestmark = pytest.mark.gpu


def _ducc(norb, nel):
    mol = qb.random_molecule(norb, nel, 11)
    pool = qb.SQOpPool()
    pool.set_orb_spaces(mol.hf_reference)
    pool.fill_pool("SD")
    return DUCC(mol.hamiltonian, pool, list(range(len(pool))), mol.hf_reference)


@pytest.mark.parametrize("mode", [True, "complex"])
@pytest.mark.parametrize("shapes", [((2, 2),), ((4, 4), (3, 3), (2, 2)), ((5, 4), (4, 4))])
def test_small_packs(cuda, shapes, mode):
    evaluator_config(mode)
    try:
        duccs = [_ducc(*s) for s in shapes]
        small, large = Pack(duccs, capacity=400), Pack(duccs + [_ducc(6, 6)], capacity=400)
        rng = np.random.default_rng(len(shapes))
        for n in (1, 7, 400):
            members = np.arange(n) % len(duccs)
            grads = (np.arange(n) % 3 != 1).astype(np.int32)
            params = [rng.uniform(-0.3, 0.3, duccs[m].nparam) for m in members]
            e, g = small.run(members, params, grads)
            e2, g2 = large.run(members, params, grads)
            assert np.array_equal(e, e2)
            for i in range(n):
                assert (g[i] is None) == (not grads[i])
                assert g[i] is None or np.array_equal(g[i], g2[i])
            for m, d in enumerate(duccs):
                at = np.flatnonzero(members == m)
                if not len(at):
                    continue
                E, G = d.energy_grad(np.stack([params[i] for i in at]))
                # 64-bit rounding of some fifty rotations
                assert np.max(np.abs(e[at] - E)) < 1e-11
                for k, i in enumerate(at):
                    assert g[i] is None or np.max(np.abs(g[i] - G[k])) < 1e-11
    finally:
        evaluator_config(True)


def test_no_such_member(cuda):
    import torch

    pack = Pack([_ducc(4, 4)], capacity=3)
    items, params, energy, _ = pack.tensors()
    items.copy_(torch.tensor([[0, 1], [1, 1], [0, 0]], dtype=torch.int32))
    params.zero_()
    pack.launch(3)
    torch.cuda.synchronize()
    e = energy.cpu().numpy()
    assert np.isfinite(e[0]) and np.isnan(e[1]) and e[2] == e[0]
