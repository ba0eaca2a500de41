"""The forward program with two parameter sets a CTA, at the batches that reach it
(odd and even, above what the SMs take at once), against one set a CTA: energies,
gradients, and the sweep alone on the states an energy-only run saved."""

import numpy as np
import pytest

import qforte_b200 as qb
from qforte_b200.ucc import DUCC, evaluator_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,seed,pool_type", [(4, 11, "SD"), (5, 9, "GSD"), (8, 2, "SD")])
@pytest.mark.parametrize("more", [-1, 1, 2])
def test_paired_forward_matches_one_set(cuda, norb, seed, pool_type, more):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    mol = qb.random_molecule(norb, norb, seed=seed)
    pool = qb.SQOpPool()
    pool.set_orb_spaces(mol.hf_reference)
    pool.fill_pool(pool_type)
    tops = list(range(0, len(pool), 1 if len(pool) < 400 else 3))
    # large blocks pair from one set an SM on, small ones from two
    B = (2 if more > 0 else 1) * sms + more
    P = np.random.default_rng(norb + B).uniform(-0.1, 0.1, (B, len(tops)))

    def evaluator(mode):
        evaluator_config(mode)
        try:
            return DUCC(mol.hamiltonian, pool, tops, mol.hf_reference, pool_type=pool_type).evaluator(B)
        finally:
            evaluator_config(True)

    ev, one = evaluator(True), evaluator("one-set")
    assert ev.path == 2 and ev.sets_per_cta == 2 and ev.forward_sets == (2 if more > 0 else 1)
    assert one.sets_per_cta == 1 and one.forward_sets == 1
    E, G = ev.eval(P, True)
    E1, G1 = one.eval(P, True)
    # 64-bit rounding of a few hundred rotations
    assert np.max(np.abs(E - E1)) < 1e-12 and np.max(np.abs(G - G1)) < 1e-11
    d_par, _, d_gr = ev.tensors()
    d_par.copy_(torch.from_numpy(P))
    ev.run(0)
    ev.run(2)
    torch.cuda.synchronize()
    assert np.max(np.abs(d_gr.cpu().numpy() - G1)) < 1e-11
