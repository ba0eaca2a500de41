"""Runs of steps whose lists outgrow a window are cut into shorter windows, not into
single steps: hops of one spin on 1,716 strings, against the shared-memory path and
by the kernels launched."""

import ctypes
import types

import numpy as np
import pytest

from qforte_b200._lib import check, lib
from qforte_b200.device import DeviceProg, DeviceSum
from qforte_b200.ucc import Evaluator, evaluator_config

pytestmark = pytest.mark.gpu

NORB, NQ, STEPS = 13, 26, 60


def _hops(count, seed):
    """(XY - YX) / 2 between beta orbitals p and q, no sign strings."""
    rng = np.random.default_rng(seed)
    x, z, c, par = [], [], [], []
    for k in range(count):
        p, q = (2 * int(v) + 1 for v in rng.choice(NORB, 2, replace=False))
        x += [1 << p | 1 << q] * 2
        z += [1 << p, 1 << q]
        c += [0.5, -0.5]
        par += [k, k]
    return x, z, c, par


def _launches():
    n = ctypes.c_uint64()
    check(lib().qfb_launch_count(ctypes.byref(n)))
    return n.value


@pytest.mark.parametrize("mode", ["global", "global-complex"])
def test_long_lists_are_cut_into_windows(cuda, mode):
    x, z, c, par = _hops(STEPS, 3)
    dp = DeviceProg(x, z, c, par, STEPS)
    # H: occupations, their products, and symmetric hops (XX + YY) / 2
    rng = np.random.default_rng(4)
    hx, hz, hc = [], [], []
    for q in range(1, NQ, 2):
        hx += [0, 0]
        hz += [1 << q, 1 << q | 1 << ((q + 2) % NQ)]
        hc += list(rng.normal(size=2))
    for k in range(30):
        m = x[2 * k]
        f = 0.5 * rng.normal()
        hx += [m, m]
        hz += [0, m]
        hc += [f, f]
    H = DeviceSum(np.array(hc, complex), hx, hz)
    ref = sum(1 << (2 * q + 1) for q in range(6))
    problem = types.SimpleNamespace(fwd=dp, grad_prog=dp, unrot_prog=dp, H=H, nqubit=NQ, ref_index=ref,
                                    nparam=STEPS)
    P = np.random.default_rng(5).uniform(-0.6, 0.6, (2, STEPS))

    def run(m):
        evaluator_config(m)
        try:
            ev = Evaluator(problem, 2, capture=False)
        finally:
            evaluator_config(True)
        n0 = _launches()
        out = ev.eval(P, True)
        return out, ev.path, _launches() - n0

    (E, G), path, launches = run(mode)
    (E0, G0), path0, _ = run(True)
    assert (path, path0) == (3, 2)
    # 64-bit rounding of 60 rotations
    assert np.max(np.abs(E - E0)) < 1e-11 and np.max(np.abs(G - G0)) < 1e-11
    assert np.max(np.abs(G0)) > 1e-3
    # a step's list takes at most 462 words of a window's 6,144: twelve steps and
    # more a window, forward and sweep, and a few launches for the rest
    assert launches < STEPS
