"""Sums of Pauli strings in every form their kernels take, against numpy: batches of
states smaller than a tile of 256 outputs (a last tile in part, more states than a
grid dimension holds), groups cut between warps (one group, one that outweighs the
others), and the forms of few groups on large states, one state and batches that
are no multiple of the states a thread works."""

import ctypes

import numpy as np
import pytest

from qforte_b200._lib import check, lib, ptr
from qforte_b200.device import DeviceSum

pytestmark = pytest.mark.gpu


def _sum(n, groups, seed, kind):
    """groups: terms of each x-group (the first one diagonal)."""
    rng = np.random.default_rng(seed)
    x, z, c = [], [], []
    seen = set()
    for g, terms in enumerate(groups):
        gx = 0 if g == 0 else int(rng.integers(1 << n))
        while g and gx in seen and len(seen) < 1 << n:
            gx = int(rng.integers(1 << n))
        seen.add(gx)
        for _ in range(terms):
            gz = int(rng.integers(1 << n))
            odd = bin(gx & gz).count("1") & 1
            v = complex(rng.normal(), rng.normal())
            if kind == "real":
                v = 1j * v.real if odd else v.real
            x.append(gx)
            z.append(gz)
            c.append(v)
    return np.array(c, dtype=complex), np.array(x, np.uint64), np.array(z, np.uint64)


def _parity(v):
    for s in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> np.uint64(s))
    return (v & np.uint64(1)).astype(bool)


def _apply(c, x, z, psi):
    j = np.arange(psi.shape[-1], dtype=np.uint64)
    out = np.zeros_like(psi)
    for ck, xk, zk in zip(c, x, z):
        ph = ck * 1j ** (bin(int(xk & zk)).count("1") % 4)
        out[:, (j ^ xk).astype(np.int64)] += ph * np.where(_parity(j & zk), -1.0, 1.0) * psi
    return out


def _states(n, B, count):
    h = [ctypes.c_void_p() for _ in range(count)]
    for k in range(count):
        check(lib().qfb_state_create(n, B, ctypes.byref(h[k])))
    return h


@pytest.mark.parametrize("kind", ["real", "mixed"])
@pytest.mark.parametrize("n,B,groups", [
    (1, 1, [2, 3]), (1, 2100, [2, 3]), (2, 1, [3, 1, 5]), (3, 45, [9, 2, 2]), (3, 515, [5, 5]), (5, 1, [40]),
    (5, 1, [1] * 16), (6, 1, [3] * 17), (6, 7, [1, 8, 3] * 11), (6, 70, [7, 2, 9]),
    (7, 3, [5, 70, 2]), (8, 5, [200]), (9, 1, [1]), (10, 2, [300, 1, 1, 1]), (12, 1, [200]), (12, 3, [33, 2]),
    (16, 4, [1]), (16, 5, [120]), (16, 7, [20, 3, 4]), (18, 1, [1, 1]), (18, 1, [3, 90]), (18, 2, [250]),
])
def test_forms_match_numpy(cuda, n, B, groups, kind):
    c, x, z = _sum(n, groups, 100 * n + B, kind)
    rng = np.random.default_rng(n + B)
    v = rng.normal(size=(2, B, 1 << n)) + 1j * rng.normal(size=(2, B, 1 << n))
    v /= np.linalg.norm(v, axis=2, keepdims=True)
    ds = DeviceSum(c, x, z)
    h = _states(n, B, 3)
    try:
        for k in range(2):
            for b in range(B):
                a = np.ascontiguousarray(v[k, b])
                check(lib().qfb_state_upload(h[k], b, ptr(a), a.size))
        check(lib().qfb_sum_apply(ds.h, h[2], h[0]))
        out, e = np.empty(1 << n, dtype=complex), np.empty(B, dtype=complex)
        check(lib().qfb_sum_expval(ds.h, h[1], h[0], ptr(e)))
        want = _apply(c, x, z, v[0])
        # at most a few hundred terms of size ~1 on amplitudes of a unit vector
        for b in range(B):
            check(lib().qfb_state_download(h[2], b, ptr(out), out.size))
            assert np.max(np.abs(out - want[b])) < 1e-12
            assert abs(e[b] - np.vdot(v[1, b], want[b])) < 1e-12
    finally:
        for s in h:
            lib().qfb_state_destroy(s)


@pytest.mark.parametrize("n,B,groups", [(2, 70001, [2, 1, 3]), (2, 70001, [60, 50, 40, 50]), (6, 5001, [3] * 30)])
def test_large_batches_of_small_states(cuda, n, B, groups):
    """(two of them more states than a grid dimension holds)"""
    c, x, z = _sum(n, groups, 5, "mixed")
    ds = DeviceSum(c, x, z)
    h = _states(n, B, 2)
    rng = np.random.default_rng(0)
    try:
        v = rng.normal(size=(1, 1 << n)) + 1j * rng.normal(size=(1, 1 << n))
        slots = [0, 1, 2, 3, B // 2, B - 6, B - 5, B - 2, B - 1]
        for b in slots:
            a = np.ascontiguousarray(v[0] * (1 + b % 7))
            check(lib().qfb_state_upload(h[0], b, ptr(a), a.size))
        check(lib().qfb_sum_apply(ds.h, h[1], h[0]))
        out = np.empty(1 << n, dtype=complex)
        want = _apply(c, x, z, v)[0]
        for b in slots:
            check(lib().qfb_state_download(h[1], b, ptr(out), out.size))
            # at most 200 terms of size ~1 on amplitudes of size ~10
            assert np.max(np.abs(out - want * (1 + b % 7))) < 1e-11
    finally:
        for s in h:
            lib().qfb_state_destroy(s)
