"""Sums of Pauli strings on states of 8 qubits and more, by tiles of 256 outputs
(H psi, and <bra|H|ket> as one sum), against numpy: the smallest tile, groups of
every remainder modulo a block of four terms, real, imaginary and mixed
coefficients, fewer groups than warps and more blocks than a warp stages, several
states, states of fewer amplitudes than the expectation value's line."""

import ctypes

import numpy as np
import pytest

from qforte_b200._lib import check, lib, ptr
from qforte_b200.device import DeviceSum

pytestmark = pytest.mark.gpu


def _sum(n, ngroups, seed, kind):
    rng = np.random.default_rng(seed)
    x, z, c = [], [], []
    for g in range(ngroups):
        gx = 0 if g == 0 else int(rng.integers(1 << n))
        for _ in range(int(rng.integers(1, 14)) if g % 5 else 70):
            gz = int(rng.integers(1 << n))
            x.append(gx)
            z.append(gz)
            v = complex(rng.normal(), rng.normal())
            odd = bin(gx & gz).count("1") & 1
            if kind == "real":  # real matrix elements: c i^popcount(x & z) real
                v = 1j * v.real if odd else v.real
            elif kind == "imaginary":
                v = v.real if odd else 1j * v.real
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


@pytest.mark.parametrize("n,ngroups,B,kind", [
    (8, 1, 1, "real"), (8, 40, 3, "mixed"), (9, 7, 1, "imaginary"), (10, 90, 4, "real"),
    (10, 33, 2, "mixed"), (12, 60, 1, "real"), (12, 25, 1, "imaginary"), (13, 12, 2, "mixed"),
])
def test_tiles_match_numpy(cuda, n, ngroups, B, kind):
    c, x, z = _sum(n, ngroups, 10 * n + ngroups, kind)
    rng = np.random.default_rng(n)
    v = rng.normal(size=(2, B, 1 << n)) + 1j * rng.normal(size=(2, B, 1 << n))
    v /= np.linalg.norm(v, axis=2, keepdims=True)
    ds = DeviceSum(c, x, z)
    h = [ctypes.c_void_p() for _ in range(3)]
    try:
        for k in range(3):
            check(lib().qfb_state_create(n, B, ctypes.byref(h[k])))
        for k in range(2):
            for b in range(B):
                a = np.ascontiguousarray(v[k, b])
                check(lib().qfb_state_upload(h[k], b, ptr(a), a.size))
        check(lib().qfb_sum_apply(ds.h, h[2], h[0]))
        out, e = np.empty(1 << n, dtype=complex), np.empty(B, dtype=complex)
        check(lib().qfb_sum_expval(ds.h, h[1], h[0], ptr(e)))
        want = _apply(c, x, z, v[0])
        # at most ~1,000 terms of size ~1 on amplitudes of a unit vector
        for b in range(B):
            check(lib().qfb_state_download(h[2], b, ptr(out), out.size))
            assert np.max(np.abs(out - want[b])) < 1e-12
            assert abs(e[b] - np.vdot(v[1, b], want[b])) < 1e-12
    finally:
        for k in range(3):
            lib().qfb_state_destroy(h[k])
