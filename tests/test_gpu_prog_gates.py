"""Programs of Pauli exponentials on at most two qubits as gate lists (states of 14
qubits and more) and programs that hold a longer string, against numpy: every
kind of one- and two-qubit string, forward and inverse, one and several states,
a state of the fused tile form."""

import ctypes

import numpy as np
import pytest

from qforte_b200._lib import check, lib, ptr
from qforte_b200.device import DeviceProg

pytestmark = pytest.mark.gpu


def _strings(n, count, seed, longest):
    rng = np.random.default_rng(seed)
    x, z = [], []
    for k in range(count):
        m = longest if k == count // 2 else k % 3
        xs = zs = 0
        for q in rng.choice(n, m, replace=False):
            p = int(rng.integers(1, 4))
            xs |= (p & 1) << int(q)
            zs |= (p >> 1) << int(q)
        x.append(xs)
        z.append(zs)
    return np.array(x, np.uint64), np.array(z, np.uint64), rng.uniform(-1.5, 1.5, count)


def _parity(v):
    for s in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> np.uint64(s))
    return (v & np.uint64(1)).astype(bool)


def _exp(psi, x, z, phi):
    j = np.arange(psi.size, dtype=np.uint64)
    out = np.empty_like(psi)
    ph = 1j ** (bin(int(x & z)).count("1") % 4)
    out[(j ^ x).astype(np.int64)] = ph * np.where(_parity(j & z), -1.0, 1.0) * psi
    return np.cos(phi) * psi + 1j * np.sin(phi) * out


@pytest.mark.parametrize("n,count,B,longest", [(14, 40, 1, 2), (14, 31, 3, 2), (15, 30, 1, 3),
                                               (13, 20, 1, 2), (20, 25, 1, 2)])
@pytest.mark.parametrize("sign", [1, -1])
def test_short_strings_match_numpy(cuda, n, count, B, longest, sign):
    x, z, scale = _strings(n, count, n + count, longest)
    theta = np.array([0.7, -0.4])
    param = np.arange(count, dtype=np.int32) % 2
    dp = DeviceProg(x, z, scale, param, 2)
    rng = np.random.default_rng(n)
    v = rng.normal(size=(B, 1 << n)) + 1j * rng.normal(size=(B, 1 << n))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    h = ctypes.c_void_p()
    check(lib().qfb_state_create(n, B, ctypes.byref(h)))
    try:
        for b in range(B):
            a = np.ascontiguousarray(v[b])
            check(lib().qfb_state_upload(h, b, ptr(a), a.size))
        check(lib().qfb_prog_apply(dp.h, h, ptr(theta), 1, sign))
        out = np.empty(1 << n, dtype=complex)
        for b in range(B):
            want = v[b]
            for k in range(count) if sign > 0 else reversed(range(count)):
                want = _exp(want, x[k], z[k], sign * scale[k] * theta[param[k]])
            check(lib().qfb_state_download(h, b, ptr(out), out.size))
            # some forty 64-bit rotations of amplitudes below 1
            assert np.max(np.abs(out - want)) < 1e-13
    finally:
        lib().qfb_state_destroy(h)
