"""Programs of short Pauli strings whose angles are small, or near a multiple of 2 pi,
so that cos phi rounds to 1: what a string moves is sin phi in full, for every
kind of one- and two-qubit string, window by window (13 qubits), in gate tiles
(14) and in the fused tile form (20)."""

import ctypes
import itertools
import math

import numpy as np
import pytest

from qforte_b200._lib import check, lib, ptr
from qforte_b200.device import DeviceProg

pytestmark = pytest.mark.gpu

KINDS = ["".join(k) for k in itertools.product("XYZ", repeat=2)] + ["X", "Y", "Z"]


def _masks(kind, qubits):
    x = z = 0
    for p, q in zip(kind, qubits):
        x |= (p in "XY") << q
        z |= (p in "YZ") << q
    return x, z


def _parity(v):
    for s in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> np.uint64(s))
    return (v & np.uint64(1)).astype(bool)


def _exp(psi, x, z, phi):
    j = np.arange(psi.size, dtype=np.uint64)
    out = np.empty_like(psi)
    ph = 1j ** (bin(x & z).count("1") % 4)
    out[(j ^ np.uint64(x)).astype(np.int64)] = ph * np.where(_parity(j & np.uint64(z)), -1.0, 1.0) * psi
    return math.cos(phi) * psi + 1j * math.sin(phi) * out


def _run(n, x, z, scale, ref, sign):
    dp = DeviceProg(x, z, scale, np.zeros(len(x), np.int32), 1)
    one = np.ones(1)
    h = ctypes.c_void_p()
    check(lib().qfb_state_create(n, 1, ctypes.byref(h)))
    try:
        psi = np.zeros(1 << n, dtype=complex)
        psi[ref] = 1.0
        check(lib().qfb_state_upload(h, 0, ptr(psi), psi.size))
        check(lib().qfb_prog_apply(dp.h, h, ptr(one), 1, sign))
        out = np.empty(1 << n, dtype=complex)
        check(lib().qfb_state_download(h, 0, ptr(out), out.size))
    finally:
        lib().qfb_state_destroy(h)
    want = psi
    for k in range(len(x)) if sign > 0 else reversed(range(len(x))):
        want = _exp(want, x[k], z[k], sign * scale[k])
    return out, want


PHI = [1e-7, 5e-9, 1e-9, 1e-12, 2 * math.pi + 5e-9]


@pytest.mark.parametrize("n", [13, 14, 20])
@pytest.mark.parametrize("sign", [1, -1])
def test_one_string_moves_sin_phi(cuda, n, sign):
    for kind, phi in itertools.product(KINDS, PHI):
        # both places of the pair, neighbours and far apart, a set and a clear qubit
        for qubits in ((5, 6), (n - 1, 2)):
            x, z = _masks(kind, qubits)
            ref = 1 << 5 | 1 << 2
            out, want = _run(n, [x], [z], [phi], ref, sign)
            s = abs(math.sin(phi))
            if x:
                # a product of a cosine, a sine and signs
                assert abs(out[ref ^ x] - want[ref ^ x]) <= 4e-16 * s, (kind, phi, qubits)
                assert np.count_nonzero(out) <= 2
            else:
                # sin phi, or sin phi cos 2 phi - cos phi sin 2 phi
                assert abs(out[ref].imag - want[ref].imag) <= 2e-15 * s, (kind, phi, qubits)
            assert abs(out[ref] - want[ref]) < 4e-16


@pytest.mark.parametrize("n", [13, 14, 20])
@pytest.mark.parametrize("sign", [1, -1])
def test_many_strings_move_sin_phi(cuda, n, sign):
    rng = np.random.default_rng(n)
    x, z = [], []
    for k in range(36):
        kind = KINDS[k % len(KINDS)]
        xs, zs = _masks(kind, [int(q) for q in rng.choice(n, len(kind), replace=False)])
        x.append(xs)
        z.append(zs)
    ref = int(rng.integers(1 << n))
    for phi in PHI:
        out, want = _run(n, x, z, [phi] * len(x), ref, sign)
        s = abs(math.sin(phi))
        off = np.abs(out - want)
        # amplitudes elsewhere are sums of at most 36 products of order sin phi,
        # the reference's own a sum of 36 steps' changes to a number near 1
        assert off[ref] < 1e-14
        off[ref] = 0.0
        assert np.max(off) <= 1e-13 * s, phi
        assert np.max(np.abs(np.delete(out, ref))) > 0.9 * s
