"""The work that users of this framework have it do, as cases to be timed.

Every case goes through the public entry points (``DUCC``, ``ucc_energy``,
``Pack``, ``Computer``) with seeded synthetic inputs: random-integral
molecules, random layered circuits, the transverse-field Ising model.  The
compiled problem (Hamiltonian, pool and ansatz programs) is what a program
keeps over a whole optimisation, so it is built once per problem; the seed
draws what changes from call to call: the amplitudes, the circuit, the state.

``listed`` names the sizes to watch, ``draw`` gives others of the same ranges,
``prepare`` / ``run`` do one pass, ``exact`` computes the same outputs in
64 bits with plain torch, and ``work`` counts the bytes and operations the
path needs.
"""

import itertools
import math
from functools import lru_cache

import numpy as np
import torch

import qforte_b200 as qb
from qforte_b200.autograd import ucc_energy
from qforte_b200.systems import sq_hamiltonian
from qforte_b200.ucc import DUCC, Pack

INTEGRAL_SEED = 11

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # one optimiser call of a small molecule: launches and the host path count
        dict(name="vqe_12q_one", kind="vqe", norb=6, nel=6, batch=1, api="host"),
        # a parameter scan / batched optimiser, energy and adjoint gradient
        dict(name="vqe_16q_256", kind="vqe", norb=8, nel=8, batch=256, api="torch"),
        # an off-half-filling molecule of odd size, a few amplitude vectors at once
        dict(name="vqe_18q_8", kind="vqe", norb=9, nel=8, batch=8, api="torch"),
        # one optimiser call of a large molecule
        dict(name="vqe_20q_one", kind="vqe", norb=10, nel=10, batch=1, api="torch"),
        # a server's batch: requests of several problems in one packed launch
        dict(name="serving_mix", kind="pack", norb_min=5, norb_max=8, items=29),
        # ADAPT-VQE's operator selection: every generalised single and double
        dict(name="adapt_20q", kind="pool", norb=10, nel=10, nops=12),
        # projective (PQE) residual vectors, ragged batch, odd electron count
        dict(name="residuals_14q_37", kind="residuals", norb=7, nel=7, batch=37),
        # gate circuits from |0...0>: a small one, an ordinary one, a large one
        dict(name="circuit_12q", kind="circuit", nqubit=12, layers=8),
        dict(name="circuit_21q", kind="circuit", nqubit=21, layers=25),
        dict(name="circuit_27q", kind="circuit", nqubit=27, layers=40),
        # H psi and <psi|H|psi> of a molecular Hamiltonian on a full-space state
        # (Krylov and imaginary-time loops, per-call drivers)
        dict(name="operator_16q", kind="operator", norb=8),
        # Trotterised time evolution of a spin chain
        dict(name="evolve_23q", kind="evolve", nqubit=23, steps=6),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["vqe", "vqe", "vqe", "pack", "pool", "residuals", "circuit", "circuit",
                       "operator", "evolve"])
    if kind == "vqe":
        norb = rng.randint(4, 10)
        nel = norb + rng.randint(-2, 1)
        return dict(kind="vqe", norb=norb, nel=nel,
                    batch=_log_int(rng, 1, {9: 24, 10: 6}.get(norb, 256)),
                    api=rng.choice(["host", "torch"]))
    if kind == "pack":
        lo = rng.randint(4, 7)
        return dict(kind="pack", norb_min=lo, norb_max=rng.randint(lo, 8),
                    items=_log_int(rng, 1, 64))
    if kind == "pool":
        norb = rng.randint(5, 10)
        return dict(kind="pool", norb=norb, nel=norb + rng.randint(-1, 1), nops=rng.randint(3, 20))
    if kind == "residuals":
        norb = rng.randint(4, 9)
        return dict(kind="residuals", norb=norb, nel=norb + rng.randint(-1, 1),
                    batch=_log_int(rng, 1, 12 if norb > 8 else 128))
    if kind == "circuit":
        n = rng.randint(5, 26)
        return dict(kind="circuit", nqubit=n, layers=_log_int(rng, 1, 40))
    if kind == "operator":
        return dict(kind="operator", norb=rng.randint(3, 8))
    return dict(kind="evolve", nqubit=rng.randint(6, 25), steps=_log_int(rng, 1, 10))


# ---------------------------------------------------------------------------
# what a program keeps over many calls: molecules and compiled problems
# ---------------------------------------------------------------------------


def _integrals(norb, seed=INTEGRAL_SEED):
    """Real symmetric one-electron integrals and (pq|rs) = sum_l L^l_pq L^l_rs."""
    rng = np.random.default_rng(seed)
    h = rng.normal(0.0, 0.1, size=(norb, norb))
    h = np.triu(h, 1) + np.triu(h, 1).T
    h[np.diag_indices(norb)] = rng.uniform(-2.0, -0.5, size=norb)
    g = np.zeros((norb,) * 4)
    for _ in range(6):
        f = rng.normal(0.0, 0.1, size=(norb, norb))
        f = np.triu(f) + np.triu(f, 1).T
        g += np.einsum("pq,rs->pqrs", f, f)
    return h, g


@lru_cache(maxsize=16)
def _hamiltonian(norb):
    return sq_hamiltonian(*_integrals(norb)).jw_transform()


def _pool_object(norb, nel, kind):
    pool = qb.SQOpPool()
    pool.set_orb_spaces([1] * nel + [0] * (2 * norb - nel))
    pool.fill_pool(kind)
    return pool


@lru_cache(maxsize=8)
def _problem(norb, nel):
    """The compiled dUCCSD problem."""
    pool = _pool_object(norb, nel, "SD")
    return DUCC(_hamiltonian(norb), pool, range(len(pool)), [1] * nel + [0] * (2 * norb - nel))


def _adapt_tops(norb, nops, npool):
    return [int(v) for v in np.random.default_rng(1000 * norb + nops).choice(npool, nops, False)]


@lru_cache(maxsize=4)
def _adapt_problem(norb, nel, nops):
    """An ADAPT-VQE ansatz of nops operators of the generalised pool."""
    pool = _pool_object(norb, nel, "GSD")
    return DUCC(_hamiltonian(norb), pool, _adapt_tops(norb, nops, len(pool)),
                [1] * nel + [0] * (2 * norb - nel))


@lru_cache(maxsize=4)
def _pack(norb_min, norb_max, items):
    duccs = [_problem(n, n) for n in range(norb_min, norb_max + 1)]
    return Pack(duccs, capacity=items), [d.nparam for d in duccs]


@lru_cache(maxsize=2)
def _tfim(n):
    return qb.system_factory("model", "TFIM", n=n, h=0.7, J=1.0).hamiltonian


# ---------------------------------------------------------------------------
# inputs from the seed
# ---------------------------------------------------------------------------


def _amplitudes(seed, *shape):
    return np.random.default_rng(seed).uniform(-0.1, 0.1, shape)


def _pack_items(case, seed, nparams):
    """Members, gradient flags (two of three) and parameters of the requests of a batch."""
    rng, items = np.random.default_rng(seed), np.arange(case["items"])
    members = items * 7 % len(nparams)
    grads = (items % 3 != 1).astype(np.int32)
    return members, grads, [rng.uniform(-0.1, 0.1, nparams[m]) for m in members]


ONE_QUBIT = ("H", "X", "Y", "Z", "S", "T", "Rx", "Ry", "Rz")
TWO_QUBIT = ("cX", "cZ", "SWAP", "cR")


def _circuit_spec(case, seed):
    """Layers of one random gate per qubit, then random two-qubit gates on a
    random perfect matching (one qubit idles when their number is odd)."""
    n, rng, spec = case["nqubit"], np.random.default_rng(seed), []
    for _ in range(case["layers"]):
        for q in range(n):
            spec.append((ONE_QUBIT[rng.integers(9)], q, q, float(rng.uniform(0, 2 * math.pi))))
        perm = rng.permutation(n)
        for i in range(0, n - 1, 2):
            spec.append((TWO_QUBIT[rng.integers(4)], int(perm[i]), int(perm[i + 1]),
                         float(rng.uniform(0, 2 * math.pi))))
    return spec


def _random_state(n, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    v = torch.randn(1 << n, 2, dtype=torch.float64, device="cuda", generator=gen)
    return torch.view_as_complex(v / v.norm())


def _evolution_time(seed):
    return float(np.random.default_rng(seed).uniform(0.2, 1.0))


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------


def prepare(case, seed):
    k = case["kind"]
    s = {"kind": k}
    if k == "vqe":
        s["ducc"] = _problem(case["norb"], case["nel"])
        P = _amplitudes(seed, case["batch"], s["ducc"].nparam)
        if case["api"] == "torch":
            s["P"] = torch.from_numpy(P).cuda().requires_grad_()
        else:
            s["P"] = P[0] if case["batch"] == 1 else P
    elif k == "residuals":
        s["ducc"] = _problem(case["norb"], case["nel"])
        s["P"] = _amplitudes(seed, case["batch"], s["ducc"].nparam)
    elif k == "pool":
        s["ducc"] = _adapt_problem(case["norb"], case["nel"], case["nops"])
        s["P"] = _amplitudes(seed, case["nops"])
    elif k == "pack":
        s["pack"], nparams = _pack(case["norb_min"], case["norb_max"], case["items"])
        s["items"] = _pack_items(case, seed, nparams)
    elif k == "circuit":
        s["circ"] = qb.Circuit()
        for kind, t, c, p in _circuit_spec(case, seed):
            s["circ"].add(qb.gate(kind, t, c, p))
        s["qc"] = qb.Computer(case["nqubit"])
    elif k == "operator":
        s["H"] = _hamiltonian(case["norb"])
        s["qc"] = qb.Computer(2 * case["norb"])
        s["qc"].tensor().copy_(_random_state(2 * case["norb"], seed))
    elif k == "evolve":
        s["circ"], _ = qb.trotterize(_tfim(case["nqubit"]), factor=-1j * _evolution_time(seed),
                                     trotter_number=case["steps"])
        s["qc"] = qb.Computer(case["nqubit"])
    return s


def _amplitudes_of(qc):
    """The state as a tensor that keeps its Computer alive."""
    t = qc.tensor()
    t.computer = qc
    return t


def run(s):
    k = s["kind"]
    if k == "vqe":
        if isinstance(s["P"], np.ndarray):
            return s["ducc"].energy_grad(s["P"])
        s["P"].grad = None
        E = ucc_energy(s["P"], s["ducc"])
        E.sum().backward()
        return E.detach(), s["P"].grad
    if k == "residuals":
        return s["ducc"].residuals(s["P"])
    if k == "pool":
        return s["ducc"].pool_gradients(s["P"])
    if k == "pack":
        members, grads, params = s["items"]
        e, g = s["pack"].run(members, params, grads)
        return e, np.concatenate([x for x in g if x is not None])
    if k == "operator":
        sigma = qb.Computer(s["qc"])
        sigma.apply_operator(s["H"])
        e = s["qc"].direct_op_exp_val(s["H"])
        return _amplitudes_of(sigma), e.real
    s["qc"].reset()
    s["qc"].apply_circuit(s["circ"])
    return _amplitudes_of(s["qc"])


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, in plain torch
# ---------------------------------------------------------------------------


def _parity(v):
    for o in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> o)
    return v & 1


class _Fermions:
    """Products of creation and annihilation operators (Jordan-Wigner order:
    spin orbital 2p + spin) on the determinants of one particle-number sector,
    or on all of them."""

    def __init__(self, norb, nel=None):
        self.norb, n = norb, 2 * norb
        d = torch.arange(1 << n, dtype=torch.int64, device="cuda")
        if nel is not None:
            cnt = lambda m: sum((d >> (2 * p + m)) & 1 for p in range(norb))  # noqa: E731
            d = d[(cnt(0) == (nel + 1) // 2) & (cnt(1) == nel // 2)]
        self.det = d
        self.at = torch.zeros(1 << n, dtype=torch.int64, device="cuda")
        self.at[d] = torch.arange(d.numel(), device="cuda")
        self.h, self.g = (torch.from_numpy(x).cuda() for x in _integrals(norb))

    def move(self, cre, ann):
        """(from, to, sign) of a+_cre[0] a+_cre[1] .. a_ann[0] a_ann[1] ..."""
        d, src = self.det, torch.arange(self.det.numel(), device="cuda")
        odd = torch.zeros_like(d)
        for q, want in [(q, 1) for q in reversed(ann)] + [(q, 0) for q in reversed(cre)]:
            keep = ((d >> q) & 1) == want
            d, src, odd = d[keep], src[keep], odd[keep]
            odd = odd ^ _parity(d & ((1 << q) - 1))
            d = d ^ (1 << q)
        return src, self.at[d], (1 - 2 * odd).to(torch.float64)

    def hpsi(self, psi):
        """H psi for psi [..., determinants]: E_pq E_rs contracted with the integrals."""
        m = self.norb
        E = [[[self.move([2 * p + s], [2 * q + s]) for s in (0, 1)] for q in range(m)]
             for p in range(m)]
        out = torch.zeros_like(psi)
        hh = self.h - 0.5 * torch.einsum("prqr->pq", self.g)
        for b in range(psi.shape[0]):
            D = torch.zeros((m, m) + psi.shape[1:], dtype=psi.dtype, device="cuda")
            for r, s in itertools.product(range(m), repeat=2):
                for src, dst, sg in E[r][s]:
                    D[r, s][dst] += sg * psi[b][src]
            G = (0.5 * self.g.reshape(m * m, m * m)).to(psi.dtype) @ D.reshape(m * m, -1)
            G = G.reshape(D.shape)
            for p, q in itertools.product(range(m), repeat=2):
                t = G[p, q] + hh[p, q] * psi[b]
                for src, dst, sg in E[p][q]:
                    out[b][dst] += sg * t[src]
        return out

    def start(self, nel, batch):
        psi = torch.zeros(batch, self.det.numel(), dtype=torch.float64, device="cuda")
        psi[:, self.at[(1 << nel) - 1]] = 1.0
        return psi

    @staticmethod
    def rotate(psi, mv, t):
        """exp(t (T - T+)) in place; t is [batch]."""
        i, j, sg = mv
        c, s = torch.cos(t)[:, None], torch.sin(t)[:, None] * sg
        a, b = psi[:, i], psi[:, j]
        psi[:, i] = c * a - s * b
        psi[:, j] = c * b + s * a

    @staticmethod
    def inner(sig, psi, mv):
        """<sig|T - T+|psi> per row."""
        i, j, sg = mv
        return ((sig[:, j] * psi[:, i] - sig[:, i] * psi[:, j]) * sg).sum(1)


def _sd_excitations(norb, nel):
    """Spin-conserving singles and doubles of the reference, by the basis index
    of the determinant they reach: (creators, annihilators), highest first."""
    n, out = 2 * norb, []
    occ, vir = list(range(nel)), list(range(nel, n))
    for rank in (1, 2):
        for o in itertools.combinations(occ, rank):
            for v in itertools.combinations(vir, rank):
                if sum(x % 2 for x in o) == sum(x % 2 for x in v):
                    det = (1 << nel) - 1
                    for x in o + v:
                        det ^= 1 << x
                    out.append((det, v[::-1], o[::-1]))
    return [(list(v), list(o)) for _, v, o in sorted(out)]


def _gsd_excitations(norb):
    """Generalised singles and doubles in the pool's order."""
    out, seen = [], set()
    for i in range(norb):
        for a in range(i + 1, norb):
            out += [([2 * a], [2 * i]), ([2 * a + 1], [2 * i + 1])]
    for i in range(norb):
        for j in range(i, norb):
            for a in range(norb):
                for b in range(a, norb):
                    for sa, sb, si, sj in ((0, 0, 0, 0), (1, 1, 1, 1), (0, 1, 0, 1), (1, 0, 1, 0),
                                           (0, 1, 1, 0), (1, 0, 0, 1)):
                        c, d = [2 * a + sa, 2 * b + sb], [2 * i + si, 2 * j + sj]
                        if c[0] == c[1] or d[0] == d[1] or set(c) == set(d):
                            continue
                        key = frozenset((frozenset(c), frozenset(d)))
                        if key not in seen:
                            seen.add(key)
                            out.append((c, d))
    return out


def _exact_vqe(norb, nel, P, grad=True, residuals=False):
    F, exc = _Fermions(norb, nel), _sd_excitations(norb, nel)
    T = torch.from_numpy(np.atleast_2d(P)).cuda()
    mv = [F.move(c, o) for c, o in exc]
    psi = F.start(nel, T.shape[0])
    ref = psi[0].argmax()
    for k, m in enumerate(mv):
        F.rotate(psi, m, T[:, k])
    sig = F.hpsi(psi)
    E = (psi * sig).sum(1)
    if residuals:
        for k in reversed(range(len(mv))):
            F.rotate(sig, mv[k], -T[:, k])
        R = torch.empty_like(T)
        for k, (i, j, sg) in enumerate(mv):  # the determinant T_k|ref> and its sign
            at = (i == ref).nonzero()[0, 0]
            R[:, k] = sig[:, j[at]] * sg[at]
        return E, R
    G = torch.empty_like(T)
    for k in reversed(range(len(mv))) if grad else ():
        G[:, k] = 2.0 * F.inner(sig, psi, mv[k])
        F.rotate(psi, mv[k], -T[:, k])
        F.rotate(sig, mv[k], -T[:, k])
    return E, G


def _exact_pool(case, P):
    exc = _gsd_excitations(case["norb"])
    F = _Fermions(case["norb"], case["nel"])
    psi = F.start(case["nel"], 1)
    for top, t in zip(_adapt_tops(case["norb"], case["nops"], len(exc)), P):
        F.rotate(psi, F.move(*exc[top]), torch.tensor([t], dtype=torch.float64, device="cuda"))
    sig = F.hpsi(psi)
    return torch.cat([2.0 * F.inner(sig, psi, F.move(c, o)) for c, o in exc])


def _matrix(kind, p):
    """The 2 x 2 matrix of a one-qubit gate, or of a controlled gate's block."""
    r, c, s = math.sqrt(0.5), math.cos(p / 2), math.sin(p / 2)
    e = lambda x: complex(math.cos(x), math.sin(x))  # noqa: E731
    return {"H": (r, r, r, -r), "X": (0, 1, 1, 0), "Y": (0, -1j, 1j, 0), "Z": (1, 0, 0, -1),
            "S": (1, 0, 0, 1j), "T": (1, 0, 0, e(math.pi / 4)), "Rx": (c, -1j * s, -1j * s, c),
            "Ry": (c, -s, s, c), "Rz": (e(-p / 2), 0, 0, e(p / 2)), "cX": (0, 1, 1, 0),
            "cZ": (1, 0, 0, -1), "cR": (1, 0, 0, e(p))}[kind]


def _exact_circuit(case, seed):
    n = case["nqubit"]
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1.0
    for kind, t, c, p in _circuit_spec(case, seed):
        hi, lo = max(t, c), min(t, c)
        if t == c:
            v = psi.view(-1, 2, 1 << t)
            a, b = v[:, 0], v[:, 1]
        else:
            v = psi.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
            pick = lambda ct, tt: v[:, ct, :, tt] if c == hi else v[:, tt, :, ct]  # noqa: E731
            a, b = pick(1, 0), pick(1, 1)
        if kind == "SWAP":
            a, b = pick(0, 1), pick(1, 0)
        m00, m01, m10, m11 = _matrix("X" if kind == "SWAP" else kind, p)
        if m01 == 0:
            if m00 != 1:
                a.mul_(m00)
            if m11 != 1:
                b.mul_(m11)
        else:
            a0 = a.clone()
            a.mul_(m00).add_(b, alpha=m01)
            b.mul_(m11).add_(a0, alpha=m10)
    return psi


def _exact_evolve(case, seed):
    n, r = case["nqubit"], case["steps"]
    dt = _evolution_time(seed) / r
    i = torch.arange(1 << n, dtype=torch.int64, device="cuda")
    zsum = sum(1 - 2 * ((i >> q) & 1) for q in range(n)).to(torch.float64)
    zrot = torch.polar(torch.ones_like(zsum), 0.7 * dt * zsum)  # exp(i dt h sum Z)
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1.0
    c, s = math.cos(dt), math.sin(dt)
    for _ in range(r):
        psi = psi * zrot
        for q in range(n - 1):
            v = psi.view(-1, 2, 2, 1 << q)
            psi = (c * v + 1j * s * v.flip(1, 2)).view(-1)  # exp(i dt J X X)
    return psi


def exact(case, seed):
    k = case["kind"]
    if k in ("vqe", "residuals"):
        d = len(_sd_excitations(case["norb"], case["nel"]))
        one = k == "vqe" and case["api"] == "host" and case["batch"] == 1
        E, G = _exact_vqe(case["norb"], case["nel"], _amplitudes(seed, case["batch"], d),
                          residuals=k == "residuals")
        return (float(E[0]), G[0]) if one else (E, G)
    if k == "pool":
        return _exact_pool(case, _amplitudes(seed, case["nops"]))
    if k == "pack":
        norbs = range(case["norb_min"], case["norb_max"] + 1)
        items = _pack_items(case, seed, [len(_sd_excitations(n, n)) for n in norbs])
        members, grads, params = items
        E, G = torch.empty(len(members), dtype=torch.float64), [None] * len(members)
        for m, norb in enumerate(norbs):
            at = [i for i in range(len(members)) if members[i] == m]
            if at:
                e, g = _exact_vqe(norb, norb, np.stack([params[i] for i in at]))
                for j, i in enumerate(at):
                    E[i], G[i] = e[j], g[j]
        return E, torch.cat([g for g, w in zip(G, grads) if w])
    if k == "operator":
        psi = _random_state(2 * case["norb"], seed)
        sig = _Fermions(case["norb"]).hpsi(psi[None])[0]
        return sig, float(torch.vdot(psi, sig).real)
    if k == "circuit":
        return _exact_circuit(case, seed)
    return _exact_evolve(case, seed)


# ---------------------------------------------------------------------------
# bytes and operations of one pass
# ---------------------------------------------------------------------------


def _sector(norb, nel):
    """(amplitudes, entries of a molecular H, amplitude pairs of all SD excitations, parameters)."""
    na, nb = (nel + 1) // 2, nel // 2
    C = math.comb
    size = C(norb, na) * C(norb, nb)
    va, vb = norb - na, norb - nb
    row = 1 + na * va + nb * vb + C(na, 2) * C(va, 2) + C(nb, 2) * C(vb, 2) + na * va * nb * vb
    exc = _sd_excitations(norb, nel)
    pairs = 0
    for cre, _ in exc:
        kb = sum(x % 2 for x in cre)
        ka = len(cre) - kb
        pairs += C(norb - 2 * ka, na - ka) * C(norb - 2 * kb, nb - kb)
    return size, size * row, pairs, len(exc)


def _vqe_work(norb, nel, grad):
    """Rotations: 6 operations a pair and state; H: 2 an entry; inner products: 4 a pair."""
    size, nnz, pairs, npar = _sector(norb, nel)
    return 8 + npar * (16 if grad else 8), 2 * nnz + 2 * size + pairs * (6 + (16 if grad else 0))


def work(case):
    k = case["kind"]
    if k in ("vqe", "residuals"):
        b, f = _vqe_work(case["norb"], case["nel"], k == "vqe")
        if k == "residuals":
            _, _, pairs, npar = _sector(case["norb"], case["nel"])
            b, f = b + 8 * npar, f + 6 * pairs
        return {"bytes": b * case["batch"], "flops": f * case["batch"]}
    if k == "pool":
        size, nnz, _, _ = _sector(case["norb"], case["nel"])
        m = case["norb"]
        npool = len(_gsd_excitations(m))
        return {"bytes": 8 * (case["nops"] + npool),
                "flops": 2 * nnz + npool * size // 4}  # an operator connects about 1/8 of the pairs
    if k == "pack":
        w = [_vqe_work(n, n, True) for n in range(case["norb_min"], case["norb_max"] + 1)]
        return {"bytes": case["items"] * sum(x for x, _ in w) / len(w),
                "flops": case["items"] * sum(x for _, x in w) / len(w)}
    if k == "operator":
        N = 4 ** case["norb"]
        nnz = sum(math.comb(case["norb"], a) * math.comb(case["norb"], b) *
                  (_row(case["norb"], a, b)) for a in range(case["norb"] + 1)
                  for b in range(case["norb"] + 1))
        return {"bytes": 32 * N, "flops": 4 * nnz + 8 * N}
    N = 1 << case["nqubit"]
    if k == "circuit":
        # a mixing gate: two complex multiplications an amplitude; a phase: one on half of them
        per_layer = case["nqubit"] * (3 * 14 + 4 * 3) / 9 + (case["nqubit"] // 2) * (2 * 3 / 4)
        return {"bytes": 16 * N, "flops": N * case["layers"] * per_layer / 2}
    return {"bytes": 16 * N, "flops": N * case["steps"] * (6 + 6 * (case["nqubit"] - 1))}


def _row(norb, na, nb):
    C = math.comb
    va, vb = norb - na, norb - nb
    return 1 + na * va + nb * vb + C(na, 2) * C(va, 2) + C(nb, 2) * C(vb, 2) + na * va * nb * vb
