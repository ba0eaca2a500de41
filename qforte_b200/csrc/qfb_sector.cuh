// Compact particle-number sector evaluator.
//
// When every step of a dUCC evaluator's programs keeps the reference's
// numbers of alpha (even) and beta (odd) electrons, psi = U(t)|ref> and
// sigma = H psi live in the sector of those numbers.  That sector is stored
// compactly: index i = ra * nbeta + rb for the alpha string of rank ra and
// the beta string of rank rb (ranks in ascending order of the strings' bits).
// A 16-qubit, 8-electron sector is 4,900 amplitudes, so one CTA holds psi and
// sigma of one parameter set in shared memory and runs the whole evaluation
// there: the forward program, sigma = H psi from a sparse row list of H built
// once per evaluator, the energy, and the adjoint reverse sweep, with one
// barrier per program step and no global traffic besides the H rows, the
// steps' pair lists (read-only, L2-resident, shared by every CTA) and one save
// of psi and sigma between the kernels.
//
// When every step's pair coefficients and H are real (particle-hole and
// generalised pools of real excitations, real integrals), psi and sigma stay
// real and are stored as doubles (V = double): half the shared memory and
// half the shared-memory traffic of complex storage (V = double2).
//
// Each step is one of the Givens-form steps of the full-space program: the
// pairs (j0, j1 = j0 ^ x) with j0's bits on the step's pattern positions equal
// to one of its active patterns (bit h of x clear).  Restricted to the sector,
// such a j0 factors into an alpha string and a beta string matching the
// pattern's alpha and beta bits, so the pairs of one pattern are the product
// of an alpha list and a beta list, each entry holding a string's rank, its
// partner's rank (string ^ x) and its share of the sign
// sigma(j0) = (-1)^popcount(j0 & zbase).  The global-memory path
// (qfb_csec.cuh) reads those lists (records of RHead / RPat / SEntry); the
// shared-memory kernels here read the product expanded on the host into one
// word per amplitude pair, laid out in rounds of a block's threads (RStream)
// and ordered so that each half warp (quarter warp for 16-byte words) touches
// distinct banks.  The pool kernel reads pair lists (PHead / PStream).
//
// Forward and sweep are bound by one round after another, so the rounds are
// what was made short.  us, before (a record at a time, tests and look-ups
// between its barriers) / now: one set, 12 qubits (117 steps) forward 35 / 9.5,
// sweep 54 / 15; 16 qubits (360 steps) 128 / 56 and 227 / 116; 256 sets of 16
// qubits 157 / 95 and 320 / 215.
#pragma once

#include <cstdint>

namespace qfbs {

struct SEntry {  // one string of an alpha or beta list
    uint16_t r0, r1;  // rank, partner's rank
    uint32_t s;       // parity of string & zbase
};

// A step record: the 16-byte header, the patterns, then the entries of their
// lists, contiguous in one stream of 16-byte words.  Records run in the order
// a kernel executes them.
struct RHead {
    int32_t npf;   // patterns | flags << 8
    int32_t row;   // partial row of an inner product
    double gamma;
};
struct RPat {
    uint16_t a0, na, b0, nb;  // lists: entries [a0, a0 + na) and [b0, b0 + nb) of the record
    uint32_t inv;             // ceil(2^32 / nb), 0 when nb == 1
    uint32_t pad;
    double2 gn, hn;
};
enum : int { R_ROT = 1, R_IP = 2, R_TWO = 4 };

struct SStream {          // one kernel's records
    const uint4 *rec;     // records, 16-byte words
    const int2 *span;     // per record: first word, words
    const int32_t *param; // per record: parameter of its angle
    int n;
    int maxw;             // longest record (words)
};

// A step record on the pair list, used by the pool kernel: the pairs of the
// step's patterns as explicit sector index pairs, ordered on the host so that
// the lanes of a warp reach distinct shared-memory banks, and the step's
// constants.  A stream's headers, pairs and pattern coefficients are three
// arrays.
struct PHead {
    int32_t p0;     // first pair
    int32_t np;     // pairs
    int32_t fl;     // flags (R_ROT | R_IP | R_TWO) | patterns << 8
    int32_t row;    // partial row of an inner product
    double gamma;
    int32_t c0;     // first pattern's (gn, hn) in coef
    int32_t param;  // parameter of the record's angle
};
static_assert(sizeof(PHead) == 32, "PHead is two 16-byte words");

// A pair word: i0 (bits 0-13) | i1 << 14 | neg << 28 | pattern << 29 (a
// Givens-form step has at most 8 active patterns).
constexpr int kPairIdxBits = 14;  // sector indices below 16384
constexpr int kStepThreads = 512;  // block of the step kernels, at most
constexpr int kPairPatterns = 8;
struct PStream {
    const PHead *hd;
    const uint32_t *pair;
    const double2 *coef;  // per pattern: gn, hn
    int n;
};

// A stream as the step kernels run it: rounds of nth pairs, one pair a thread,
// a barrier after each.  A record takes as many rounds as its pairs need; the
// lanes left over rotate amplitudes past the sector's end (kRoundPad of them,
// zero), so no thread tests anything.  A word holds both indices as byte
// offsets of 8-byte amplitudes: last round of its record (bit 0), first round
// (bit 1), i0 (bits 3-16), i1 (bits 17-30), neg (bit 31).  The number of rounds
// is a multiple of 4 (the last ones are an empty record's), with 4 unused
// rounds of words on either side.
struct RRec {
    double gamma;
    int32_t param;
    int32_t fl;  // R_ROT | R_IP
    double2 gn, hn;
};
static_assert(sizeof(RRec) == 48, "RRec layout");
constexpr int kRoundPad = 32;
constexpr uint32_t kWordIdx = ((1u << kPairIdxBits) - 1u) << 3;
struct RStream {
    const RRec *hd;
    const uint32_t *word;
    int n, nr, nth, pad;
};

struct SLaunch {
    int nsec, nbeta, ref_i, nparam;
    RStream fwd, sweep;
    const int32_t *rowptr;     // H rows
    const uint32_t *col;
    const double *val_r;       // real H (val_c == nullptr) ...
    const double2 *val_c;      // ... or complex
    const double *params;      // [B][nparam]
    double *energy;            // [B]
    double *grad;              // [B][nparam]
    const int2 *prange;        // rounds of the sweep of each parameter's inner products
    double *partial;           // [B][sweep rounds / 4][warps][4]
    void *save;                // V [B][2][nsec]: psi after the forward program, sigma
};

__device__ __forceinline__ double2 s_cadd(double2 a, double2 b) {
    return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 s_cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 s_cjmul(double2 a, double2 b) {  // conj(a) b
    return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}

// Amplitude arithmetic for both storage types (complex double2, real double).
__device__ __forceinline__ double2 v_zero(double2) { return make_double2(0.0, 0.0); }
__device__ __forceinline__ double v_zero(double) { return 0.0; }
__device__ __forceinline__ void v_one(double2 &v) { v = make_double2(1.0, 0.0); }
__device__ __forceinline__ void v_one(double &v) { v = 1.0; }
template <class V>
__device__ __forceinline__ V v_one_of() {
    V v;
    v_one(v);
    return v;
}
// coefficient g times amplitude x (real storage: g is real)
__device__ __forceinline__ double2 v_mul(double2 g, double2 x) { return s_cmul(g, x); }
__device__ __forceinline__ double v_mul(double2 g, double x) { return g.x * x; }
__device__ __forceinline__ double v_mul(double g, double x) { return g * x; }
// c x + s y
__device__ __forceinline__ double2 v_lin(double c, double2 x, double s, double2 y) {
    return make_double2(c * x.x + s * y.x, c * x.y + s * y.y);
}
__device__ __forceinline__ double v_lin(double c, double x, double s, double y) { return c * x + s * y; }
// conj(a) b as a complex number
__device__ __forceinline__ double2 v_cj(double2 a, double2 b) { return s_cjmul(a, b); }
__device__ __forceinline__ double2 v_cj(double a, double b) { return make_double2(a * b, 0.0); }
// acc += f x (f a real matrix entry)
__device__ __forceinline__ void v_acc(double2 &acc, double f, double2 x) {
    acc.x += f * x.x;
    acc.y += f * x.y;
}
__device__ __forceinline__ void v_acc(double &acc, double f, double x) { acc += f * x; }
__device__ __forceinline__ double2 v_add(double2 a, double2 b) { return s_cadd(a, b); }
__device__ __forceinline__ double v_add(double a, double b) { return a + b; }
__device__ __forceinline__ double v_shfl_down(double v, int o) {
    return __shfl_down_sync(0xffffffffu, v, o);
}
__device__ __forceinline__ double2 v_shfl_down(double2 v, int o) {
    return make_double2(__shfl_down_sync(0xffffffffu, v.x, o), __shfl_down_sync(0xffffffffu, v.y, o));
}

// A pair's share of <w|K|v>: conj(w0) hn v1 + conj(w1) gn v0
__device__ __forceinline__ double v_ip(double w0, double w1, double v0, double v1, double gn,
                                       double hn) {
    return w0 * (hn * v1) + w1 * (gn * v0);
}
__device__ __forceinline__ double2 v_ip(double2 w0, double2 w1, double2 v0, double2 v1, double2 gn,
                                        double2 hn) {
    return s_cadd(s_cjmul(w0, s_cmul(hn, v1)), s_cjmul(w1, s_cmul(gn, v0)));
}
__device__ __forceinline__ double2 v_as2(double x) { return make_double2(x, 0.0); }
__device__ __forceinline__ double2 v_as2(double2 x) { return x; }

__device__ __forceinline__ PHead p_head(const PHead *p) {
    const int4 a = __ldg(reinterpret_cast<const int4 *>(p));
    const int4 b = __ldg(reinterpret_cast<const int4 *>(p) + 1);
    PHead h;
    h.p0 = a.x;
    h.np = a.y;
    h.fl = a.z;
    h.row = a.w;
    h.gamma = __hiloint2double(b.y, b.x);
    h.c0 = b.z;
    h.param = b.w;
    return h;
}

// The coefficients (gn, hn) of pattern k of a stream: real parts only for
// real amplitudes.
__device__ __forceinline__ void p_ldcoef(const PStream &S, int k, double &gn, double &hn) {
    gn = __ldg(reinterpret_cast<const double *>(S.coef + 2 * k));
    hn = __ldg(reinterpret_cast<const double *>(S.coef + 2 * k + 1));
}
__device__ __forceinline__ void p_ldcoef(const PStream &S, int k, double2 &gn, double2 &hn) {
    gn = __ldg(S.coef + 2 * k);
    hn = __ldg(S.coef + 2 * k + 1);
}

// Re of conj(w0) h v1 + conj(w1) g v0
__device__ __forceinline__ double v_ip_re(double w0, double w1, double v0, double v1, double g, double h) {
    return w0 * (h * v1) + w1 * (g * v0);
}
__device__ __forceinline__ double v_ip_re(double2 w0, double2 w1, double2 v0, double2 v1, double2 g, double2 h) {
    const double2 a = s_cmul(h, v1), b = s_cmul(g, v0);
    return (w0.x * a.x + w0.y * a.y) + (w1.x * b.x + w1.y * b.y);
}
__device__ __forceinline__ double v_of(double, double2 z, double f) { return z.x * f; }
__device__ __forceinline__ double2 v_of(double2, double2 z, double f) { return make_double2(z.x * f, z.y * f); }
// a, negated when bit 31 of w is set
__device__ __forceinline__ double v_flip(double a, uint32_t w) {
    return __hiloint2double(__double2hiint(a) ^ (int)(w & 0x80000000u), __double2loint(a));
}
__device__ __forceinline__ double2 v_flip(double2 a, uint32_t w) {
    return make_double2(v_flip(a.x, w), v_flip(a.y, w));
}
// c x + a y
__device__ __forceinline__ double v_rot(double c, double x, double a, double y) { return c * x + a * y; }
__device__ __forceinline__ double2 v_rot(double c, double2 x, double2 a, double2 y) {
    return make_double2(c * x.x + (a.x * y.x - a.y * y.y), c * x.y + (a.x * y.y + a.y * y.x));
}

// What a record's pairs are worked with, for one parameter set: cos, sin times
// the two coefficients and, in the sweep, gamma times them (zero without an
// inner product; cos 1 and sin 0 without a rotation).
template <bool SWEEP, class V>
struct __align__(16) PCoef;
template <class V>
struct __align__(16) PCoef<false, V> {
    V a, b;  // sin hn, sin gn
    double c, pad;
};
template <class V>
struct __align__(16) PCoef<true, V> {
    V a, b, h, g;
    double c, pad;
};
static_assert(sizeof(PCoef<true, double>) == 48 && sizeof(PCoef<true, double2>) == 80, "PCoef layout");

__device__ __forceinline__ RRec r_head(const RRec *p) {
    RRec h;
    const int4 a = __ldg(reinterpret_cast<const int4 *>(p));
    h.gamma = __hiloint2double(a.y, a.x);
    h.param = a.z;
    h.fl = a.w;
    h.gn = __ldg(&p->gn);
    h.hn = __ldg(&p->hn);
    return h;
}

// Every record's PCoef for the angles sign * gamma * theta, record r at cf[r + 1].
template <bool SWEEP, class V>
__device__ __forceinline__ void p_angles(const RStream &S, const double *par, int sign,
                                         PCoef<SWEEP, V> *cf) {
    for (int r = threadIdx.x; r < S.n; r += blockDim.x) {
        const RRec h = r_head(S.hd + r);
        double sn = 0.0, cs = 1.0;
        if (h.fl & R_ROT) sincos((double)sign * h.gamma * par[h.param], &sn, &cs);
        PCoef<SWEEP, V> o;
        o.c = cs;
        o.pad = 0.0;
        o.a = v_of(V(), h.hn, sn);
        o.b = v_of(V(), h.gn, sn);
        if constexpr (SWEEP) {
            const double f = (h.fl & R_IP) ? h.gamma : 0.0;
            o.h = v_of(V(), h.hn, f);
            o.g = v_of(V(), h.gn, f);
        }
        cf[r + 1] = o;
    }
}

__device__ __forceinline__ double v_shfl_xor(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double2 v_shfl_xor(double2 v, int o) {
    return make_double2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

template <class V>
__device__ __forceinline__ V p_sum1(V a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a = v_add(a, v_shfl_down(a, o));
    return a;
}

// Warp sums of four rounds' values on the FP64 matrix units: round j's lane
// values, as a 4 x 8 matrix, are multiplied from the left by ones in row j, so
// row j of the accumulators holds their 8 column sums (two per lane, lanes
// 4 j .. 4 j + 3).  One instruction a round instead of three shuffles.
struct RSum {
    double d0 = 0.0, d1 = 0.0;
    __device__ __forceinline__ void add(int j, double x) {
        const double a = ((threadIdx.x & 31) >> 2) == j ? 1.0 : 0.0;
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
            : "+d"(d0), "+d"(d1)
            : "d"(a), "d"(x));
    }
    // round j's sum in lanes 4 j .. 4 j + 3
    __device__ __forceinline__ double sum() const {
        double t = d0 + d1;
        t += v_shfl_xor(t, 1);
        return t + v_shfl_xor(t, 2);
    }
};

template <class V>
__device__ __forceinline__ V &r_at0(V *v, uint32_t w) {
    return *reinterpret_cast<V *>(reinterpret_cast<char *>(v) + (w & kWordIdx) * (uint32_t)(sizeof(V) / 8));
}
template <class V>
__device__ __forceinline__ V &r_at1(V *v, uint32_t w) {
    return *reinterpret_cast<V *>(reinterpret_cast<char *>(v) +
                                  ((w >> kPairIdxBits) & kWordIdx) * (uint32_t)(sizeof(V) / 8));
}

// One round: f rotates (and accumulates) the pair of `word` with the record's
// constants; the constants of the next round's record are loaded meanwhile.
template <bool REV, class C, class F>
__device__ __forceinline__ void r_round(uint32_t word, C &c, const C *&cf, int nth, const F &f) {
    cf += REV ? -(int)((word >> 1) & 1u) : (int)(word & 1u);
    const C next = *cf;
    f(word, c);
    c = next;
    asm volatile("bar.sync 1, %0;" ::"r"(nth) : "memory");
}

// Run a stream's rounds (REV: in reverse order), f(word, constants, j) per
// pair, j the round's number modulo 4, and done(r) after rounds r .. r + 3.
// Threads past S.nth do nothing.
//
// Bound by the latency of one round after another: a barrier, the amplitudes'
// way through shared memory, two dependent FP64 operations.  So nothing else
// lies on that path: no thread tests for its pair or its record's kind, the
// word was loaded four rounds before (L2), the constants one round before.
template <bool REV, class C, class F, class G>
__device__ __forceinline__ void r_run(const RStream &S, const C *cf, const F &f, const G &done) {
    const int nth = S.nth, tid = threadIdx.x;
    if (S.nr == 0 || tid >= nth) return;
    const int step = REV ? -nth : nth;
    const uint32_t *wp = S.word + (REV ? (size_t)(S.nr - 1) * nth : 0) + tid;
    cf += REV ? S.n : 1;
    C c = *cf;
    uint32_t w0 = __ldg(wp), w1 = __ldg(wp + step), w2 = __ldg(wp + 2 * step), w3 = __ldg(wp + 3 * step);
    for (int r = 0; r < S.nr; r += 4) {
        wp += 4 * step;
        const uint32_t n0 = __ldg(wp);
        r_round<REV>(w0, c, cf, nth, [&](uint32_t w, const C &k) { f(w, k, 0); });
        const uint32_t n1 = __ldg(wp + step);
        r_round<REV>(w1, c, cf, nth, [&](uint32_t w, const C &k) { f(w, k, 1); });
        const uint32_t n2 = __ldg(wp + 2 * step);
        r_round<REV>(w2, c, cf, nth, [&](uint32_t w, const C &k) { f(w, k, 2); });
        const uint32_t n3 = __ldg(wp + 3 * step);
        r_round<REV>(w3, c, cf, nth, [&](uint32_t w, const C &k) { f(w, k, 3); });
        done(r);
        w0 = n0;
        w1 = n1;
        w2 = n2;
        w3 = n3;
    }
}

// The forward program (REV: its inverse, with the angles' sign) on v.
template <bool REV, class V>
__device__ __forceinline__ void p_forward(const RStream &S, const PCoef<false, V> *cf, V *v) {
    r_run<REV>(
        S, cf,
        [&](uint32_t w, const PCoef<false, V> &k, int) {
            V &x0 = r_at0(v, w), &x1 = r_at1(v, w);
            const V v0 = x0, v1 = x1;
            x0 = v_rot(k.c, v0, v_flip(k.a, w), v1);
            x1 = v_rot(k.c, v1, v_flip(k.b, w), v0);
        },
        [](int) {});
}

// psi and sigma of the sweep in shared memory: complex amplitudes as two
// arrays, real ones interleaved (both states' amplitude in one 16-byte access).
template <class V>
struct SweepState;
template <>
struct SweepState<double> {
    double2 *x;
    __device__ __forceinline__ SweepState(unsigned char *raw, int) : x(reinterpret_cast<double2 *>(raw)) {}
    __device__ __forceinline__ void set(int i, double p, double s) { x[i] = make_double2(p, s); }
    __device__ __forceinline__ double round(uint32_t w, const PCoef<true, double> &k) {
        double2 &r0 = r_at0(x, w), &r1 = r_at1(x, w);
        const double2 v0 = r0, v1 = r1;
        const double a = v_flip(k.a, w), b = v_flip(k.b, w);
        r0 = make_double2(v_rot(k.c, v0.x, a, v1.x), v_rot(k.c, v0.y, a, v1.y));
        r1 = make_double2(v_rot(k.c, v1.x, b, v0.x), v_rot(k.c, v1.y, b, v0.y));
        return v_flip(v_ip_re(v0.y, v1.y, v0.x, v1.x, k.g, k.h), w);
    }
};
template <>
struct SweepState<double2> {
    double2 *v, *w;
    __device__ __forceinline__ SweepState(unsigned char *raw, int nsec)
        : v(reinterpret_cast<double2 *>(raw)), w(v + nsec + kRoundPad) {}
    __device__ __forceinline__ void set(int i, double2 p, double2 s) {
        v[i] = p;
        w[i] = s;
    }
    __device__ __forceinline__ double round(uint32_t word, const PCoef<true, double2> &k) {
        double2 &x0 = r_at0(v, word), &x1 = r_at1(v, word), &y0 = r_at0(w, word), &y1 = r_at1(w, word);
        const double2 v0 = x0, v1 = x1, w0 = y0, w1 = y1;
        const double2 a = v_flip(k.a, word), b = v_flip(k.b, word);
        x0 = v_rot(k.c, v0, a, v1);
        x1 = v_rot(k.c, v1, b, v0);
        y0 = v_rot(k.c, w0, a, w1);
        y1 = v_rot(k.c, w1, b, w0);
        return v_flip(v_ip_re(w0, w1, v0, v1, k.g, k.h), word);
    }
};
// psi and sigma of one slot from the save buffer (sig: its sigma)
template <class V>
__device__ __forceinline__ void sweep_load(SweepState<V> &st, const V *psi, const V *sig, int nsec) {
    for (int i = threadIdx.x; i < nsec + kRoundPad; i += blockDim.x)
        st.set(i, i < nsec ? psi[i] : v_zero(V()), i < nsec ? sig[i] : v_zero(V()));
}

// The reverse sweep; partial: this slot's [rounds / 4][warps][4] warp sums of
// the rounds' inner products.
template <class V>
__device__ __forceinline__ void p_sweep(const RStream &S, const PCoef<true, V> *cf, SweepState<V> &st,
                                        double *partial) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = S.nth >> 5;
    RSum ip;
    r_run<false>(
        S, cf, [&](uint32_t word, const PCoef<true, V> &k, int j) { ip.add(j, st.round(word, k)); },
        [&](int r) {
            const double t = ip.sum();
            if ((lane & 3) == 0 && lane < 16) partial[((size_t)(r >> 2) * nw + warp) * 4 + (lane >> 2)] = t;
            ip = RSum();
        });
}

// grad[mu] = 2 x the sums of parameter mu's rounds, in round and warp order
// (after a barrier that follows p_sweep).
__device__ __forceinline__ void p_grad(const int2 *prange, int nparam, int nw, const double *partial,
                                       double *grad) {
    for (int mu = threadIdx.x; mu < nparam; mu += blockDim.x) {
        const int2 pr = prange[mu];
        double acc = 0.0;
        for (int r = pr.x; r < pr.y; ++r)
            for (int k = 0; k < nw; ++k) acc += partial[((size_t)(r >> 2) * nw + k) * 4 + (r & 3)];
        grad[mu] = 2.0 * acc;
    }
}

// Shared memory of the step kernels: nstates states, each with kRoundPad unused
// amplitudes, then the records' constants (one unused on either side).
template <class C>
__host__ __device__ inline size_t step_smem(int nstates, int nsec, size_t elem, int nrec) {
    return ((nstates * (size_t)(nsec + kRoundPad) * elem + 15) & ~(size_t)15) + sizeof(C) * (size_t)(nrec + 2);
}
template <class C>
__device__ __forceinline__ C *step_coef(unsigned char *raw, int nstates, int nsec, size_t elem) {
    return reinterpret_cast<C *>(raw + ((nstates * (size_t)(nsec + kRoundPad) * elem + 15) & ~(size_t)15));
}
template <class V>
__device__ __forceinline__ void step_pad(V *v, int nsec) {
    for (int i = threadIdx.x; i < kRoundPad; i += blockDim.x) v[nsec + i] = v_zero(V());
}

// The evaluation runs as three kernels: the forward program (one CTA per
// parameter set, psi in shared memory), sigma = H psi with the energy (a few
// parameter sets and a slice of the rows per CTA, sigma rows straight to the
// save buffer), and the reverse sweep (one CTA per parameter set, psi and
// sigma in shared memory) with the gradient.

template <class V>
__global__ void __launch_bounds__(kStepThreads, 2) k_sector_forward(SLaunch L) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    V *psi = reinterpret_cast<V *>(s_raw);
    PCoef<false, V> *cf = step_coef<PCoef<false, V>>(s_raw, 1, L.nsec, sizeof(V));
    const int b = blockIdx.x, tid = threadIdx.x, nth = blockDim.x;
    const double *par = L.params + (size_t)b * L.nparam;
    for (int i = tid; i < L.nsec; i += nth) psi[i] = i == L.ref_i ? v_one_of<V>() : v_zero(V());
    step_pad(psi, L.nsec);
    p_angles<false, V>(L.fwd, par, 1, cf);
    __syncthreads();
    p_forward<false, V>(L.fwd, cf, psi);
    __syncthreads();
    V *sv = reinterpret_cast<V *>(L.save) + (size_t)b * 2 * L.nsec;
    for (int i = tid; i < L.nsec; i += nth) sv[i] = psi[i];
}

// sigma = H psi and the energy, P parameter sets per CTA.  CTA x works on
// group g = x / Q (sets g P .. g P + P - 1) and row slice q = x % Q: it loads
// the group's psi into shared memory, streams the slice's H rows once for all
// P sets (one warp per row, U entries in flight per lane, each entry's column
// gathered from every set), writes the sigma rows to the save
// buffer and one partial energy per set to epart[set][q].  The CTA that
// completes a group last (a ticket on count[g], which it resets) sums the
// group's partials in q order into energy, so the sum's order is fixed.
template <bool REAL, class V, int P, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_sector_h(
    SLaunch L, int nbatch, int Q, double *__restrict__ epart, unsigned *__restrict__ count) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ double s_red[NT / 32][P];
    __shared__ unsigned s_ticket;
    // real states of an even number of sets sit in pairs, [P / 2][nsec] of
    // double2 (sets 2h, 2h + 1): one 16-byte gather reads two sets
    constexpr bool PAIR = REAL && sizeof(V) == sizeof(double) && P % 2 == 0;
    V *psi = reinterpret_cast<V *>(s_raw);  // [P][nsec] unless PAIR
    double2 *ps2 = reinterpret_cast<double2 *>(s_raw);
    const int g = blockIdx.x / Q, q = blockIdx.x - g * Q, tid = threadIdx.x;
    const int b0 = g * P, nb = min(P, nbatch - b0), n = L.nsec;
    V *save = reinterpret_cast<V *>(L.save);
    if constexpr (PAIR) {
        const double *sd = reinterpret_cast<const double *>(L.save);
#pragma unroll
        for (int h = 0; h < P / 2; ++h) {
            const double *s0 = sd + (size_t)(b0 + (2 * h < nb ? 2 * h : 0)) * 2 * n;
            const double *s1 = sd + (size_t)(b0 + (2 * h + 1 < nb ? 2 * h + 1 : 0)) * 2 * n;
            for (int i = tid; i < n; i += NT) ps2[h * n + i] = make_double2(s0[i], s1[i]);
        }
    } else {
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const V *sv = save + (size_t)(b0 + (p < nb ? p : 0)) * 2 * n;
            for (int i = tid; i < n; i += NT) psi[p * n + i] = sv[i];
        }
    }
    __syncthreads();
    const int r0 = (int)((int64_t)q * n / Q), r1 = (int)((int64_t)(q + 1) * n / Q);
    const int lane = tid & 31, warp = tid >> 5;
    constexpr int U = P >= 2 ? 4 : 8;  // H row entries in flight per lane
    // after a row's reduction, lane GL p holds set p's sum (GL lanes per set)
    constexpr int GL = 32 / P;
    const int lp = lane / GL;
    double en = 0.0;  // energy share of set lp (lanes lane % GL == 0)
    for (int i = r0 + warp; i < r1; i += NT / 32) {
        V acc[P];
#pragma unroll
        for (int p = 0; p < P; ++p) acc[p] = v_zero(V());
        const int e1 = L.rowptr[i + 1];
        for (int e0 = L.rowptr[i] + lane; e0 < e1; e0 += 32 * U) {
            uint32_t c[U];
            double fr[REAL ? U : 1];
            double2 fc[REAL ? 1 : U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + 32 * u;
                c[u] = (e < e1) ? __ldg(&L.col[e]) : 0u;
                if (REAL) fr[u] = (e < e1) ? __ldg(&L.val_r[e]) : 0.0;
                else fc[REAL ? 0 : u] = (e < e1) ? __ldg(&L.val_c[e]) : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if constexpr (PAIR) {
#pragma unroll
                    for (int h = 0; h < P / 2; ++h) {
                        const double2 x = ps2[h * n + (int)c[u]];
                        v_acc(acc[2 * h], fr[u], x.x);
                        v_acc(acc[2 * h + 1], fr[u], x.y);
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < P; ++p) {
                        const V x = psi[p * n + (int)c[u]];
                        if constexpr (REAL) {
                            v_acc(acc[p], fr[u], x);
                        } else {
                            acc[p] = v_add(acc[p], v_mul(fc[REAL ? 0 : u], x));
                        }
                    }
                }
            }
        }
        // reduce-scatter: each exchange halves the values a lane carries
        V m;
        if constexpr (P == 4) {
            const bool b4 = lane & 16, b3 = lane & 8;
            const V k0 = v_add(b4 ? acc[2] : acc[0], v_shfl_xor(b4 ? acc[0] : acc[2], 16));
            const V k1 = v_add(b4 ? acc[3] : acc[1], v_shfl_xor(b4 ? acc[1] : acc[3], 16));
            m = v_add(b3 ? k1 : k0, v_shfl_xor(b3 ? k0 : k1, 8));
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) m = v_add(m, v_shfl_down(m, o));
        } else if constexpr (P == 2) {
            const bool b4 = lane & 16;
            m = v_add(b4 ? acc[1] : acc[0], v_shfl_xor(b4 ? acc[0] : acc[1], 16));
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) m = v_add(m, v_shfl_down(m, o));
        } else {
            m = acc[0];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = v_add(m, v_shfl_down(m, o));
        }
        if ((lane & (GL - 1)) == 0) {
            if (lp < nb) save[(size_t)(b0 + lp) * 2 * n + n + i] = m;
            V pv;
            if constexpr (PAIR) {
                const double2 x = ps2[(lp >> 1) * n + i];
                pv = (lp & 1) ? x.y : x.x;
            } else {
                pv = psi[lp * n + i];
            }
            en += v_cj(pv, m).x;
        }
    }
    if ((lane & (GL - 1)) == 0) s_red[warp][lp] = en;
    __syncthreads();
    if (tid == 0) {
        for (int p = 0; p < nb; ++p) {
            double t = 0.0;
            for (int k = 0; k < NT / 32; ++k) t += s_red[k][p];
            epart[(size_t)(b0 + p) * Q + q] = t;
        }
        __threadfence();
        s_ticket = atomicAdd(&count[g], 1u);
    }
    __syncthreads();
    if (s_ticket == (unsigned)Q - 1u) {  // every slice of the group is in
        __threadfence();
        if (tid < nb) {
            double t = 0.0;
            for (int k = 0; k < Q; ++k) t += __ldcg(&epart[(size_t)(b0 + tid) * Q + k]);
            L.energy[b0 + tid] = t;
        }
        if (tid == 0) count[g] = 0u;
    }
}

template <class V>
__global__ void __launch_bounds__(kStepThreads, sizeof(V) == sizeof(double) ? 2 : 1) k_sector_sweep(SLaunch L) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    SweepState<V> st(s_raw, L.nsec);
    PCoef<true, V> *cf = step_coef<PCoef<true, V>>(s_raw, 2, L.nsec, sizeof(V));
    const int b = blockIdx.x;
    const V *sv = reinterpret_cast<const V *>(L.save) + (size_t)b * 2 * L.nsec;
    sweep_load(st, sv, sv + L.nsec, L.nsec);
    p_angles<true, V>(L.sweep, L.params + (size_t)b * L.nparam, -1, cf);
    __syncthreads();
    double *part = L.partial + (size_t)b * L.sweep.nr * (L.sweep.nth >> 5);
    p_sweep<V>(L.sweep, cf, st, part);
    __syncthreads();
    p_grad(L.prange, L.nparam, L.sweep.nth >> 5, part, L.grad + (size_t)b * L.nparam);
}

// PQE residuals on the compact states: sigma of slot blockIdx.x from the save
// buffer, U^dagger applied to it in shared memory (the forward rounds in
// reverse order, angles negated), then
// res[b][k] = Re(sigma[idx[k]] * phase[k]) (0 where idx[k] < 0).
template <class V>
__global__ void __launch_bounds__(kStepThreads, 2) k_sector_resid(SLaunch L, const int64_t *__restrict__ idx,
                                                                  const double2 *__restrict__ phase,
                                                                  int nres, double *__restrict__ res) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    V *sig = reinterpret_cast<V *>(s_raw);
    PCoef<false, V> *cf = step_coef<PCoef<false, V>>(s_raw, 1, L.nsec, sizeof(V));
    const int b = blockIdx.x, tid = threadIdx.x, nth = blockDim.x;
    const double *par = L.params + (size_t)b * L.nparam;
    const V *sv = reinterpret_cast<const V *>(L.save) + (size_t)b * 2 * L.nsec + L.nsec;
    for (int i = tid; i < L.nsec; i += nth) sig[i] = sv[i];
    step_pad(sig, L.nsec);
    p_angles<false, V>(L.fwd, par, -1, cf);
    __syncthreads();
    p_forward<true, V>(L.fwd, cf, sig);
    __syncthreads();
    for (int k = tid; k < nres; k += nth) {
        const int64_t i = idx[k];
        double r = 0.0;
        if (i >= 0) {
            const double2 v = v_cj(v_one_of<V>(), sig[i]), ph = phase[k];
            r = v.x * ph.x - v.y * ph.y;
        }
        res[(size_t)b * nres + k] = r;
    }
}

// Pool inner products on the compact states: each CTA loads psi and sigma of
// slot blockIdx.y and runs the inner-product records r = blockIdx.x,
// blockIdx.x + gridDim.x, ... of the pool stream.  The records leave the
// states unchanged, so they need no barrier between them.
template <class V>
__global__ void __launch_bounds__(512, 2) k_sector_pool(SLaunch L, PStream P, double2 *__restrict__ partial) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    V *psi = reinterpret_cast<V *>(s_raw), *sig = psi + L.nsec;
    const int b = blockIdx.y, tid = threadIdx.x, nth = blockDim.x, nw = nth >> 5;
    const V *sv = reinterpret_cast<const V *>(L.save) + (size_t)b * 2 * L.nsec;
    for (int i = tid; i < 2 * L.nsec; i += nth) psi[i] = sv[i];
    __syncthreads();
    for (int r = blockIdx.x; r < P.n; r += gridDim.x) {
        const PHead h = p_head(P.hd + r);
        const bool one = (h.fl >> 8) == 1;
        V gn = v_zero(V()), hn = gn;
        if (one) p_ldcoef(P, h.c0, gn, hn);
        V acc = v_zero(V());
        for (int k = tid; k < h.np; k += nth) {
            const uint32_t word = __ldg(P.pair + h.p0 + k);
            constexpr uint32_t M = (1u << kPairIdxBits) - 1u;
            const uint32_t i0 = word & M, i1 = (word >> kPairIdxBits) & M;
            if (!one) p_ldcoef(P, h.c0 + (int)(word >> (2 * kPairIdxBits + 1)), gn, hn);
            const double f = (word >> (2 * kPairIdxBits)) & 1u ? -h.gamma : h.gamma;
            v_acc(acc, f, v_ip(sig[i0], sig[i1], psi[i0], psi[i1], gn, hn));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc = v_add(acc, v_shfl_down(acc, o));
        if ((tid & 31) == 0) partial[((size_t)h.row * gridDim.y + b) * nw + (tid >> 5)] = v_as2(acc);
    }
}

// ---------------------------------------------------------------------------
// Two real parameter sets per CTA (forward program)
// ---------------------------------------------------------------------------
// With real states, sets 2g and 2g + 1 share one CTA of the forward program:
// amplitude slot i holds both sets' values as one double2 (.x set 2g, .y set
// 2g + 1), so every pair word, record header, shared-memory load / store and
// barrier serves both sets, while each set keeps its own angle (cos / sin per
// set in the record).  The arithmetic on each set is that of k_sector_forward.
// (The reverse sweep stays one set per CTA: its 16-byte slot holds the set's
// psi and sigma.)

struct __align__(16) PCoefPR {
    double2 c, a, b;  // cos, sin hn, sin gn: .x first set, .y second
};

__device__ __forceinline__ void p_angles_pr(const RStream &S, const double *parA, const double *parB,
                                            PCoefPR *cf) {
    for (int r = threadIdx.x; r < S.n; r += blockDim.x) {
        const RRec h = r_head(S.hd + r);
        double sa = 0.0, ca = 1.0, sb = 0.0, cb = 1.0;
        if (h.fl & R_ROT) {
            sincos(h.gamma * parA[h.param], &sa, &ca);
            sincos(h.gamma * parB[h.param], &sb, &cb);
        }
        cf[r + 1] = PCoefPR{make_double2(ca, cb), make_double2(sa * h.hn.x, sb * h.hn.x),
                            make_double2(sa * h.gn.x, sb * h.gn.x)};
    }
}

__device__ __forceinline__ void pr_forward(const RStream &S, const PCoefPR *cf, double2 *v) {
    r_run<false>(
        S, cf,
        [&](uint32_t w, const PCoefPR &k, int) {
            double2 &x0 = r_at0(v, w), &x1 = r_at1(v, w);
            const double2 v0 = x0, v1 = x1;
            const double2 a = v_flip(k.a, w), b = v_flip(k.b, w);
            x0 = make_double2(v_rot(k.c.x, v0.x, a.x, v1.x), v_rot(k.c.y, v0.y, a.y, v1.y));
            x1 = make_double2(v_rot(k.c.x, v1.x, b.x, v0.x), v_rot(k.c.y, v1.y, b.y, v0.y));
        },
        [](int) {});
}

// Forward program of sets 2g, 2g + 1 (g = blockIdx.x; a last odd set runs
// alone, its twin a copy that is not saved); psi of both into the save buffer.
__global__ void __launch_bounds__(kStepThreads, 1) k_sector_forward_pr(SLaunch L, int nbatch) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    double2 *psi = reinterpret_cast<double2 *>(s_raw);
    PCoefPR *cf = step_coef<PCoefPR>(s_raw, 1, L.nsec, sizeof(double2));
    const int b0 = 2 * blockIdx.x, tid = threadIdx.x, nth = blockDim.x;
    const bool two = b0 + 1 < nbatch;
    const double *parA = L.params + (size_t)b0 * L.nparam;
    const double *parB = two ? parA + L.nparam : parA;
    for (int i = tid; i < L.nsec; i += nth)
        psi[i] = i == L.ref_i ? make_double2(1.0, 1.0) : make_double2(0.0, 0.0);
    step_pad(psi, L.nsec);
    p_angles_pr(L.fwd, parA, parB, cf);
    __syncthreads();
    pr_forward(L.fwd, cf, psi);
    __syncthreads();
    double *sv = reinterpret_cast<double *>(L.save) + (size_t)b0 * 2 * L.nsec;
    for (int i = tid; i < L.nsec; i += nth) {
        const double2 x = psi[i];
        sv[i] = x.x;
        if (two) sv[2 * (size_t)L.nsec + i] = x.y;
    }
}

// ---------------------------------------------------------------------------
// Packed evaluations of several problems in one launch
// ---------------------------------------------------------------------------

// One problem of a packed launch: the compact evaluator data of one dUCC
// problem (its sector, forward and sweep rounds, H rows on the sector and the
// sweep rounds of each parameter).
struct PackMember {
    int nsec, ref_i, nparam;
    int Q;  // CTAs its H rows are split over (its own: an energy's sum never depends on the mix)
    RStream fwd, sweep;
    const int32_t *rowptr;
    const uint32_t *col;
    const double *val_r;   // real H (val_c == nullptr) ...
    const double2 *val_c;  // ... or complex
    const int2 *prange;    // rounds of the sweep of each parameter
};

// A packed launch's buffers.
struct PackLaunch {
    const PackMember *members;
    const int2 *items;  // (problem, with gradient)
    int nmem, maxparam;
    const double *params;  // [items][maxparam]
    double *energy, *grad;
    double *partial;       // [items][maxpart]: the sweeps' warp sums
    size_t maxpart;
    void *save;            // V [items][2][maxsec]: psi, sigma
    int maxsec, Q;         // Q: the most CTAs of a member
    double *epart;         // [items][Q]
    unsigned *count;       // [items]: CTAs done
};

// Rows r0 .. r1 of sigma = H psi (a warp per row, the lanes over the row's
// entries) and, in warp 0, this CTA's share of <psi|H|psi>, its rows' parts (s_en,
// kPackRows of them) summed in an order that does not depend on the block.
constexpr int kPackRows = 512;
template <class V>
__device__ __forceinline__ double p_hpsi(const PackMember &m, int r0, int r1, const V *psi, V *sig,
                                         double *s_en) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    constexpr int U = 4;  // row entries in flight per lane
    for (int i = r0 + warp; i < r1; i += nw) {
        V acc = v_zero(V());
        const int e1 = m.rowptr[i + 1];
        for (int e0 = m.rowptr[i] + lane; e0 < e1; e0 += 32 * U) {
            uint32_t c[U];
            double fr[U];
            double2 fc[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + 32 * u;
                const bool in = e < e1;
                c[u] = in ? __ldg(&m.col[e]) : 0u;
                if (sizeof(V) == sizeof(double2) && m.val_c) {
                    fc[u] = in ? __ldg(&m.val_c[e]) : make_double2(0.0, 0.0);
                    fr[u] = 0.0;
                } else {
                    fr[u] = in ? __ldg(&m.val_r[e]) : 0.0;
                    fc[u] = make_double2(0.0, 0.0);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const V x = psi[c[u]];
                if constexpr (sizeof(V) == sizeof(double2)) {
                    if (m.val_c) acc = v_add(acc, v_mul(fc[u], x));
                    else v_acc(acc, fr[u], x);
                } else {
                    v_acc(acc, fr[u], x);
                }
            }
        }
        acc = p_sum1(acc);
        if (lane == 0) {
            sig[i] = acc;
            s_en[i - r0] = v_cj(psi[i], acc).x;
        }
    }
    __syncthreads();
    double t = 0.0;
    if (warp == 0) {
        for (int k = lane; k < r1 - r0; k += 32) t += s_en[k];
        t = p_sum1(t);
    }
    return t;
}

// One item's forward program: psi = U(t)|ref> in shared memory.
template <class V>
__device__ __forceinline__ void pack_forward(const PackMember &m, const double *par, V *psi,
                                             PCoef<false, V> *cf) {
    const int tid = threadIdx.x, nth = blockDim.x;
    for (int i = tid; i < m.nsec; i += nth) psi[i] = i == m.ref_i ? v_one_of<V>() : v_zero(V());
    step_pad(psi, m.nsec);
    p_angles<false, V>(m.fwd, par, 1, cf);
    __syncthreads();
    p_forward<false, V>(m.fwd, cf, psi);
    __syncthreads();
}

// One item's reverse sweep on psi and sig (save buffer) and its gradient.
template <class V>
__device__ __forceinline__ void pack_sweep(const PackLaunch &P, const PackMember &m, const double *par,
                                           const V *psi, const V *sig, unsigned char *raw) {
    SweepState<V> st(raw, m.nsec);
    PCoef<true, V> *cf = step_coef<PCoef<true, V>>(raw, 2, m.nsec, sizeof(V));
    sweep_load(st, psi, sig, m.nsec);
    p_angles<true, V>(m.sweep, par, -1, cf);
    __syncthreads();
    double *pp = P.partial + (size_t)blockIdx.x * P.maxpart;
    p_sweep<V>(m.sweep, cf, st, pp);
    __syncthreads();  // this CTA's partials are visible to all its threads
    p_grad(m.prange, m.nparam, m.sweep.nth >> 5, pp, P.grad + (size_t)blockIdx.x * P.maxparam);
}

// The item of CTA x, or nothing for a number that is no problem's (its energy
// is NaN).
__device__ __forceinline__ bool pack_item(const PackLaunch &P, int x, int2 &it) {
    it = P.items[x];
    if ((unsigned)it.x < (unsigned)P.nmem) return true;
    if (threadIdx.x == 0) P.energy[x] = __longlong_as_double(0x7ff8000000000000ll);
    return false;
}

// Item x is parameter set params[x][0 .. nparam) of problem items[x].x, with its
// gradient when items[x].y != 0; energy into energy[x], gradient into
// grad[x][0 .. nparam).  Three launches serve parameter sets of different
// problems side by side: the forward programs (a CTA per item), sigma = H psi
// and the energies (up to 16 CTAs per item: one alone takes ~400 us for the 1.8 M row
// entries of a 16-qubit problem), the reverse sweeps (a CTA per item).
template <class V>
__global__ void __launch_bounds__(kStepThreads, 2) k_pack_forward(PackLaunch P) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    int2 it;
    if (!pack_item(P, blockIdx.x, it)) return;
    const PackMember m = P.members[it.x];
    V *psi = reinterpret_cast<V *>(s_raw);
    pack_forward<V>(m, P.params + (size_t)blockIdx.x * P.maxparam, psi,
                    step_coef<PCoef<false, V>>(s_raw, 1, m.nsec, sizeof(V)));
    V *sv = reinterpret_cast<V *>(P.save) + (size_t)blockIdx.x * 2 * P.maxsec;
    for (int i = threadIdx.x; i < m.nsec; i += blockDim.x) sv[i] = psi[i];
}

// CTA (q, x): row slice q of item x's sigma and its share of the energy; the
// CTA that finishes an item last (a ticket, which it resets) adds the shares
// in order.
template <class V>
__global__ void __launch_bounds__(kStepThreads, 2) k_pack_h(PackLaunch P) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ double s_en[kPackRows];
    const int x = blockIdx.y, q = blockIdx.x, tid = threadIdx.x;
    const int2 it = P.items[x];
    if ((unsigned)it.x >= (unsigned)P.nmem) return;
    const PackMember m = P.members[it.x];
    if (q >= m.Q) return;
    V *psi = reinterpret_cast<V *>(s_raw);
    V *sv = reinterpret_cast<V *>(P.save) + (size_t)x * 2 * P.maxsec;
    for (int i = tid; i < m.nsec; i += blockDim.x) psi[i] = sv[i];
    __syncthreads();
    const int r0 = (int)((int64_t)q * m.nsec / m.Q), r1 = (int)((int64_t)(q + 1) * m.nsec / m.Q);
    const double e = p_hpsi<V>(m, r0, r1, psi, sv + P.maxsec, s_en);
    if (tid == 0) {
        P.epart[(size_t)x * P.Q + q] = e;
        __threadfence();
        if (atomicAdd(&P.count[x], 1u) == (unsigned)m.Q - 1u) {
            __threadfence();
            double t = 0.0;
            for (int k = 0; k < m.Q; ++k) t += __ldcg(&P.epart[(size_t)x * P.Q + k]);
            P.energy[x] = t;
            P.count[x] = 0u;
        }
    }
}

// The three in one CTA per item, for members whose rows one CTA takes (sectors below
// 256 amplitudes): the launches would take longer than the work.  Energy and gradient,
// us, three launches / this kernel: 64 items of 4 amplitudes 14.8 / 8.3, of 36 20.6 /
// 14.4, of 100 29.8 / 21.5; 2,000 items 53 / 17, 70 / 53 and 114 / 90.
template <class V>
__global__ void __launch_bounds__(kStepThreads, sizeof(V) == sizeof(double) ? 2 : 1) k_pack_one(PackLaunch P) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ double s_en[kPackRows];
    int2 it;
    if (!pack_item(P, blockIdx.x, it)) return;
    const PackMember m = P.members[it.x];
    V *psi = reinterpret_cast<V *>(s_raw);
    const double *par = P.params + (size_t)blockIdx.x * P.maxparam;
    pack_forward<V>(m, par, psi, step_coef<PCoef<false, V>>(s_raw, 1, m.nsec, sizeof(V)));
    V *sv = reinterpret_cast<V *>(P.save) + (size_t)blockIdx.x * 2 * P.maxsec;
    const double e = p_hpsi<V>(m, 0, m.nsec, psi, sv + P.maxsec, s_en);
    if (threadIdx.x == 0) P.energy[blockIdx.x] = e;
    if (!it.y || m.nparam == 0) return;
    for (int i = threadIdx.x; i < m.nsec; i += blockDim.x) sv[i] = psi[i];
    __syncthreads();  // psi and sigma are in the save buffer
    pack_sweep<V>(P, m, par, sv, sv + P.maxsec, s_raw);
}

template <class V>
__global__ void __launch_bounds__(kStepThreads, sizeof(V) == sizeof(double) ? 2 : 1) k_pack_sweep(PackLaunch P) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int2 it = P.items[blockIdx.x];
    if ((unsigned)it.x >= (unsigned)P.nmem || !it.y) return;
    const PackMember m = P.members[it.x];
    if (m.nparam == 0) return;
    const V *sv = reinterpret_cast<const V *>(P.save) + (size_t)blockIdx.x * 2 * P.maxsec;
    pack_sweep<V>(P, m, P.params + (size_t)blockIdx.x * P.maxparam, sv, sv + P.maxsec, s_raw);
}

// Shared-memory bytes of nstates states of nsec amplitudes.
inline size_t sector_smem_states(size_t nstates, size_t nsec, bool real) {
    return ((nstates * nsec * (real ? 8 : 16)) + 15) & ~(size_t)15;
}

}  // namespace qfbs
