// Windows of program steps on blocks of a particle-number sector.
//
// The global-memory sector path (qfb_csec.cuh) keeps psi and sigma of a
// sector too large for one CTA's shared memory.  A launch per program step is
// bound by launch and L2 latency: a 20-qubit step moves ~5,000 pairs in 2.9 us.
// A step's pairs never leave the determinants that agree outside the step's
// orbitals, so for a run of consecutive steps whose x-masks lie in an orbital
// set Q the sector splits into independent blocks, one per assignment of the
// orbitals outside Q.  Alpha and beta strings factor: a block is a class of
// alpha strings (equal outside Q) times a class of beta strings.  One CTA loads
// a block, applies every step of the window to it in shared memory and writes
// it back: one launch and one read and write of the state per window.  SD
// program, one set of real amplitudes: 20 qubits (875 steps, 17 windows) forward
// 2,538 -> 216 us, sweep 3,282 -> 280 us; 18 qubits (560 steps, 9 windows)
// 1,622 -> 126 us and 2,061 -> 170 us, 8 sets 1,569 -> 155 us and 1,895 -> 238 us.
//
// A step's pairs on a block are an alpha list times a beta list of local
// (index, partner, sign) entries; the lists of all the window's items (a step
// has one item per pattern) for one class lie together (a class's blob), so a
// CTA stages two contiguous pieces.  It does so before it waits for the
// preceding grid (programmatic dependent launch), as the lists do not depend
// on the state.  Each slot (parameter set) is worked on by its own warps,
// with a warp barrier per round (one warp a slot) or a named barrier.
#pragma once

#include "qfb_csec.cuh"

namespace qfbv {

using qfbg::GLaunch;
using qfbs::v_flip;
using qfbs::v_ip_re;
using qfbs::v_of;
using qfbs::v_rot;

constexpr int kWinItems = 192;    // items of a window
constexpr int kWinIdx = 12;       // bits of a local string or amplitude index
constexpr int kWinBlobMax = 6144; // words of one class's blob
constexpr int kWinThreads = 512;  // threads of a CTA, at most

// One item: a step's pattern.
struct VItem {
    double gamma;
    int32_t ang;   // entry of the angle table
    int32_t fl;    // R_ROT | R_IP | R_TWO
    int64_t poff;  // R_IP: first partial (per slot), in units of the batch
    int32_t r0, r1;  // its rounds
    double2 gn, hn;
};
static_assert(sizeof(VItem) == 64, "VItem layout");

// A class of strings: its first rank in the rank table, its strings, and its
// blob: nitem + 1 entry offsets, nitem reciprocals ceil(2^32 / count) (0 for
// counts below 2), then the entries l0 | l1 << 12 | sign << 24.
struct VClass {
    int32_t rank0, n, blob0, words;
};

struct VWin {
    int32_t nca, ncb;    // classes: blocks are nca * ncb
    int32_t ca0, cb0;    // first alpha / beta class
    int32_t item0, nitem;
    int32_t mab, mranks, mwords;  // largest block, strings and blob words of one
    int32_t nround, lg;           // rounds of 32 << lg pairs
};

struct VTabs {
    const VClass *cls;
    const uint16_t *rank;
    const uint32_t *blob;
    const VItem *item;
};

// What a slot needs in a round: cos, sin times the two coefficients and, in
// the sweep, gamma times them (zero where the item has no inner product).
template <bool SWEEP, class V>
struct VCoef;
template <class V>
struct VCoef<false, V> {
    V a, b;  // sin hn, sin gn
    double c, pad;
};
template <class V>
struct VCoef<true, V> {
    V a, b, h, g;
    double c, pad;
};

// Shared memory of a CTA of `spc` slots and `nw` warps, in this order: states
// (each followed by 32 unused amplitudes), coefficients, items, round sums,
// blobs, ranks, amplitude indices, pair words.
__host__ __device__ inline size_t win_al(size_t x) { return (x + 15) & ~(size_t)15; }
inline size_t win_smem(const VWin &w, int spc, int nw, bool sweep, size_t elem) {
    const size_t cf = elem * (sweep ? 4 : 2) + 16;
    return win_al(elem * (size_t)(w.mab + 32) * spc * (sweep ? 2 : 1)) + cf * (size_t)w.nround * spc +
           sizeof(VItem) * w.nitem +
           (sweep ? win_al(sizeof(double) * (size_t)w.nround * nw) : 0) +
           win_al(4 * (size_t)w.mwords) + win_al(2 * (size_t)w.mranks) + win_al(4 * (size_t)w.mab) +
           4 * ((size_t)w.nround << (5 + w.lg));
}

// A slot's states in shared memory: psi, and in the sweep sigma, interleaved
// where the amplitudes are real (both in one 16-byte access).
template <bool SWEEP, class V>
struct WinState {
    V *v, *w;
    __device__ __forceinline__ WinState(unsigned char *raw, int sl, int stride, int lspc)
        : v(reinterpret_cast<V *>(raw) + sl * stride), w(v + (stride << lspc)) {}
    __device__ __forceinline__ void set(int i, V p, V s) {
        v[i] = p;
        if (SWEEP) w[i] = s;
    }
    __device__ __forceinline__ V psi(int i) const { return v[i]; }
    __device__ __forceinline__ V sig(int i) const { return w[i]; }
    // rotate the pair (l0, l1); sg: bit 31 is its sign.  The pair's inner product.
    __device__ __forceinline__ double round(uint32_t l0, uint32_t l1, uint32_t sg, const VCoef<SWEEP, V> &co) {
        const V v0 = v[l0], v1 = v[l1], a = v_flip(co.a, sg), b = v_flip(co.b, sg);
        V x0 = V(), x1 = V();
        if (SWEEP) {
            x0 = w[l0];
            x1 = w[l1];
        }
        v[l0] = v_rot(co.c, v0, a, v1);
        v[l1] = v_rot(co.c, v1, b, v0);
        if constexpr (SWEEP) {
            w[l0] = v_rot(co.c, x0, a, x1);
            w[l1] = v_rot(co.c, x1, b, x0);
            return v_flip(v_ip_re(x0, x1, v0, v1, co.g, co.h), sg);
        }
        return 0.0;
    }
};
template <>
struct WinState<true, double> {
    double2 *x;
    __device__ __forceinline__ WinState(unsigned char *raw, int sl, int stride, int)
        : x(reinterpret_cast<double2 *>(raw) + sl * stride) {}
    __device__ __forceinline__ void set(int i, double p, double s) { x[i] = make_double2(p, s); }
    __device__ __forceinline__ double psi(int i) const { return x[i].x; }
    __device__ __forceinline__ double sig(int i) const { return x[i].y; }
    __device__ __forceinline__ double round(uint32_t l0, uint32_t l1, uint32_t sg, const VCoef<true, double> &co) {
        const double2 v0 = x[l0], v1 = x[l1];
        const double a = v_flip(co.a, sg), b = v_flip(co.b, sg);
        x[l0] = make_double2(v_rot(co.c, v0.x, a, v1.x), v_rot(co.c, v0.y, a, v1.y));
        x[l1] = make_double2(v_rot(co.c, v1.x, b, v0.x), v_rot(co.c, v1.y, b, v0.y));
        return v_flip(v_ip_re(v0.y, v1.y, v0.x, v1.x, co.g, co.h), sg);
    }
};

// ang[i * B + s] = (cos, sin) of gamma_i * params[s][param_i]
__global__ void __launch_bounds__(256) k_win_angles(const double *__restrict__ gamma,
                                                    const int32_t *__restrict__ param, int n, int B,
                                                    const double *__restrict__ params, int nparam,
                                                    double2 *__restrict__ ang) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)n * B) return;
    const int i = (int)(t / B), s = (int)(t - (int64_t)i * B);
    double sn, cs;
    sincos(gamma[i] * params[(size_t)s * nparam + param[i]], &sn, &cs);
    ang[t] = make_double2(cs, sn);
}

// Apply window W to every block and the slots from slot0 on.  grid = (blocks, slot
// groups); 1 << lspc slots per CTA, 1 << W.lg warps per slot.  rev: items in reverse
// order; sign multiplies every angle (rev with sign -1: the exact inverse).
//
// Bound by the latency of one round after another (a barrier, a shared-memory
// round trip and two dependent FP64 operations: ~90 cycles with 4 warps), so
// a round holds nothing else: everything that does not depend on the state is
// done before the wait for the preceding grid.  The lists are expanded into
// one word per pair (l0 | l1 << 12 | sign << 31), padded to whole rounds with
// pairs of unused amplitudes, and the words and coefficients of a round are
// loaded one round ahead.
template <bool SWEEP, class V>
__global__ void __launch_bounds__(kWinThreads) k_win(GLaunch L, VWin W, VTabs T,
                                                     const double2 *__restrict__ ang, double sign, int rev,
                                                     int lspc, int slot0, double *__restrict__ partial) {
    extern __shared__ __align__(16) unsigned char w_raw[];
    const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nth >> 5;
    const int spc = 1 << lspc, ni = W.nitem, nr = W.nround, lg = W.lg, G = 32 << lg;
    const int ca = blockIdx.x / W.ncb, cb = blockIdx.x - ca * W.ncb;
    const int4 A = __ldg(reinterpret_cast<const int4 *>(T.cls + W.ca0 + ca));
    const int4 Bc = __ldg(reinterpret_cast<const int4 *>(T.cls + W.cb0 + cb));
    const int na = A.y, nb = Bc.y, nab = na * nb, stride = nab + 32;
    unsigned char *p = w_raw;
    p += win_al(sizeof(V) * (stride << lspc) * (SWEEP ? 2 : 1));
    VCoef<SWEEP, V> *s_cf = reinterpret_cast<VCoef<SWEEP, V> *>(p);  // [slot][round]
    p += sizeof(VCoef<SWEEP, V>) * nr << lspc;
    VItem *s_item = reinterpret_cast<VItem *>(p);
    p += sizeof(VItem) * ni;
    double *s_sum = nullptr;  // sums [warp][round]
    if (SWEEP) {
        s_sum = reinterpret_cast<double *>(p);
        p += win_al(sizeof(double) * nr * nw);
    }
    uint32_t *s_a = reinterpret_cast<uint32_t *>(p), *s_b = s_a + A.w;
    p += win_al(4 * (A.w + Bc.w));
    uint16_t *s_ra = reinterpret_cast<uint16_t *>(p), *s_rb = s_ra + na;
    p += win_al(2 * (na + nb));
    uint32_t *s_g = reinterpret_cast<uint32_t *>(p);
    p += win_al(4 * nab);
    uint32_t *s_w = reinterpret_cast<uint32_t *>(p);
    constexpr uint32_t M = (1u << kWinIdx) - 1u;

    // the window's lists (independent of the state)
    for (int i = tid; i < A.w; i += nth) s_a[i] = __ldg(T.blob + A.z + i);
    for (int i = tid; i < Bc.w; i += nth) s_b[i] = __ldg(T.blob + Bc.z + i);
    for (int i = tid; i < na; i += nth) s_ra[i] = __ldg(T.rank + A.x + i);
    for (int i = tid; i < nb; i += nth) s_rb[i] = __ldg(T.rank + Bc.x + i);
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(T.item + W.item0);
        uint4 *dst = reinterpret_cast<uint4 *>(s_item);
        for (int i = tid; i < 4 * ni; i += nth) dst[i] = __ldg(src + i);
    }
    __syncthreads();
    for (int la = warp; la < na; la += nw)
        for (int lb = lane; lb < nb; lb += 32) s_g[la * nb + lb] = (uint32_t)s_ra[la] * L.nbeta + s_rb[lb];
    for (int k = warp; k < ni; k += nw) {
        const int a0 = (int)s_a[k], b0 = (int)s_b[k], cnt = (int)s_b[k + 1] - b0;
        const int total = ((int)s_a[k + 1] - a0) * cnt;
        const uint32_t inv = s_b[ni + 1 + k];
        const int r0 = s_item[k].r0, r1 = s_item[k].r1;
        uint32_t *dst = s_w + ((rev ? nr - r1 : r0) << (5 + lg));
        for (int q = lane; q < (r1 - r0) << (5 + lg); q += 32) {
            uint32_t w = (uint32_t)(nab + lane) * (1u + (1u << kWinIdx));
            if (q < total) {
                const int ai = inv ? (int)__umulhi((uint32_t)q, inv) : q;
                const uint32_t ea = s_a[a0 + ai], eb = s_b[b0 + q - ai * cnt];
                const uint32_t l0 = (ea & M) * nb + (eb & M);
                const uint32_t l1 = ((ea >> kWinIdx) & M) * nb + ((eb >> kWinIdx) & M);
                w = l0 | l1 << kWinIdx | ((ea ^ eb) >> (2 * kWinIdx)) << 31;
            }
            dst[q] = w;
        }
    }
    __syncthreads();  // s_g is read by other threads than wrote it
    qfbg::g_pdl_enter();

    const int s0 = slot0 + ((int)blockIdx.y << lspc);
    V *psi = reinterpret_cast<V *>(L.psi), *sig = reinterpret_cast<V *>(L.sig);
    for (int i = tid; i < (nab + 32) << lspc; i += nth) {
        const int e = i >> lspc, sl = i & (spc - 1);
        const bool in = e < nab && s0 + sl < L.B;
        const size_t g = in ? (size_t)s_g[e] * L.B + s0 + sl : 0;
        WinState<SWEEP, V>(w_raw, sl, stride, lspc)
            .set(e, in ? psi[g] : qfbs::v_zero(V()), SWEEP && in ? sig[g] : qfbs::v_zero(V()));
    }
    for (int i = tid; i < ni << lspc; i += nth) {
        const int s = s0 + (i & (spc - 1));
        const VItem it = s_item[i >> lspc];
        double2 c = s < L.B ? ang[(size_t)it.ang * L.B + s] : make_double2(1.0, 0.0);
        if (!(it.fl & qfbs::R_ROT)) c = make_double2(1.0, 0.0);
        VCoef<SWEEP, V> cf;
        cf.c = c.x;
        cf.pad = 0.0;
        cf.a = v_of(V(), it.hn, sign * c.y);
        cf.b = v_of(V(), it.gn, sign * c.y);
        if constexpr (SWEEP) {
            const double f = (it.fl & qfbs::R_IP) ? it.gamma : 0.0;
            cf.h = v_of(V(), it.hn, f);
            cf.g = v_of(V(), it.gn, f);
        }
        VCoef<SWEEP, V> *dst = s_cf + (i & (spc - 1)) * nr;
        for (int r = it.r0; r < it.r1; ++r) dst[rev ? nr - 1 - r : r] = cf;
    }
    __syncthreads();

    const int sl = warp >> lg, t = tid & (G - 1);
    {
        WinState<SWEEP, V> st(w_raw, sl, stride, lspc);
        const uint32_t *wp = s_w + t;
        const VCoef<SWEEP, V> *cp = s_cf + sl * nr;
        uint32_t word = *wp;
        VCoef<SWEEP, V> cf = *cp;
        qfbs::RSum ip;
        for (int r = 0; r < nr; ++r) {
            const uint32_t sg = word;
            const VCoef<SWEEP, V> co = cf;
            if (r + 1 < nr) {
                wp += G;
                ++cp;
                word = *wp;
                cf = *cp;
            }
            const double x = st.round(sg & M, (sg >> kWinIdx) & M, sg, co);
            if (lg == 0)
                __syncwarp();
            else
                asm volatile("bar.sync %0, %1;" ::"r"(sl + 1), "r"(G) : "memory");
            if constexpr (SWEEP) {
                ip.add(r & 3, x);
                if ((r & 3) == 3 || r + 1 == nr) {
                    const double sum = ip.sum();
                    const int rr = (r & ~3) + (lane >> 2);
                    if ((lane & 3) == 0 && rr <= r) s_sum[warp * nr + rr] = sum;
                    ip = qfbs::RSum();
                }
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < nab << lspc; i += nth) {
        const int e = i >> lspc, q = i & (spc - 1);
        if (s0 + q < L.B) {
            const size_t g = (size_t)s_g[e] * L.B + s0 + q;
            const WinState<SWEEP, V> st(w_raw, q, stride, lspc);
            psi[g] = st.psi(e);
            if (SWEEP) sig[g] = st.sig(e);
        }
    }
    if (SWEEP) {
        for (int i = tid; i < ni << lspc; i += nth) {
            const int k = i >> lspc, q = i & (spc - 1);
            if (s0 + q >= L.B || !(s_item[k].fl & qfbs::R_IP)) continue;
            double x = 0.0;
            for (int j = 0; j < 1 << lg; ++j)
                for (int r = s_item[k].r0; r < s_item[k].r1; ++r)
                    x += s_sum[((q << lg) + j) * nr + (rev ? nr - 1 - r : r)];
            partial[(size_t)s_item[k].poff * L.B + (size_t)(s0 + q) * gridDim.x + blockIdx.x] = x;
        }
    }
}

// grad[s][mu] = 2 x the partials of parameter mu's inner-product items, in
// order: spans [pspan[mu].x, pspan[mu].y) of (offset, blocks).  grid = (M, B).
__global__ void __launch_bounds__(128) k_win_grad(const double *__restrict__ partial,
                                                  const int2 *__restrict__ pspan,
                                                  const longlong2 *__restrict__ span,
                                                  double *__restrict__ grad) {
    const int mu = blockIdx.x, s = blockIdx.y, B = gridDim.y;
    const int2 r = pspan[mu];
    double acc = 0.0;
    for (int i = r.x; i < r.y; ++i) {
        const longlong2 sp = span[i];
        const double *q = partial + (size_t)sp.x * B + (size_t)s * sp.y;
        for (int c = threadIdx.x; c < (int)sp.y; c += blockDim.x) acc += q[c];
    }
    const double2 t = block_sum(make_double2(acc, 0.0));
    if (threadIdx.x == 0) grad[(size_t)s * gridDim.x + mu] = 2.0 * t.x;
}

}  // namespace qfbv
