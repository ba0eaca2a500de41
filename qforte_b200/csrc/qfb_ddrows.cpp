// Products of gate matrices in double-double: error-free products by fused
// multiply-add and error-free sums (Dekker 1971, Knuth's two-sum), four columns a
// register.  The entries of m are doubles, so a term costs a product, its error, the
// low part's product and one sum with its error; a zero entry costs nothing (real
// and purely imaginary gates, diagonals).
//
// The rounding of a product repeats wherever its layer does and adds up over all
// amplitudes alike, so the products of the fused tile form are rounded once.  Rx layers
// with cX-Rz-cX couplings, 10 layers on 15 qubits, mean error of 10 draws against long
// double: products rounded gate by gate 2.73e-15, rounded once 1.05e-15, gate by gate on
// the state 1.03e-15.  The whole call, 20 random layers (planning included), us, doubles /
// long double / this: 20 qubits 801 / 1,125 / 826, 21 qubits 931 / 1,263 / 967, 23 qubits
// 2,707 / 2,811 / 2,726.
#include "qfb_ddrows.h"

#if defined(__x86_64__)
#include <immintrin.h>

namespace qfbh {

#define QFB_AVX2 __attribute__((target("avx2,fma")))
#define QFB_AVX2_INLINE __attribute__((target("avx2,fma"), always_inline)) inline

struct Acc {
    __m256d h, l;
    bool any;
};

// a += f (xh + xl)
QFB_AVX2_INLINE static void term(Acc &a, double f, __m256d xh, __m256d xl) {
    if (f == 0.0) return;
    const __m256d v = _mm256_set1_pd(f);
    __m256d p = _mm256_mul_pd(v, xh);
    asm("" : "+x"(p));  // (the product as rounded: not to be fused into the sum below)
    const __m256d e = _mm256_fmadd_pd(v, xl, _mm256_fmsub_pd(v, xh, p));
    if (!a.any) {
        a = Acc{p, e, true};
        return;
    }
    const __m256d s = _mm256_add_pd(a.h, p), b = _mm256_sub_pd(s, a.h);
    const __m256d d = _mm256_add_pd(_mm256_sub_pd(a.h, _mm256_sub_pd(s, b)), _mm256_sub_pd(p, b));
    a.h = s;
    a.l = _mm256_add_pd(a.l, _mm256_add_pd(d, e));
}

QFB_AVX2_INLINE static void put(const Acc &a, double *h, double *l) {
    // (terms that cancel can leave the larger part in l)
    const __m256d s = _mm256_add_pd(a.h, a.l), b = _mm256_sub_pd(s, a.h);
    _mm256_store_pd(h, s);
    _mm256_store_pd(l, _mm256_add_pd(_mm256_sub_pd(a.h, _mm256_sub_pd(s, b)), _mm256_sub_pd(a.l, b)));
}

template <int N>
QFB_AVX2 static void mix(Rows8 &r, const int *k, const double *m, unsigned halves) {
    for (int c = 0; c < 8; c += 4) {
        if (!(halves >> (c / 4) & 1u)) continue;
        __m256d xh[N], xl[N], yh[N], yl[N];
        for (int j = 0; j < N; ++j) {
            xh[j] = _mm256_load_pd(&r.xh[k[j]][c]);
            xl[j] = _mm256_load_pd(&r.xl[k[j]][c]);
            yh[j] = _mm256_load_pd(&r.yh[k[j]][c]);
            yl[j] = _mm256_load_pd(&r.yl[k[j]][c]);
        }
        for (int i = 0; i < N; ++i) {
            const __m256d z = _mm256_setzero_pd();
            Acc re{z, z, false}, im{z, z, false};
            for (int j = 0; j < N; ++j) {
                const double fx = m[2 * (N * i + j)], fy = m[2 * (N * i + j) + 1];
                term(re, fx, xh[j], xl[j]);
                term(re, -fy, yh[j], yl[j]);
                term(im, fx, yh[j], yl[j]);
                term(im, fy, xh[j], xl[j]);
            }
            put(re, &r.xh[k[i]][c], &r.xl[k[i]][c]);
            put(im, &r.yh[k[i]][c], &r.yl[k[i]][c]);
        }
    }
}

bool dd_available() {
    static const bool ok = __builtin_cpu_supports("avx2") && __builtin_cpu_supports("fma");
    return ok;
}

void dd_mix(Rows8 &r, const int *k, int n, const double *m, unsigned halves) {
    if (n == 1)
        mix<1>(r, k, m, halves);
    else if (n == 2)
        mix<2>(r, k, m, halves);
    else
        mix<4>(r, k, m, halves);
}

}  // namespace qfbh

#else  // other hosts: the products in long double

namespace qfbh {
bool dd_available() { return false; }
void dd_mix(Rows8 &, const int *, int, const double *, unsigned) {}
}  // namespace qfbh

#endif
