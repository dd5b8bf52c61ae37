// inv.cuh — modular inversion by division steps, for both fields.
//
// The algorithm of Bernstein and Yang, "Fast constant-time gcd computation and
// modular inversion" (TCHES 2019/3), with the division step that starts at
// delta = 1/2 (Pieter Wuille's variant, described with 30-bit limbs in
// libsecp256k1's "The safegcd implementation in libsecp256k1 explained"): from f = m, g = a, each step replaces (delta, f, g) by
// (1 - delta, g, (g - f)/2) if delta > 0 and g is odd, and by
// (1 + delta, f, (g + (g mod 2) f)/2) otherwise, until g = 0 and f = +-1.
// Thirty steps at a time depend on the low words of f and g only; they give a
// 2 x 2 matrix of 30-bit entries that is then applied to f, g and, modulo m, to
// the coefficients d, e with d a = f and e a = g.  The lanes of a warp run the
// same steps (a step is branch-free, a warp ends when its last lane does), and
// the steps run on the ALU pipe, so a warp inverts 32 values in the time of
// ~40 products: a Fermat power takes ~570, a binary extended Euclid, whose
// lanes diverge, ~300.
#pragma once
#include <cstdint>

#include "field.cuh"

namespace mzk {

// Elements as L signed limbs of 30 bits: limbs below the top in [0, 2^30), the
// top one signed.
template <class P>
struct Limbs30 {
    static constexpr int L = P::N == 12 ? 13 : 9;
    static constexpr uint32_t kMask = 0x3fffffffu;
    // limb i of an N-word constant given by the functor
    template <class W>
    __host__ __device__ static constexpr uint32_t limb(W w, int i) {
        const int bit = 30 * i, k = bit >> 5, s = bit & 31;
        const uint64_t lo = w(k), hi = k + 1 < P::N ? w(k + 1) : 0u;
        return (uint32_t)(((hi << 32 | lo) >> s) & kMask);
    }
    __host__ __device__ static constexpr uint32_t modulus(int i) { return limb([](int k) { return P::mod(k); }, i); }
    __host__ __device__ static constexpr uint32_t r2(int i) { return limb([](int k) { return P::r2(k); }, i); }
    // limb i of k times the modulus, k = 2^log_k, the top limb unmasked
    __host__ __device__ static constexpr int32_t modulus_times(int i, int log_k) {
        const uint32_t below = i > 0 && log_k > 0 ? modulus(i - 1) >> (30 - log_k) : 0u;
        const uint32_t v = (modulus(i) << log_k) | below;
        return (int32_t)(i + 1 < L ? v & kMask : v);
    }
    // modulus^-1 mod 2^30, from P::N0 = -modulus^-1 mod 2^32
    static constexpr uint32_t kInv = (0u - P::N0) & kMask;
};

__device__ __forceinline__ int64_t mad_s64(int32_t a, int32_t b, int64_t c) { return (int64_t)a * b + c; }

// Thirty division steps on the low words of f and g: the matrix
// (u v; q r) with 2^30 f' = u f + v g and 2^30 g' = q f + r g, absolute row
// sums at most 2^30.  theta = delta - 1/2.  Entries of 15 steps fit 16 bits, so
// a row is one word (first entry + second entry 2^16, added as a whole), and
// the two halves are multiplied together.
__device__ __forceinline__ void divsteps30(int32_t& theta, uint32_t f, uint32_t g, int32_t (&t)[4]) {
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
        uint32_t u = 1, q = 1u << 16;
#pragma unroll
        for (int i = 0; i < 15; i++) {
            const uint32_t odd = 0u - (g & 1u);
            const uint32_t sw = odd & ~(uint32_t)(theta >> 31);  // delta > 0 and g odd
            g = g + ((f & odd) ^ sw) - sw;
            q = q + ((u & odd) ^ sw) - sw;
            f += g & sw;
            u += q & sw;
            g >>= 1;
            u <<= 1;
            theta = (int32_t)((uint32_t)theta ^ sw) + 1;
        }
        // entries lie in (-2^15, 2^15]; the upper end occurs (15 steps without
        // an exchange leave u = 2^15, or v = 2^15 after one at the first)
        const int32_t u0 = (int16_t)(u - 1u) + 1, q0 = (int16_t)(q - 1u) + 1;
        const int32_t v0 = ((int32_t)(u - (uint32_t)u0 - 0x10000u) >> 16) + 1;
        const int32_t r0 = ((int32_t)(q - (uint32_t)q0 - 0x10000u) >> 16) + 1;
        if (half == 0) {
            t[0] = u0;
            t[1] = v0;
            t[2] = q0;
            t[3] = r0;
        } else {
            const int32_t a = t[0], b = t[1], c = t[2], d = t[3];
            t[0] = u0 * a + v0 * c;
            t[1] = u0 * b + v0 * d;
            t[2] = q0 * a + r0 * c;
            t[3] = q0 * b + r0 * d;
        }
    }
}

// out = a^-1 R^2 mod m (R = 2^(32 N)): the Montgomery form of 1/x for a = x R.
// a below 2^(32 N - 1), canonical or not; returns false (out undefined) when a
// is not invertible, that is a = 0 mod m.
template <class P>
static __device__ __noinline__ bool inv_divsteps(uint32_t* out, const uint32_t* a) {
    using S = Limbs30<P>;
    constexpr int L = S::L, N = P::N;
    int32_t f[L], g[L], d[L], e[L];
#pragma unroll
    for (int i = 0; i < L; i++) {
        const int k = (30 * i) >> 5, s = (30 * i) & 31;
        const uint32_t w = k + 1 < N ? __funnelshift_r(a[k], a[k + 1], s) : a[k] >> s;
        f[i] = (int32_t)S::modulus(i);
        g[i] = (int32_t)(w & S::kMask);
        d[i] = 0;
        e[i] = (int32_t)S::r2(i);
    }
    int32_t theta = 0;
    // 27 rounds end every 381-bit input tried and 18 every 255-bit one; the
    // bound only keeps the loop finite
    for (int it = 0; it < 40; it++) {
        int32_t t[4];
        divsteps30(theta, (uint32_t)f[0] | ((uint32_t)f[1] << 30), (uint32_t)g[0] | ((uint32_t)g[1] << 30), t);
        // f, g: exact division by 2^30
        int64_t cf = mad_s64(t[1], g[0], (int64_t)t[0] * f[0]) >> 30;
        int64_t cg = mad_s64(t[3], g[0], (int64_t)t[2] * f[0]) >> 30;
#pragma unroll
        for (int i = 1; i < L; i++) {
            cf = mad_s64(t[1], g[i], mad_s64(t[0], f[i], cf));
            cg = mad_s64(t[3], g[i], mad_s64(t[2], f[i], cg));
            f[i - 1] = (int32_t)((uint32_t)cf & S::kMask);
            g[i - 1] = (int32_t)((uint32_t)cg & S::kMask);
            cf >>= 30;
            cg >>= 30;
        }
        f[L - 1] = (int32_t)cf;
        g[L - 1] = (int32_t)cg;
        // d, e: the same modulo m; the multiple of m, at most m / 2 after the
        // division, keeps |d|, |e| below (it / 2 + 1) m
        int64_t cd = mad_s64(t[1], e[0], (int64_t)t[0] * d[0]);
        int64_t ce = mad_s64(t[3], e[0], (int64_t)t[2] * d[0]);
        const int32_t md = (int32_t)((0u - (uint32_t)cd * S::kInv) << 2) >> 2;
        const int32_t me = (int32_t)((0u - (uint32_t)ce * S::kInv) << 2) >> 2;
        cd = mad_s64(md, (int32_t)S::modulus(0), cd) >> 30;
        ce = mad_s64(me, (int32_t)S::modulus(0), ce) >> 30;
#pragma unroll
        for (int i = 1; i < L; i++) {
            cd = mad_s64(md, (int32_t)S::modulus(i), mad_s64(t[1], e[i], mad_s64(t[0], d[i], cd)));
            ce = mad_s64(me, (int32_t)S::modulus(i), mad_s64(t[3], e[i], mad_s64(t[2], d[i], ce)));
            d[i - 1] = (int32_t)((uint32_t)cd & S::kMask);
            e[i - 1] = (int32_t)((uint32_t)ce & S::kMask);
            cd >>= 30;
            ce >>= 30;
        }
        d[L - 1] = (int32_t)cd;
        e[L - 1] = (int32_t)ce;
        int32_t nz = 0;
#pragma unroll
        for (int i = 0; i < L; i++) nz |= g[i];
        if (nz == 0) break;
    }
    // f = 1 or -1 (limbs 2^30 - 1 .., top -1), d its coefficient
    const int32_t neg = f[L - 1] >> 31;
    int32_t diff = (f[0] ^ (neg ? (int32_t)S::kMask : 1)) | (f[L - 1] ^ neg);
#pragma unroll
    for (int i = 1; i < L - 1; i++) diff |= f[i] ^ (neg & (int32_t)S::kMask);
    int32_t c = 0;
#pragma unroll
    for (int i = 0; i < L; i++) {  // d = neg ? -d : d
        c += (d[i] ^ neg) - neg;
        d[i] = i + 1 < L ? (int32_t)((uint32_t)c & S::kMask) : c;
        c >>= 30;
    }
    // |d| < 21 m: into [0, 32 m), then down by halves
    c = 0;
    const int32_t below = d[L - 1] >> 31;
#pragma unroll
    for (int i = 0; i < L; i++) {
        c += d[i] + (S::modulus_times(i, 5) & below);
        d[i] = i + 1 < L ? (int32_t)((uint32_t)c & S::kMask) : c;
        c >>= 30;
    }
#pragma unroll
    for (int k = 4; k >= 0; k--) {
        int32_t s[L];
        c = 0;
#pragma unroll
        for (int i = 0; i < L; i++) {
            c += d[i] - S::modulus_times(i, k);
            s[i] = i + 1 < L ? (int32_t)((uint32_t)c & S::kMask) : c;
            c >>= 30;
        }
        const bool keep = s[L - 1] < 0;
#pragma unroll
        for (int i = 0; i < L; i++) d[i] = keep ? d[i] : s[i];
    }
#pragma unroll
    for (int k = 0; k < N; k++) out[k] = ((uint32_t)d[k] >> (2 * k)) | ((uint32_t)d[k + 1] << (30 - 2 * k));
    return diff == 0;
}

// 1/a (Montgomery), canonical; zero gives zero
// (by value: the caller's variable keeps its registers)
__device__ __forceinline__ Fp fp_invert(const Fp a) {
    Fp r;
    return inv_divsteps<FpP>(r.l, a.l) ? r : fp_zero();
}
__device__ __forceinline__ Fr fr_invert(const Fr a) {
    Fr r;
    return inv_divsteps<FrP>(r.l, a.l) ? r : fr_zero();
}

}  // namespace mzk
