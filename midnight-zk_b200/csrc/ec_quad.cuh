// ec_quad.cuh — G1 additions and doublings by four lanes together.
#pragma once
#include "ec.cuh"

namespace mzk {

// ---- one point per quad of lanes --------------------------------------------
//
// Where few points are left (partial sums, the upper levels of a bucket
// reduction) an addition by one lane is a chain of 14 dependent products,
// ~0.92 us each on an otherwise idle SM sub-partition (B200, 1.965 GHz): 12.8
// us.  A quad holds one coordinate per lane (X, Y, ZZ, ZZZ in lanes 0..3, 12
// registers) and runs the same formulas four products at a time: 4 levels per
// addition, 3 per doubling, the operands exchanged by shuffles.  16 product
// slots for 14 products, so the throughput stays within 1/8 of the
// one-lane form while the latency falls to a third.  Every lane of the warp
// takes part in every call.
__device__ __forceinline__ Fp fp_shfl4(const Fp& a, int src) {  // lane `src` of the quad
    Fp r;
#pragma unroll
    for (int j = 0; j < 12; j++) r.l[j] = __shfl_sync(0xffffffffu, a.l[j], src, 4);
    return r;
}
__device__ __forceinline__ Fp fp_shfl_xor2(const Fp& a) {
    Fp r;
#pragma unroll
    for (int j = 0; j < 12; j++) r.l[j] = __shfl_xor_sync(0xffffffffu, a.l[j], 2);
    return r;
}

// dbl-2008-s-1 (a = 0); infinity (ZZ = 0) stays infinity
static __device__ __noinline__ Fp quad_dbl(const Fp a) {
    const int q = threadIdx.x & 3;
    const Fp o1 = fp_select(q == 1, fp_dbl(a), a);           // lane 1: U = 2Y
    const Fp m1 = fp_mul(o1, o1);                            // 0: XX, 1: V = U^2
    const Fp v = fp_shfl4(m1, 1);
    const Fp xx = fp_shfl4(m1, 0);
    const Fp m = fp_add(fp_dbl(xx), xx);                     // M = 3 XX
    const Fp m2 = fp_mul(fp_select(q == 3, m, o1), fp_select(q == 3, m, v));  // 0: S, 1: W, 2: ZZ3, 3: M^2
    const Fp s = fp_shfl4(m2, 0), w = fp_shfl4(m2, 1);
    const Fp x3 = fp_sub(fp_shfl4(m2, 3), fp_dbl(s));
    const Fp m3 = fp_mul(fp_select(q == 0, m, w), fp_select(q == 0, fp_sub(s, x3), a));  // 0: M (S - X3), 1: W Y, 3: ZZZ3
    const Fp y3 = fp_sub(fp_shfl4(m3, 0), m3);               // lane 1
    return fp_select(q < 2, fp_select(q == 0, x3, y3), fp_select(q == 2, m2, m3));
}

// add-2008-s with all special cases
static __device__ __noinline__ Fp quad_add(const Fp a, const Fp b) {
    const int q = threadIdx.x & 3;
    const uint32_t base = threadIdx.x & 28;  // the quad's first lane
    const uint32_t az = __ballot_sync(0xffffffffu, fp_is_zero_raw(a)), bz = __ballot_sync(0xffffffffu, fp_is_zero_raw(b));
    const bool a_inf = (az >> (base + 2)) & 1u, b_inf = (bz >> (base + 2)) & 1u;
    // nothing to add in any quad of the warp: empty buckets, which are most of
    // them where scalars are few or small (2^22 points of 8 bits: the reduction
    // 2.98 ms without this line, 0.36 with it)
    if (((az | bz) & 0x44444444u) == 0x44444444u) return fp_select(a_inf, b, a);
    const Fp m1 = fp_mul(a, fp_shfl_xor2(b));                // U1, S1, U2, S2
    const Fp t = fp_shfl_xor2(m1);
    const Fp d = fp_sub(fp_select(q < 2, t, m1), fp_select(q < 2, m1, t));  // lanes 0, 2: P, lanes 1, 3: R
    const uint32_t dz = __ballot_sync(0xffffffffu, fp_is_zero(d)) >> base;
    const Fp m2 = fp_mul(fp_select(q < 2, d, a), fp_select(q < 2, d, b));   // PP, RR, ZZ1 ZZ2, ZZZ1 ZZZ2
    const Fp pp = fp_shfl4(m2, 0), p = fp_shfl4(d, 0);
    const Fp m3 = fp_mul(fp_select(q == 0, m1, fp_select(q == 1, p, m2)), fp_select(q == 3, p, pp));  // Q, PPP, ZZ3, ZZZ1 ZZZ2 P
    const Fp qq = fp_shfl4(m3, 0);
    const Fp x3 = fp_sub(fp_sub(m2, m3), fp_dbl(qq));        // lane 1: RR - PPP - 2Q
    const Fp s1 = fp_shfl4(m1, 1), ppp = fp_shfl4(m3, 1);
    // S1 PPP, R (Q - X3), -, ZZZ3
    const Fp m4 = fp_mul(fp_select(q == 0, s1, fp_select(q == 1, d, m3)),
                         fp_select(q == 0, ppp, fp_select(q == 1, fp_sub(qq, x3), pp)));
    const Fp y3 = fp_sub(m4, fp_shfl4(m4, 0));               // lane 1
    const Fp x3b = fp_shfl4(x3, 1);
    Fp r = fp_select(q < 2, fp_select(q == 0, x3b, y3), fp_select(q == 2, m3, m4));
    const bool equal_x = !a_inf && !b_inf && (dz & 1u);
    if (__any_sync(0xffffffffu, equal_x)) {  // rare: equal or opposite points
        const Fp dbl = quad_dbl(a);
        r = fp_select(equal_x, fp_select((dz & 2u) != 0, dbl, fp_zero()), r);
    }
    return fp_select(a_inf, b, fp_select(b_inf, a, r));
}

// lane q's coordinate of a stored point, 48 bytes at a 16-byte boundary
__device__ __forceinline__ Fp quad_load(const Xyzz* src) {
    const uint4* s = reinterpret_cast<const uint4*>(src) + 3 * (threadIdx.x & 3);
    Fp r;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint4 v = s[k];
        r.l[4 * k] = v.x;
        r.l[4 * k + 1] = v.y;
        r.l[4 * k + 2] = v.z;
        r.l[4 * k + 3] = v.w;
    }
    return r;
}
__device__ __forceinline__ void quad_store(Xyzz* dst, const Fp& a) {
    uint4* d = reinterpret_cast<uint4*>(dst) + 3 * (threadIdx.x & 3);
#pragma unroll
    for (int k = 0; k < 3; k++) d[k] = make_uint4(a.l[4 * k], a.l[4 * k + 1], a.l[4 * k + 2], a.l[4 * k + 3]);
}

}  // namespace mzk
