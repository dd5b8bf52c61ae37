// msm.cu — Pippenger multi-scalar multiplication over BLS12-381 G1.
//
// Replaces curves::msm::msm_best (curves/src/msm.rs:460-532) and the
// blst Pippenger behind G1Affine::multi_exp_affine (g1.rs:427-446) that
// proofs::poly::kzg::msm::msm_specific (kzg/msm.rs:174-201) dispatches to.
// The result is the same group element; the schedule is built for the GPU:
//
//  1. histogram   one thread per scalar: Montgomery -> canonical (one Fr
//                 multiplication by 1, the reference's `to_repr`), signed
//                 c-bit window digits d_w in [-2^(c-1), 2^(c-1)], count of
//                 entries per key (window, |d|-1) with warp-aggregated atomics;
//                 the digits are also stored, window-major.
//  2. scan        exclusive prefix sum of the counts = start of every bucket
//                 in the sorted entry array (a counting sort).
//  3. scatter     one window at a time from the stored digits: each
//                 (point index | sign) goes to its bucket's slice; a window's
//                 slices (4n bytes) stay in L2 while it is scattered, so the
//                 random 4-byte writes leave L2 as whole sectors.  Zero digits
//                 produce no entry, so zero and sparse scalars cost nothing
//                 (msm_specific drops zero scalars).
//  4. pair sums   for large inputs, up to three rounds that replace the points of
//                 every bucket by the affine sums of neighbours, hundreds of
//                 sums to one inversion (k_pair_sums).
//  5. accumulate  the entries that are left split into equal chunks, one per thread:
//                 every thread walks its chunk adding points into an XYZZ
//                 accumulator (mixed addition, affine bases gathered from HBM).
//                 Buckets entirely inside a chunk are written directly; a bucket
//                 cut by a chunk edge leaves partial sums.  Equal chunks keep
//                 every thread busy whatever the scalar distribution.
//  6. fixup       the chunk where a cut bucket starts sums its partials.
//  7. reduce      per window, sum_b (b+1) B_b by a tree over its buckets whose
//                 nodes carry their sum and the sums over every bit plane of
//                 the index, four lanes per addition; where buckets fill the
//                 GPU, running sums over groups of buckets come first.
//  8. finish      one block per window shifts the planes and adds them up.
//  9. host        sum_w 2^(c w) S_w (c doublings between windows) and the
//                 affine normalisation on the host: a few hundred group
//                 operations that one GPU thread would take ~1 ms for.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "ec.cuh"
#include "ec_quad.cuh"
#include "host_ec.hpp"
#include "runtime.hpp"

namespace mzk {

namespace {

constexpr int kAccThreads = 128;   // threads per block of the accumulate kernel
constexpr int kReduceThreads = 128;
constexpr uint32_t kNoKey = 0xffffffffu;

struct MsmShape {
    int c;          // window width in bits
    int windows;    // number of windows
    uint32_t nb;    // buckets per window = 2^(c-1)
    uint32_t keys;  // windows * nb
};

MsmShape make_shape(int c) {
    MsmShape s;
    s.c = c;
    s.windows = (256 + c - 1) / c;
    s.nb = 1u << (c - 1);
    s.keys = s.nb * (uint32_t)s.windows;
    return s;
}

__device__ __forceinline__ uint32_t fr_limb(const Fr& s, int i) {
    uint32_t v = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) v = (i == j) ? s.l[j] : v;
    return v;
}

// bits [bit, bit + c) of the canonical scalar, c <= 31
__device__ __forceinline__ uint32_t window_bits(const Fr& s, int bit, int c) {
    const int limb = bit >> 5, sh = bit & 31;
    uint64_t v = (uint64_t)fr_limb(s, limb) | ((uint64_t)fr_limb(s, limb + 1) << 32);
    return (uint32_t)(v >> sh) & ((1u << c) - 1u);
}

__device__ __forceinline__ Fr load_fr(const Fr* p, size_t i) {
    const uint4* src = reinterpret_cast<const uint4*>(p + i);
    uint4 a = __ldg(src), b = __ldg(src + 1);
    Fr r;
    r.l[0] = a.x; r.l[1] = a.y; r.l[2] = a.z; r.l[3] = a.w;
    r.l[4] = b.x; r.l[5] = b.y; r.l[6] = b.z; r.l[7] = b.w;
    return r;
}

// Signed digit recoding: returns key (window * nb + |d| - 1) or kNoKey for a
// zero digit, and the sign; carries between windows through `carry`.
__device__ __forceinline__ uint32_t next_digit(const Fr& s, int w, int c, uint32_t nb, uint32_t& carry, bool& neg) {
    uint32_t v = window_bits(s, w * c, c) + carry;
    uint32_t mag;
    if (v > nb) {  // v - 2^c is negative
        mag = (1u << c) - v;
        carry = 1;
        neg = true;
    } else {
        mag = v;
        carry = 0;
        neg = false;
    }
    return mag == 0 ? kNoKey : (uint32_t)w * nb + (mag - 1);
}

// digits (optional): every point's signed digit per window, window-major
// (digits[w * n + i] = key | sign << 31, kNoKey for a zero digit), for the
// window-by-window scatter
__global__ void k_histogram(const Fr* __restrict__ scalars, size_t n, int c, int windows, uint32_t nb,
                            uint32_t* __restrict__ counts, uint32_t* __restrict__ digits) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < n; base += stride) {
        const size_t i = base + threadIdx.x;
        const bool valid = i < n;
        Fr s = valid ? fr_from_mont(load_fr(scalars, i)) : fr_zero();
        uint32_t carry = 0;
        for (int w = 0; w < windows; w++) {
            bool neg;
            uint32_t key = next_digit(s, w, c, nb, carry, neg);
            if (!valid) key = kNoKey;
            if (digits && valid) digits[(size_t)w * n + i] = key == kNoKey ? kNoKey : key | (neg ? 0x80000000u : 0u);
            const uint32_t peers = __match_any_sync(0xffffffffu, key);
            if (key != kNoKey && lane == __ffs(peers) - 1) atomicAdd(&counts[key], (uint32_t)__popc(peers));
        }
    }
}

// All-windows scatter of the fixed-scratch path (n <= 2^16, whose sorted
// array fits in L2): windows whose cursor atomics a warp keeps in flight.
constexpr int kScatterWindows = 8;

// The cursor of bucket `key` is cursor[key] (= offsets + 1 of the caller):
// it starts at the bucket's first slot (the exclusive scan written one place
// to the right) and each atomic returns absolute positions.  After the
// scatter cursor[key] = end of bucket key = start of bucket key + 1, so the
// array from offsets[0] = 0 is exactly the bucket offset table.
__device__ __forceinline__ void scatter_group(const uint32_t (&key)[kScatterWindows],
                                              const bool (&neg)[kScatterWindows], uint32_t value, int lane,
                                              uint32_t* __restrict__ cursor, uint32_t* __restrict__ sorted) {
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t peers[kScatterWindows], slot[kScatterWindows];
#pragma unroll
    for (int j = 0; j < kScatterWindows; j++) {
        peers[j] = __match_any_sync(0xffffffffu, key[j]);
        slot[j] = 0;
        if (key[j] != kNoKey && lane == __ffs(peers[j]) - 1) slot[j] = atomicAdd(&cursor[key[j]], (uint32_t)__popc(peers[j]));
    }
#pragma unroll
    for (int j = 0; j < kScatterWindows; j++) {
        const uint32_t first = __shfl_sync(0xffffffffu, slot[j], __ffs(peers[j]) - 1);
        if (key[j] != kNoKey) sorted[first + (uint32_t)__popc(peers[j] & lt_mask)] = value | (neg[j] ? 0x80000000u : 0u);
    }
}

// The scatter of one window from the stored digits.  Its entries go to that
// window's slice of the sorted array (4n bytes: 67 MB at 2^24, inside the
// 126 MB L2), so the scattered 4-byte writes merge into whole sectors in L2
// instead of each costing a DRAM sector read and write.
__global__ void k_scatter_window(const uint32_t* __restrict__ digits, size_t n, uint32_t w0,
                                 uint32_t* __restrict__ cursor, uint32_t* __restrict__ sorted) {
    const uint32_t* __restrict__ digits_w = digits + (size_t)(w0 + blockIdx.y) * n;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < n; base += stride) {
        const size_t i = base + threadIdx.x;
        const uint32_t d = i < n ? __ldg(digits_w + i) : kNoKey;
        const uint32_t key = d == kNoKey ? kNoKey : d & 0x7fffffffu;
        const uint32_t peers = __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(peers) - 1;
        uint32_t slot = 0;
        if (key != kNoKey && lane == leader) slot = atomicAdd(&cursor[key], (uint32_t)__popc(peers));
        slot = __shfl_sync(0xffffffffu, slot, leader);
        if (key != kNoKey) sorted[slot + (uint32_t)__popc(peers & lt_mask)] = (uint32_t)i | (d & 0x80000000u);
    }
}

// Windows scattered by one launch of k_scatter_window(_batch): as many as keep
// their entries (4 bytes each) within a quarter of L2.  A launch per window
// costs 3.5 us whatever its size: 1000 points (32 windows) 744 -> 620 us per
// call, a proof of 2^14 rows 7.30 -> 6.75 ms.  At 10^6 points one launch of 8
// windows or 16 measures the same (7.37 ms, 7.45 window by window).
constexpr size_t kScatterBytes = 32u << 20;

uint32_t scatter_together(size_t windows, size_t points) {
    return (uint32_t)std::min(windows, std::max<size_t>(1, kScatterBytes / (points * 4)));
}

__global__ void k_scatter(const Fr* __restrict__ scalars, size_t n, int c, int windows, uint32_t nb,
                          uint32_t* __restrict__ cursor, uint32_t* __restrict__ sorted) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < n; base += stride) {
        const size_t i = base + threadIdx.x;
        const bool valid = i < n;
        Fr s = valid ? fr_from_mont(load_fr(scalars, i)) : fr_zero();
        uint32_t carry = 0;
        for (int w0 = 0; w0 < windows; w0 += kScatterWindows) {
            uint32_t key[kScatterWindows];
            bool neg[kScatterWindows];
#pragma unroll
            for (int j = 0; j < kScatterWindows; j++) {
                key[j] = kNoKey;
                neg[j] = false;
                if (w0 + j < windows) {
                    key[j] = next_digit(s, w0 + j, c, nb, carry, neg[j]);
                    if (!valid) key[j] = kNoKey;
                }
            }
            scatter_group(key, neg, (uint32_t)i, lane, cursor, sorted);
        }
    }
}

// ---- exclusive scan of u32 (3 phases) ----
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* smem_warp, uint32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (int)(blockDim.x >> 5) ? smem_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        smem_warp[lane] = w;
    }
    __syncthreads();
    total = smem_warp[(blockDim.x >> 5) - 1];
    uint32_t prefix = warp > 0 ? smem_warp[warp - 1] : 0;
    __syncthreads();
    return prefix + x - v;
}

// kHalves: `in` is an offset table of len - 1 buckets and the scanned values
// are the buckets' sizes after one round of pair sums (half, rounded up), then 0
template <bool kHalves>
__global__ void k_scan_tiles(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t len,
                             uint32_t* __restrict__ tile_sums) {
    __shared__ uint32_t sw[32];
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems], sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (kHalves) v[k] = base + k + 1 < len ? (in[base + k + 1] - in[base + k] + 1) >> 1 : 0;
        else v[k] = base + k < len ? in[base + k] : 0;
        sum += v[k];
    }
    uint32_t total;
    uint32_t pre = block_exclusive_scan(sum, sw, total);
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < len) out[base + k] = pre;
        pre += v[k];
    }
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void k_scan_sums(uint32_t* __restrict__ tile_sums, uint32_t tiles) {
    __shared__ uint32_t sw[32];
    uint32_t carry = 0;
    for (uint32_t b = 0; b < tiles; b += blockDim.x) {
        const uint32_t i = b + threadIdx.x;
        uint32_t v = i < tiles ? tile_sums[i] : 0, total;
        uint32_t pre = block_exclusive_scan(v, sw, total);
        if (i < tiles) tile_sums[i] = pre + carry;
        carry += total;
    }
}

__global__ void k_scan_add(uint32_t* __restrict__ out, uint32_t len, const uint32_t* __restrict__ tile_sums) {
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    const uint32_t add = tile_sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
        if (base + k < len) out[base + k] += add;
}

// ---- bucket accumulation ----
__device__ __forceinline__ uint32_t find_key(const uint32_t* offsets, uint32_t keys, uint32_t pos) {
    // largest k in [0, keys) with offsets[k] <= pos (offsets[keys] = total > pos)
    uint32_t lo = 0, hi = keys;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (offsets[mid] <= pos) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The walk over a chunk's buckets takes empty ones one at a time up to kWalk,
// then by seek_key: where scalars are few or small, 2^17 empty buckets may lie
// between two windows, and one load after another takes 4 ms (2^22 points with
// one scalar: 99 ms of pair sums and accumulation, three rounds each with its
// own walk, against 33 without pair sums; 17 ms now).
constexpr int kWalk = 4;

// the bucket of entry `pos`, which is at or after bucket k: steps that double, then halve
__device__ __forceinline__ uint32_t seek_key(const uint32_t* offsets, uint32_t keys, uint32_t k, uint32_t pos) {
    uint32_t step = 1;
    while (k + step < keys && offsets[k + step] <= pos) {
        k += step;
        step <<= 1;
    }
    uint32_t hi = min(k + step, keys);
    while (hi - k > 1) {
        const uint32_t mid = k + (hi - k) / 2;
        if (offsets[mid] <= pos) k = mid;
        else hi = mid;
    }
    return k;
}

__device__ __forceinline__ void store_xyzz(Xyzz* dst, const Xyzz& v) {
    uint4* d = reinterpret_cast<uint4*>(dst);
    const uint32_t* s = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
    for (int k = 0; k < 12; k++) d[k] = make_uint4(s[4 * k], s[4 * k + 1], s[4 * k + 2], s[4 * k + 3]);
}
__device__ __forceinline__ Xyzz load_xyzz(const Xyzz* src) {
    Xyzz v;
    const uint4* s = reinterpret_cast<const uint4*>(src);
    uint32_t* d = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
    for (int k = 0; k < 12; k++) {
        uint4 q = s[k];
        d[4 * k] = q.x;
        d[4 * k + 1] = q.y;
        d[4 * k + 2] = q.z;
        d[4 * k + 3] = q.w;
    }
    return v;
}

__device__ __forceinline__ void chunk_range(uint32_t total, uint32_t t, uint32_t nthreads, uint32_t& s, uint32_t& e) {
    const uint32_t len = (total + nthreads - 1) / nthreads;
    s = min(total, t * len);
    e = min(total, s + len);
}

// The chunks that a cut bucket starts in, queued for k_fixup
struct Owners {
    uint32_t* count;
    uint2* list;  // (chunk, bucket key)
};

__device__ __forceinline__ void flush_bucket(const Xyzz& acc, uint32_t k, uint32_t seg_lo, uint32_t seg_hi, uint32_t s,
                                             uint32_t e, uint32_t t, Xyzz* buckets, Xyzz* partials, const Owners& own) {
    if (seg_lo >= s && seg_hi <= e) {
        store_xyzz(&buckets[k], acc);
    } else if (seg_lo < s) {
        store_xyzz(&partials[2 * (size_t)t], acc);
    } else {
        store_xyzz(&partials[2 * (size_t)t + 1], acc);
        own.list[atomicAdd(own.count, 1u)] = make_uint2(t, k);
    }
}

// One flat loop over the chunk, so every thread of a warp runs the same number
// of additions whatever its bucket boundaries; a boundary only costs a short
// divergent flush.  kGather: entry j is the point sorted[j] (index | sign);
// otherwise point j of `bases` itself (the pair sums of k_pair_sums).
template <bool kGather>
__global__ void __launch_bounds__(kAccThreads, 1) k_accumulate(const Affine* __restrict__ bases,
                                                            const uint32_t* __restrict__ sorted,
                                                            const uint32_t* __restrict__ offsets, uint32_t keys,
                                                            Xyzz* __restrict__ buckets, Xyzz* __restrict__ partials,
                                                            const Owners own) {
    const uint32_t nthreads = gridDim.x * blockDim.x;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t total = offsets[keys];
    uint32_t s, e;
    chunk_range(total, t, nthreads, s, e);
    if (s >= e) return;
    uint32_t k = find_key(offsets, keys, s);
    uint32_t seg_lo = offsets[k], seg_hi = offsets[k + 1];
    // the end of the following bucket, loaded one bucket ahead (offsets has
    // keys + 2 entries, so k + 2 <= keys + 1 is in range)
    uint32_t nxt_hi = __ldg(offsets + k + 2);
    Xyzz acc;
    xyzz_set_inf(acc);
    // the next entry's base is loaded one iteration ahead, and the entry after
    // it (its index) two ahead, to hide the gather latency
    uint32_t ent = kGather ? __ldg(sorted + s) : s;
    uint32_t ent2 = s + 1 < e ? (kGather ? __ldg(sorted + s + 1) : s + 1) : 0u;
    Affine nxt = load_affine(bases, kGather ? ent & 0x7fffffffu : ent);
    for (uint32_t j = s; j < e; j++) {
        if (j == seg_hi) {
            flush_bucket(acc, k, seg_lo, seg_hi, s, e, t, buckets, partials, own);
            xyzz_set_inf(acc);
            k++;
            seg_lo = seg_hi;
            seg_hi = nxt_hi;
            for (int i = 0; seg_hi <= j; i++) {  // empty buckets
                k = i < kWalk ? k + 1 : seek_key(offsets, keys, k, j);
                seg_hi = offsets[k + 1];
            }
            nxt_hi = __ldg(offsets + k + 2);
        }
        Affine p = nxt;
        const uint32_t cur = ent;
        if (j + 1 < e) {
            ent = ent2;
            nxt = load_affine(bases, kGather ? ent & 0x7fffffffu : ent);
            if (j + 2 < e) ent2 = kGather ? __ldg(sorted + j + 2) : j + 2;
        }
        if (aff_is_inf(p)) continue;
        if (kGather) p.y = fp_select((cur >> 31) != 0, fp_neg(p.y), p.y);
        if (xyzz_is_inf(acc)) {
            acc.x = p.x;
            acc.y = p.y;
            acc.zz = fp_one();
            acc.zzz = fp_one();
        } else {
            xyzz_add_affine_fast(acc, p);
        }
    }
    flush_bucket(acc, k, seg_lo, seg_hi, s, e, t, buckets, partials, own);
}

// ---- pair sums ----
//
// One round replaces the points of every bucket by the sums of neighbours, in
// affine coordinates, so that half as many are left for k_accumulate.  An
// affine addition takes 5 products, a square and an inversion; each thread
// shares one inversion among its B additions by Montgomery's trick (3 of the
// products).  With ~40 products' worth of time for the inversion
// (inv_divsteps) an addition costs ~7 products against the 10 of a mixed XYZZ
// addition, at the price of writing the sums (96 bytes each) and reading them
// again.  The multiply pipe is ~75 % busy (88 % in k_accumulate): the rest are
// waits for loads that one sum's lead does not cover and, with two warps per
// scheduler, the latency of the products themselves.  A third
// warp spills (168 registers) and is slower; the x coordinates two sums ahead
// are 1 % slower.  Per call with 64 / 96 / 128 / 256 sums per inversion: 1000003
// points 6.61 / 6.62 / 6.32 / 6.17 ms, 2^24 points 87.1 / 85.7 / 84.0 / 82.0, eight
// proofs of 2^16 rows 55.4 / 54.2 / 53.8 / 52.5 (7.34, 92.0 and 58.9 ms without
// pair sums).
//
// A thread takes a run of consecutive sums: forward it multiplies up the
// denominators and keeps the partial products, then inverts, then backward it
// forms the sums.  A bucket's odd last point is copied.
__device__ __forceinline__ Fp load_fp(const Fp* p) {
    const uint4* s = reinterpret_cast<const uint4*>(p);
    Fp r;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint4 v = __ldg(s + k);
        r.l[4 * k] = v.x;
        r.l[4 * k + 1] = v.y;
        r.l[4 * k + 2] = v.z;
        r.l[4 * k + 3] = v.w;
    }
    return r;
}
__device__ __forceinline__ void store_affine(Affine* dst, const Affine& a) {
    uint4* d = reinterpret_cast<uint4*>(dst);
    const uint32_t* s = reinterpret_cast<const uint32_t*>(&a);
#pragma unroll
    for (int k = 0; k < 6; k++) d[k] = make_uint4(s[4 * k], s[4 * k + 1], s[4 * k + 2], s[4 * k + 3]);
}

// The cases of a + b whose sum is not the chord's: what to do, the denominator
// that enters the shared inversion and the slope's numerator.  By value, so
// that the loop's points stay in registers.
enum PairKind : int { kPairAdd, kPairFirst, kPairSecond, kPairDouble, kPairInfinity };
struct PairCase {
    Fp den, num;
    int kind;
};
static __device__ __noinline__ PairCase pair_case(const Affine a, const Affine b) {
    PairCase c;
    c.den = fp_sub(b.x, a.x);
    c.num = fp_sub(b.y, a.y);
    if (aff_is_inf(a)) {
        c.kind = kPairSecond;
    } else if (aff_is_inf(b)) {
        c.kind = kPairFirst;
    } else if (!fp_is_zero(c.den)) {
        c.kind = kPairAdd;
    } else if (!fp_is_zero(c.num) || fp_is_zero(a.y)) {  // b = -a
        c.kind = kPairInfinity;
    } else {
        const Fp xx = fp_mul(a.x, a.x);
        c.kind = kPairDouble;
        c.num = fp_add(fp_dbl(xx), xx);
        c.den = fp_dbl(a.y);  // not zero: a zero here would spoil the sums of the whole batch
    }
    return c;
}

constexpr int kPairThreads = 128;
// Whether a + b may not be the chord's (d = x_b - x_a zero, a point at
// infinity): by the first words, wrong in 2^30 for sums that are, which
// pair_case then sorts out.
__device__ __forceinline__ bool maybe_special(const Fp& d, const Fp& xa, const Fp& xb) {
    return d.l[0] == 0u || d.l[0] == FpP::mod(0) || xa.l[0] == 0u || xb.l[0] == 0u;
}

constexpr int kPairBatch = 256;  // sums that share an inversion

// What a thread keeps of its batch, element i of thread t at i * threads + t
// (a partial product in three planes of 16 bytes), so that a warp's accesses
// are contiguous: 56 bytes per sum, 543 MB for 37888 threads.
struct PairScratch {
    uint4* prefix;
    uint32_t *ent1, *ent2;
};
constexpr size_t pair_scratch_bytes(size_t threads) { return threads * kPairBatch * (sizeof(Fp) + 2 * sizeof(uint32_t)); }
PairScratch pair_scratch_at(void* p, size_t threads) {
    uint4* prefix = static_cast<uint4*>(p);
    uint32_t* ent = reinterpret_cast<uint32_t*>(prefix + 3 * threads * kPairBatch);
    return {prefix, ent, ent + threads * kPairBatch};
}

// Sum j of bucket k: points off_in[k] + 2 (j - off_out[k]) and the next, if
// that is below off_in[k + 1].  kGather: point i is src[sorted[i]] with the
// entry's sign, otherwise src[i].
template <bool kGather>
__global__ void __launch_bounds__(kPairThreads, 2) k_pair_sums(const Affine* __restrict__ src,
                                                               const uint32_t* __restrict__ sorted,
                                                               const uint32_t* __restrict__ off_in,
                                                               const uint32_t* __restrict__ off_out, uint32_t keys,
                                                               Affine* __restrict__ out, const PairScratch scratch) {
    constexpr uint32_t B = kPairBatch;
    const uint32_t threads = gridDim.x * blockDim.x;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t s, e;
    chunk_range(off_out[keys], t, threads, s, e);
    if (s >= e) return;
    // the point of an entry: index | sign << 31 when gathering, else the index
    auto point = [&](uint32_t ent) { return load_affine(src, kGather ? ent & 0x7fffffffu : ent); };
    auto signed_point = [&](Affine a, uint32_t ent) {
        if (kGather) a.y = fp_select((ent >> 31) != 0, fp_neg(a.y), a.y);
        return a;
    };
    auto point_x = [&](uint32_t ent) { return load_fp(&src[kGather ? ent & 0x7fffffffu : ent].x); };
    uint32_t k = find_key(off_out, keys, s);
    uint32_t lo = off_out[k], hi = off_out[k + 1], in_lo = off_in[k], in_hi = off_in[k + 1];
    const uint32_t rounds = (e - s + B - 1) / B, per = (e - s + rounds - 1) / rounds;
    uint32_t* const ents1 = scratch.ent1 + t;
    uint32_t* const ents2 = scratch.ent2 + t;
    auto ent1 = [&](int i) -> uint32_t& { return ents1[(size_t)i * threads]; };
    auto ent2 = [&](int i) -> uint32_t& { return ents2[(size_t)i * threads]; };
    auto put_prefix = [&](int i, const Fp& v) {
#pragma unroll
        for (int p = 0; p < 3; p++)
            scratch.prefix[((size_t)i * 3 + p) * threads + t] = make_uint4(v.l[4 * p], v.l[4 * p + 1], v.l[4 * p + 2], v.l[4 * p + 3]);
    };
    auto get_prefix = [&](int i) {
        Fp v;
#pragma unroll
        for (int p = 0; p < 3; p++) {
            const uint4 q = scratch.prefix[((size_t)i * 3 + p) * threads + t];
            v.l[4 * p] = q.x;
            v.l[4 * p + 1] = q.y;
            v.l[4 * p + 2] = q.z;
            v.l[4 * p + 3] = q.w;
        }
        return v;
    };
    for (uint32_t j0 = s; j0 < e; j0 += per) {
        const int n = (int)min(per, e - j0);
        for (int i = 0; i < n; i++) {
            const uint32_t j = j0 + (uint32_t)i;
            if (j >= hi) {
                lo = hi;  // buckets in between are empty
                for (int w = 0; j >= hi; w++) {
                    k = w < kWalk ? k + 1 : seek_key(off_out, keys, k, j);
                    hi = off_out[k + 1];
                }
                in_lo = off_in[k];
                in_hi = off_in[k + 1];
            }
            const uint32_t p = in_lo + 2 * (j - lo);
            const bool two = p + 1 < in_hi;
            ent1(i) = kGather ? __ldg(sorted + p) : p;
            ent2(i) = !two ? kNoKey : kGather ? __ldg(sorted + p + 1) : p + 1;
        }
        // forward: the x of the next sum's points are loaded one sum ahead and
        // its entries two, so that no address waits on a load
        uint32_t c1 = ent1(0), c2 = ent2(0), e1 = 0, e2 = kNoKey;
        Fp acc = fp_one(), n1 = fp_zero(), n2 = fp_zero();
        if (c2 != kNoKey) {
            n1 = point_x(c1);
            n2 = point_x(c2);
        }
        if (n > 1) {
            e1 = ent1(1);
            e2 = ent2(1);
        }
        for (int i = 0; i < n; i++) {
            const Fp x1 = n1, x2 = n2;
            const uint32_t p1 = c1, p2 = c2;
            c1 = e1;
            c2 = e2;
            e2 = kNoKey;
            if (i + 2 < n) {
                e1 = ent1(i + 2);
                e2 = ent2(i + 2);
            }
            if (c2 != kNoKey) {
                n1 = point_x(c1);
                n2 = point_x(c2);
            }
            if (p2 == kNoKey) continue;
            Fp d = fp_sub(x2, x1);
            if (maybe_special(d, x1, x2)) {
                const PairCase c = pair_case(signed_point(point(p1), p1), signed_point(point(p2), p2));
                if (c.kind == kPairFirst || c.kind == kPairSecond || c.kind == kPairInfinity) continue;
                d = c.den;
            }
            put_prefix(i, acc);
            acc = fp_mul(acc, d);
        }
        Fp inv = fp_invert(acc);
        // backward: points and partial product one sum ahead, entries two
        c1 = ent1(n - 1);
        c2 = ent2(n - 1);
        if (n > 1) {
            e1 = ent1(n - 2);
            e2 = ent2(n - 2);
        }
        Affine na = point(c1), nb = na;
        Fp npre = get_prefix(n - 1);
        if (c2 != kNoKey) nb = point(c2);
        for (int i = n - 1; i >= 0; i--) {
            Affine a = signed_point(na, c1);
            const Affine b = signed_point(nb, c2);
            const Fp pre = npre;
            const bool two = c2 != kNoKey;
            c1 = e1;
            c2 = e2;
            if (i > 1) {
                e1 = ent1(i - 2);
                e2 = ent2(i - 2);
            }
            if (i > 0) {
                na = point(c1);
                if (c2 != kNoKey) {
                    nb = point(c2);
                    npre = get_prefix(i - 1);
                }
            }
            if (two) {
                Fp d = fp_sub(b.x, a.x), num = fp_sub(b.y, a.y);
                int kind = kPairAdd;
                if (maybe_special(d, a.x, b.x)) {  // as in the forward pass
                    const PairCase c = pair_case(a, b);
                    kind = c.kind;
                    d = c.den;
                    num = c.num;
                }
                if (kind == kPairSecond) {
                    a = b;
                } else if (kind == kPairInfinity) {
                    a.x = fp_zero();
                    a.y = fp_zero();
                } else if (kind != kPairFirst) {
                    Fp di, next;
                    fp_mul2(di, inv, pre, next, inv, d);
                    inv = next;
                    const Fp lam = fp_mul(num, di);
                    const Fp x3 = fp_sub(fp_sub(fp_sqr(lam), a.x), b.x);
                    a.y = fp_sub(fp_mul(lam, fp_sub(a.x, x3)), a.y);
                    a.x = x3;
                }
            }
            store_affine(&out[j0 + (uint32_t)i], a);
        }
    }
}

// The same walk with one quad of lanes per chunk, for inputs too small to fill
// the GPU with lanes (accumulate_quad_blocks): bound by the latency of the
// additions, which a quad finishes in less than half the time.  An affine
// point enters quad_add with ZZ = ZZZ = 1.
__global__ void __launch_bounds__(kAccThreads) k_accumulate_quads(const Affine* __restrict__ bases,
                                                                  const uint32_t* __restrict__ sorted,
                                                                  const uint32_t* __restrict__ offsets, uint32_t keys,
                                                                  Xyzz* __restrict__ buckets,
                                                                  Xyzz* __restrict__ partials, const Owners own) {
    const uint32_t chunks = (gridDim.x * blockDim.x) >> 2;
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
    const uint32_t q = threadIdx.x & 3, base = threadIdx.x & 28;
    const uint32_t total = offsets[keys];
    const uint32_t len = (total + chunks - 1) / chunks;
    uint32_t s, e;
    chunk_range(total, t, chunks, s, e);
    uint32_t k = 0, seg_lo = 0, seg_hi = 0;
    if (s < e) {
        k = find_key(offsets, keys, s);
        seg_lo = offsets[k];
        seg_hi = offsets[k + 1];
    }
    // lanes 0 and 1 load x and y, one entry ahead
    auto load = [&](uint32_t ent) {
        const uint4* src = reinterpret_cast<const uint4*>(bases + (ent & 0x7fffffffu)) + 3 * q;
        Fp r = fp_one();
        if (q < 2) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const uint4 v = __ldg(src + i);
                r.l[4 * i] = v.x;
                r.l[4 * i + 1] = v.y;
                r.l[4 * i + 2] = v.z;
                r.l[4 * i + 3] = v.w;
            }
        }
        return r;
    };
    auto flush = [&](const Fp& acc) {
        if (seg_lo >= s && seg_hi <= e) {
            quad_store(&buckets[k], acc);
        } else if (seg_lo < s) {
            quad_store(&partials[2 * (size_t)t], acc);
        } else {
            quad_store(&partials[2 * (size_t)t + 1], acc);
            if (q == 0) own.list[atomicAdd(own.count, 1u)] = make_uint2(t, k);
        }
    };
    Fp acc = fp_zero(), nxt = fp_zero();
    uint32_t ent = 0;
    if (s < e) {
        ent = __ldg(sorted + s);
        nxt = load(ent);
    }
    for (uint32_t i = 0; i < len; i++) {  // the same count for every quad
        const uint32_t j = s + i;
        const bool on = j < e;
        if (on && j == seg_hi) {
            flush(acc);
            acc = fp_zero();
            seg_lo = seg_hi;
            for (int w = 0; seg_hi <= j; w++) {  // past empty buckets
                k = w < kWalk ? k + 1 : seek_key(offsets, keys, k, j);
                seg_hi = offsets[k + 1];
            }
        }
        Fp p = nxt;
        const uint32_t cur = ent;
        if (j + 1 < e) {
            ent = __ldg(sorted + j + 1);
            nxt = load(ent);
        }
        const uint32_t z = (__ballot_sync(0xffffffffu, fp_is_zero_raw(p)) >> base) & 3u;  // x and y both zero: infinity
        p = fp_select(q == 1 && (cur >> 31) != 0, fp_neg(p), p);
        acc = quad_add(acc, fp_select(on && z != 3u, p, fp_zero()));
    }
    if (s < e) flush(acc);
}

// A cut bucket is finished by one quad of lanes, since the additions of its
// span are a serial chain.  The buckets come from a list that the accumulation
// made, so that the quads of a warp all have one: where a bucket spans many
// chunks few chunks start one, and walking the chunks instead left most quads
// idle (proof of 2^14 rows, six calls: 699 us).  A bucket spanning many chunks
// (a heavy bucket: scalars 0/1, a nearly empty top window) is queued for
// k_fixup_pieces: the chain of 12 additions that a quad still takes itself costs
// ~55 us, a block's tree ~30 for any span up to 64.
constexpr uint32_t kShortSpan = 12;

// Long spans in two steps: pieces of kPiece chunks, each one block's tree of
// quads, whose sums take the place of the piece's first partial; then the
// pieces of a span.  A span of 600 chunks (a column of small values in a proof
// of 2^14 rows) is a chain of 6 + 4 additions instead of the 10 + 6 of a block
// that strides over it.
constexpr uint32_t kPiece = 64;
struct LongSpans {
    uint32_t* count;  // spans, pieces
    uint4* list;      // (first chunk, last chunk, bucket key, -)
    uint4* pieces;    // (first chunk of the span, piece, its last chunk, -)
};
__host__ __device__ constexpr uint32_t pieces_of(uint32_t first, uint32_t last) {
    return (last - first) / kPiece + 1;
}
// where the sum of a span's piece lives
__device__ __forceinline__ size_t piece_slot(uint32_t first, uint32_t piece) {
    return 2 * ((size_t)first + (size_t)piece * kPiece) + (piece == 0 ? 1u : 0u);
}

__global__ void __launch_bounds__(kReduceThreads) k_fixup(const uint32_t* __restrict__ offsets, uint32_t keys,
                                                          uint32_t chunks, const Xyzz* __restrict__ partials,
                                                          const Owners own, Xyzz* __restrict__ buckets,
                                                          const LongSpans spans) {
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 2, n = *own.count;
    if ((i & ~7u) >= n) return;  // the whole warp
    bool mine = i < n;
    uint32_t u = 1, last = 0, k = 0;
    Fp acc = fp_zero();
    if (mine) {
        const uint2 o = own.list[i];
        const uint32_t t = o.x, total = offsets[keys], len = (total + chunks - 1) / chunks;
        k = o.y;
        last = (offsets[k + 1] - 1) / len;
        u = t + 1;
        if (last - t > kShortSpan) {
            if ((threadIdx.x & 3) == 0) {
                spans.list[atomicAdd(spans.count, 1u)] = make_uint4(t, last, k, 0);
                const uint32_t np = pieces_of(t, last), at = atomicAdd(spans.count + 1, np);
                for (uint32_t p = 0; p < np; p++) spans.pieces[at + p] = make_uint4(t, p, last, 0);
            }
            mine = false;
            last = t;
        } else {
            acc = quad_load(&partials[2 * (size_t)t + 1]);
        }
    }
    for (; __any_sync(0xffffffffu, u <= last); u++)
        acc = quad_add(acc, u <= last ? quad_load(&partials[2 * (size_t)u]) : fp_zero());
    if (mine) quad_store(&buckets[k], acc);
}

constexpr int kLongThreads = 256;  // a quad per chunk of a piece
static_assert(kLongThreads / 4 == kPiece, "one quad per chunk");

// The quads' points added pairwise (warps stay together); the result in quad 0
// and sm[0].  `live`: points beyond it are infinity.
__device__ __forceinline__ void block_sum(Fp acc, Xyzz* sm, uint32_t live) {
    const uint32_t quad = threadIdx.x >> 2;
    quad_store(&sm[quad], acc);
    __syncthreads();
    uint32_t off = kPiece / 2;
    while (off > 0 && off >= live) off >>= 1;
    for (; off > 0; off >>= 1) {
        if ((quad & ~7u) < off) {
            const Fp r = quad_add(quad_load(&sm[quad]), quad < off ? quad_load(&sm[quad + off]) : fp_zero());
            if (quad < off) quad_store(&sm[quad], r);
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kLongThreads) k_fixup_pieces(Xyzz* __restrict__ partials, const LongSpans spans) {
    __shared__ Xyzz sm[kPiece];
    const uint32_t quad = threadIdx.x >> 2;
    for (uint32_t i = blockIdx.x; i < spans.count[1]; i += gridDim.x) {
        const uint4 pc = spans.pieces[i];
        const uint32_t first = pc.x, piece = pc.y, last = pc.z;
        const uint32_t u = first + piece * kPiece + quad;
        const uint32_t live = min(kPiece, last - (first + piece * kPiece) + 1);
        const Fp acc = quad < live ? quad_load(&partials[u == first ? 2 * (size_t)u + 1 : 2 * (size_t)u]) : fp_zero();
        block_sum(acc, sm, live);
        if (quad == 0) quad_store(&partials[piece_slot(first, piece)], quad_load(&sm[0]));
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kLongThreads) k_fixup_long(const Xyzz* __restrict__ partials, const LongSpans spans,
                                                             Xyzz* __restrict__ buckets) {
    __shared__ Xyzz sm[kPiece];
    const uint32_t quad = threadIdx.x >> 2;
    for (uint32_t item = blockIdx.x; item < spans.count[0]; item += gridDim.x) {
        const uint4 sp = spans.list[item];
        const uint32_t np = pieces_of(sp.x, sp.y);
        Fp acc = quad < np ? quad_load(&partials[piece_slot(sp.x, quad)]) : fp_zero();
        for (uint32_t p = quad + kPiece; __any_sync(0xffffffffu, p < np); p += kPiece)
            acc = quad_add(acc, p < np ? quad_load(&partials[piece_slot(sp.x, p)]) : fp_zero());
        block_sum(acc, sm, np);
        if (quad == 0) quad_store(&buckets[sp.z], quad_load(&sm[0]));
        __syncthreads();
    }
}

// ---- bucket reduction over a table of windows ----
//
// A window's sum is S = sum_{b=1}^{nb} b B_b.  Its nb = 2^m buckets are merged
// pairwise in a tree whose nodes hold the sum R of their leaves and, for every
// bit t below the node's height, the plane sum P_t over the leaves whose index
// has bit t set.  Merging two nodes adds R and every P_t of the halves and
// gains the plane of its own height for free (the right half's R), so the
// whole tree takes ~2 nb additions, as many as running sums, and is only m
// additions deep.  Then S = R + sum_t 2^t P_t.
//
// k_tree runs up to kTreeFirst heights of it per launch, each block a subtree in
// shared memory with one quad of lanes per addition (a quad addition takes a third
// of the time of a one-lane addition, and these are chains).  Where a call has
// buckets enough to fill the GPU with one-lane work anyway (kTreeKeys),
// k_group_sums first folds groups of L = 2^glen buckets by running sums
// (R_g = sum of the group's buckets, T_g = sum_i (i+1) B_{gL+i}, ~1/4 less
// work per bucket than the quads) and the tree runs over the groups:
// S = sum_g T_g + L sum_t 2^t P_t.  k_tree_finish shifts the planes of a window
// side by side and adds them up.
//
// Bound by the latency of a product chain for few buckets and by the integer
// multiply pipe for many.  Device time of the whole reduction, against running
// sums over groups with one lane per addition, plane sums and a serial Horner
// step per window: 4096 buckets (1000 points) 496 -> 94 us, 81920 (2^16
// points) 1177 -> 265 us, 524288 (10^6 points) 1846 -> 895 us.
struct GroupWin {
    uint32_t key_start;    // first bucket key of the window
    uint32_t group_start;  // first running-sum group of the window
    uint32_t glen_log;     // log2 of the buckets per group
};

// The bucket sets of an MSM over the same keys (one per part of a pipelined
// MSM), added bucket by bucket; a key is empty in a set when its offsets
// say so (its bucket is then never written)
struct BucketSets {
    const Xyzz* buckets[kMaxMsmParts];
    const uint32_t* offsets[kMaxMsmParts];
    uint32_t n;
};

// group g leaves the pair T_g, R_g at out[2 g]
__global__ void __launch_bounds__(kReduceThreads) k_group_sums(const BucketSets sets,
                                                               const GroupWin* __restrict__ wins, uint32_t n_wins,
                                                               uint32_t total_groups, Xyzz* __restrict__ out) {
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= total_groups) return;
    uint32_t lo = 0, hi = n_wins;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (wins[mid].group_start <= gid) lo = mid;
        else hi = mid;
    }
    const GroupWin wd = wins[lo];
    const uint32_t key0 = wd.key_start + ((gid - wd.group_start) << wd.glen_log);
    Xyzz run, tot;
    xyzz_set_inf(run);
    xyzz_set_inf(tot);
    for (int b = (1 << wd.glen_log) - 1; b >= 0; b--) {
        const uint32_t key = key0 + (uint32_t)b;
#pragma unroll
        for (uint32_t s = 0; s < kMaxMsmParts; s++)
            if (s < sets.n && sets.offsets[s][key + 1] > sets.offsets[s][key])
                run = xyzz_add(run, load_xyzz(&sets.buckets[s][key]));
        tot = xyzz_add(tot, run);
    }
    store_xyzz(&out[2 * (size_t)gid], tot);
    store_xyzz(&out[2 * (size_t)gid + 1], run);
}

// One launch of k_tree on one window: 2^b of its nodes per block.  A node has
// v values: its planes (and T), R last; it leaves with v + b values.
struct TreeWin {
    uint32_t blk_start;  // the window's first block
    uint32_t in_start;   // its first value (points)
    uint32_t out_start;
    uint32_t v, b;
};
constexpr uint32_t kTreePoints = 256;  // points of a block's subtree (48 KB of shared memory)
constexpr uint32_t kTreeFirst = 7;      // heights of a launch over single buckets, the most of any launch (plan_reduce)

// Values are merged in place.  Value j of the node over the leaves from L sits
// in slot (L, j), its new plane t in the last slot of leaf L + 2^t (the R that
// the right half left there), its R in the last slot of leaf L.
// offsets (first launch over buckets only): key k is empty, and its bucket
// never written, when offsets[k + 1] == offsets[k].
__global__ void __launch_bounds__(256) k_tree(const Xyzz* __restrict__ in, const uint32_t* __restrict__ offsets,
                                              const TreeWin* __restrict__ wins, uint32_t n_wins,
                                              Xyzz* __restrict__ out) {
    __shared__ Xyzz sm[kTreePoints];
    uint32_t lo = 0, hi = n_wins;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (wins[mid].blk_start <= blockIdx.x) lo = mid;
        else hi = mid;
    }
    const TreeWin w = wins[lo];
    const uint32_t blk = blockIdx.x - w.blk_start, v = w.v;
    const uint32_t points = v << w.b, quads = blockDim.x >> 2, quad = threadIdx.x >> 2;
    const uint32_t first = w.in_start + blk * points;
    for (uint32_t i = quad; i < points; i += quads) {
        const bool empty = offsets && offsets[first + i + 1] == offsets[first + i];
        quad_store(&sm[i], empty ? fp_zero() : quad_load(&in[first + i]));
    }
    __syncthreads();
    for (uint32_t s = 0; s < w.b; s++) {
        const uint32_t per = v + s, ops = per << (w.b - s - 1);
        for (uint32_t o = quad; (o & ~7u) < ops; o += quads) {  // a warp's eight quads stay together
            const uint32_t m = o / per, r = o % per;
            const uint32_t left = m << (s + 1), half = 1u << s;
            uint32_t dst = left * v + r;
            if (r >= v) dst = (left + (1u << (r - v))) * v + v - 1;  // plane r - v gained below
            const bool on = o < ops;
            const uint32_t src = dst + half * v;
            const Fp sum = quad_add(on ? quad_load(&sm[dst]) : fp_zero(), on ? quad_load(&sm[src]) : fp_zero());
            // slot (left + half, v - 1), the R of the right half, is read here
            // and stays: it is the merged node's plane s
            if (on) quad_store(&sm[dst], sum);
        }
        __syncthreads();
    }
    const uint32_t nv = v + w.b;
    for (uint32_t i = quad; i < nv; i += quads) {
        const uint32_t slot = i + 1 < v ? i : i + 1 == nv ? v - 1 : (1u << (i + 1 - v)) * v + v - 1;
        quad_store(&out[w.out_start + blk * nv + i], quad_load(&sm[slot]));
    }
}

// A window's values when one node is left.  Over buckets: planes t = 0.. with
// weight 2^t, then R with weight 1.  Over groups (glen > 0): T with weight 1,
// planes t with weight 2^(glen + t), then R, which has no part.
struct FinWin {
    uint32_t start;
    uint32_t v;
    uint32_t glen_log;
};
constexpr uint32_t kFinThreads = 128;  // 32 quads: v <= 25 values (c <= 24)

__global__ void __launch_bounds__(kFinThreads) k_tree_finish(const Xyzz* __restrict__ in,
                                                             const FinWin* __restrict__ wins, Xyzz* __restrict__ out) {
    __shared__ Xyzz sm[kFinThreads / 4];
    const FinWin w = wins[blockIdx.x];
    const uint32_t i = threadIdx.x >> 2;
    Fp acc = fp_zero();
    uint32_t shift = 0;
    if (w.glen_log == 0) {
        if (i < w.v) acc = quad_load(&in[w.start + i]);
        if (i + 1 < w.v) shift = i;
    } else if (i + 1 < w.v) {
        acc = quad_load(&in[w.start + i]);
        if (i > 0) shift = w.glen_log + i - 1;
    }
    for (uint32_t k = 0; __any_sync(0xffffffffu, k < shift); k++) {
        const Fp d = quad_dbl(acc);
        acc = fp_select(k < shift, d, acc);
    }
    quad_store(&sm[i], acc);
    __syncthreads();
    for (uint32_t off = 1u << (31 - __clz(w.v - 1)); off > 0; off >>= 1) {  // w.v >= 2 values
        if ((i & ~7u) < off) {
            const Fp r = quad_add(quad_load(&sm[i]), i < off ? quad_load(&sm[i + off]) : fp_zero());
            __syncwarp();
            if (i < off) quad_store(&sm[i], r);
        }
        __syncthreads();
    }
    if (i == 0) quad_store(&out[blockIdx.x], quad_load(&sm[0]));
}

// One window of a reduction: its buckets' keys
struct Window {
    uint32_t key_start;
    uint32_t log_nb;
};

// The launches of one reduction and their tables
struct ReducePlan {
    uint32_t n_wins = 0;
    uint32_t total_groups = 0;        // running-sum groups, 0: the tree starts at the buckets
    std::vector<GroupWin> group;
    std::vector<TreeWin> tree;        // every launch's table, back to back
    struct Launch {
        uint32_t first, count, blocks, threads;
    };
    std::vector<Launch> launches;
    std::vector<FinWin> fin;
    uint64_t arena = 0;  // points: the groups' pairs, then every launch's values
    size_t table_bytes() const {
        return group.size() * sizeof(GroupWin) + tree.size() * sizeof(TreeWin) + fin.size() * sizeof(FinWin);
    }
    void pack(void* dst) const {
        char* p = static_cast<char*>(dst);
        std::memcpy(p, group.data(), group.size() * sizeof(GroupWin));
        p += group.size() * sizeof(GroupWin);
        std::memcpy(p, tree.data(), tree.size() * sizeof(TreeWin));
        p += tree.size() * sizeof(TreeWin);
        std::memcpy(p, fin.data(), fin.size() * sizeof(FinWin));
    }
};

// glen_log 0: the tree starts at the buckets
ReducePlan plan_reduce(const std::vector<Window>& wins, uint32_t glen_log) {
    ReducePlan p;
    p.n_wins = (uint32_t)wins.size();
    struct State {
        uint32_t start, log_nodes, v, glen;
    };
    std::vector<State> st;
    for (const Window& w : wins) {
        if (glen_log) {
            const uint32_t g = std::min(glen_log, w.log_nb);
            p.group.push_back({w.key_start, p.total_groups, g});
            st.push_back({2 * p.total_groups, w.log_nb - g, 2, g});
            p.total_groups += 1u << (w.log_nb - g);
        } else {
            st.push_back({w.key_start, w.log_nb, 1, 0});
        }
    }
    p.arena = 2 * (uint64_t)p.total_groups;
    bool over_leaves = glen_log == 0;
    for (;;) {
        const uint32_t at = (uint32_t)p.tree.size();
        uint32_t blocks = 0, most = 0;
        for (State& s : st) {
            if (s.log_nodes == 0) continue;
            // as many heights as fit, seven over single buckets: 32 quads then
            // have work for the first four of them.  Measured (MSM of 1000003
            // points, 524288 buckets): 6 heights with 32 / 64 quads 7.55 /
            // 8.29 ms per call, 7 with 32 / 64 7.42 / 7.79, 8 with 32 / 64
            // 7.40 / 7.59; 65536 points: all within 3 %.
            uint32_t b = 0;
            while (b < s.log_nodes && (s.v << (b + 1)) <= kTreePoints && !(s.v == 1 && b == kTreeFirst)) b++;
            TreeWin t{blocks, s.start, (uint32_t)p.arena, s.v, b};
            const uint32_t n = 1u << (s.log_nodes - b);
            most = std::max(most, s.v << (b - 1));
            blocks += n;
            s.start = (uint32_t)p.arena;
            s.v += b;
            s.log_nodes -= b;
            p.arena += (uint64_t)n * s.v;
            p.tree.push_back(t);
        }
        if (p.tree.size() == at) break;
        p.launches.push_back({at, (uint32_t)p.tree.size() - at, blocks, over_leaves || most <= 32 ? 128u : 256u});
        over_leaves = false;
    }
    for (const State& s : st) p.fin.push_back({s.start, s.v, s.glen});
    return p;
}

// Total buckets from which running sums over groups come first: the tree from
// the buckets is faster at 1.6 M buckets (commitment batch of 24 items over a
// window table: 25.0 ms per call against 26.0 with groups), the groups at 6.8 M
// (2^24 points: 92.0 against 94.0).
constexpr uint64_t kTreeKeys = 1u << 22;

// log2 of the buckets per running-sum group of a call with `keys` buckets in
// `sets` sets (0: none, the tree starts at the buckets)
uint32_t reduce_group_log(uint64_t keys, uint32_t sets) {
    if (sets == 1 && keys < kTreeKeys) return 0;
    uint32_t g = 2;
    while (g < 6 && (keys >> (g + 1)) >= 32768) g++;
    return g;
}

// The launches of `p` on `st`.  d_tab: its packed tables; arena: p.arena
// points.  Returns the launch error, if any; adds the launches to *launches
// when given.
cudaError_t launch_reduce(const ReducePlan& p, const BucketSets& sets, const void* d_tab, Xyzz* arena, Xyzz* wsum,
                          uint64_t* launches, cudaStream_t st) {
    const GroupWin* d_group = static_cast<const GroupWin*>(d_tab);
    const TreeWin* d_tree = reinterpret_cast<const TreeWin*>(d_group + p.group.size());
    const FinWin* d_fin = reinterpret_cast<const FinWin*>(d_tree + p.tree.size());
    uint64_t n = 1;
    if (p.total_groups) {
        k_group_sums<<<(p.total_groups + kReduceThreads - 1) / kReduceThreads, kReduceThreads, 0, st>>>(
            sets, d_group, p.n_wins, p.total_groups, arena);
        n++;
    }
    bool over_buckets = p.total_groups == 0;
    for (const ReducePlan::Launch& l : p.launches) {
        k_tree<<<l.blocks, l.threads, 0, st>>>(over_buckets ? sets.buckets[0] : arena,
                                               over_buckets ? sets.offsets[0] : nullptr, d_tree + l.first, l.count,
                                               arena);
        over_buckets = false;
        n++;
    }
    k_tree_finish<<<p.n_wins, kFinThreads, 0, st>>>(arena, d_fin, wsum);
    if (launches) *launches += n;
    return cudaGetLastError();
}

// the windows of one MSM, appended to `wins`
void append_windows(const MsmShape& sh, uint64_t key_base, int windows, std::vector<Window>& wins) {
    for (int w = 0; w < windows; w++)
        wins.push_back({(uint32_t)(key_base + (uint64_t)w * sh.nb), (uint32_t)(sh.c - 1)});
}

// Blocks of k_accumulate_quads for at most `entries` sorted entries, 0 where
// one lane per chunk is faster.  A lane adds one point in ~12 us, a quad in ~5,
// and a quarter as many chunks leave the cut buckets shorter spans: with up to
// ~16 entries per quad that is faster than 1..4 per lane.  Per call, lanes
// against quads: 1000 points (32000 entries) 620 -> 451 us, 4096 (119000
// entries) 590 -> 525, 8192 (213000) 592 -> 635.  Two blocks of 128 per SM: with
// one 470 us, with three 466 at 1000 points.
constexpr uint64_t kQuadEntries = 150000;

uint32_t accumulate_quad_blocks(const Context* ctx, uint64_t entries) {
    return entries > kQuadEntries ? 0u : (uint32_t)ctx->num_sms * 2;
}

// The queues of an accumulation: the counters (owners; spans, pieces) in 16
// bytes, then the long spans, their pieces (a span has more than kShortSpan
// chunks, a piece kPiece but for a span's last, and every chunk lies in one span
// but for its last bucket's: less than one per chunk of either) and the owners
// (at most one per chunk).
struct Queues {
    Owners own;
    LongSpans spans;
};
constexpr size_t queue_bytes(size_t chunks) { return 16 + chunks * (2 * sizeof(uint4) + sizeof(uint2)); }
Queues queues_at(void* p, size_t chunks) {
    uint32_t* counts = static_cast<uint32_t*>(p);
    uint4* spans = reinterpret_cast<uint4*>(counts + 4);
    uint4* pieces = spans + chunks;
    return {{counts, reinterpret_cast<uint2*>(pieces + chunks)}, {counts + 1, spans, pieces}};
}

template <bool kHalves = false>
Status scan_u32(Context* ctx, const uint32_t* in, uint32_t* out, uint32_t len, cudaStream_t st) {
    const uint32_t tiles = (len + kScanTile - 1) / kScanTile;
    void* sums;
    MZK_TRY(ctx->ensure("scan_sums", (size_t)tiles * 4 + 64, &sums));
    k_scan_tiles<kHalves><<<tiles, kScanThreads, 0, st>>>(in, out, len, (uint32_t*)sums);
    MZK_LAUNCH_CHECK(ctx);
    k_scan_sums<<<1, kScanThreads, 0, st>>>((uint32_t*)sums, tiles);
    MZK_LAUNCH_CHECK(ctx);
    k_scan_add<<<tiles, kScanThreads, 0, st>>>(out, len, (const uint32_t*)sums);
    MZK_LAUNCH_CHECK(ctx);
    return OK;
}

// What the accumulation of one sorted entry array needs
struct Accumulation {
    const Affine* bases;
    const uint32_t* sorted;
    const uint32_t* offsets;  // keys + 2
    uint32_t keys;
    Xyzz* buckets;
    Xyzz* partials;
    void* queue;           // queue_bytes of the lanes' grid, which is the larger one
    uint32_t acc_blocks;   // lanes' grid
    uint32_t quad_blocks;  // > 0: by quads
    uint32_t long_blocks;
};

// The bucket sums by quads or by lanes (gather: see k_accumulate).  Returns
// the launch error, if any.
cudaError_t launch_accumulate(const Accumulation& a, bool gather, cudaStream_t st) {
    const Queues q = queues_at(a.queue, (size_t)a.acc_blocks * kAccThreads);
    cudaError_t e = cudaMemsetAsync(a.queue, 0, 16, st);
    if (e != cudaSuccess) return e;
    if (a.quad_blocks)
        k_accumulate_quads<<<a.quad_blocks, kAccThreads, 0, st>>>(a.bases, a.sorted, a.offsets, a.keys, a.buckets,
                                                                  a.partials, q.own);
    else if (gather)
        k_accumulate<true><<<a.acc_blocks, kAccThreads, 0, st>>>(a.bases, a.sorted, a.offsets, a.keys, a.buckets,
                                                                 a.partials, q.own);
    else
        k_accumulate<false><<<a.acc_blocks, kAccThreads, 0, st>>>(a.bases, nullptr, a.offsets, a.keys, a.buckets,
                                                                  a.partials, q.own);
    return cudaGetLastError();
}

// The sums of the buckets that the chunks cut.
cudaError_t launch_fixup(const Accumulation& a, cudaStream_t st) {
    const Queues q = queues_at(a.queue, (size_t)a.acc_blocks * kAccThreads);
    const uint32_t chunks = a.quad_blocks ? a.quad_blocks * (kAccThreads / 4) : a.acc_blocks * kAccThreads;
    k_fixup<<<chunks * 4 / kReduceThreads, kReduceThreads, 0, st>>>(a.offsets, a.keys, chunks, a.partials, q.own,
                                                                   a.buckets, q.spans);
    k_fixup_pieces<<<a.long_blocks, kLongThreads, 0, st>>>(a.partials, q.spans);
    k_fixup_long<<<a.long_blocks, kLongThreads, 0, st>>>(a.partials, q.spans, a.buckets);
    return cudaGetLastError();
}

// Rounds of pair sums by `threads` threads for `entries` entries over `keys`
// buckets.  A sum costs less than a mixed addition only while a thread has ~48 to
// share an inversion, and a round halves buckets of four points or more.  Per
// call without and with them: 200000 points (4.0 M entries, one round) 2.10 and
// 2.00 ms, 262144 (5.0 M) 2.51 and 2.36, 524288 (8.4 M, two) 4.29 and 3.96,
// 1000003 (16.0 M, three) 7.28 and 6.15, 2^24 (218 M) 91.8 and 81.9.  The line was
// set with batches of 64 sums, where 5.0 M entries gained nothing (2.60 and 2.59;
// 1000003 points with 1 / 2 / 3 rounds 6.86 / 6.73 / 6.66).
constexpr uint64_t kPairsPerThread = 48;
constexpr int kPairRounds = 3;

int pair_rounds(uint64_t entries, uint64_t keys, uint64_t threads) {
    int r = 0;
    while (r < kPairRounds && (entries >> (r + 1)) >= kPairsPerThread * threads && (entries >> r) >= 4 * keys) r++;
    return r;
}

// ---- memory of the pair sums ----
//
// A context holds at most pair_limit bytes for them, whatever the call: the
// scratch of k_pair_sums, and for one part of the keys at a time two arrays of
// sums and two of offsets.  The parts are cut by the true counts (k_part_keys),
// not by the callers' items or windows, since one bucket set may hold every
// entry of a call (an item over a window table).  Where a single bucket and its
// neighbours exceed the room their entries are accumulated as they are.
constexpr size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Where a part's arrays lie behind the scratch.  A round leaves at most half of
// its points and one more per bucket.
struct PairLayout {
    size_t sums[2], offs[2], bytes;
};
PairLayout pair_layout(uint64_t entries, uint64_t keys, int rounds) {
    const uint64_t n0 = std::min(entries, (entries + keys) / 2), n1 = std::min(n0, (n0 + keys) / 2);
    PairLayout l;
    l.offs[0] = 0;
    l.offs[1] = l.offs[0] + align256((keys + 2) * 4);
    l.sums[0] = l.offs[1] + (rounds > 1 ? align256((keys + 2) * 4) : 0);
    l.sums[1] = l.sums[0] + align256((size_t)n0 * sizeof(Affine));
    l.bytes = l.sums[1] + (rounds > 1 ? align256((size_t)n1 * sizeof(Affine)) : 0);
    return l;
}
// bytes of a part are below this much per entry and key (entries = keys = half of both)
constexpr uint64_t kPairBytes = sizeof(Affine) + 2 * sizeof(uint32_t);

// Consecutive keys whose sums are formed together
struct PairPart {
    uint32_t k0, k1;   // keys
    uint32_t first;    // offset of k0
    uint64_t entries;
    bool paired;       // false: accumulated as they are
};

// Split points i * step (i < n) of offset + key: the largest key at or below,
// and its offset
__global__ void k_part_keys(const uint32_t* __restrict__ offsets, uint32_t keys, uint64_t step, uint32_t n,
                            uint2* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t target = i * step;
    uint32_t lo = 0, hi = keys + 1;
    while (hi - lo > 1) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if ((uint64_t)offsets[mid] + mid <= target) lo = mid;
        else hi = mid;
    }
    out[i] = make_uint2(lo, offsets[lo]);
}

// A part's offsets from zero
__global__ void k_rebase(const uint32_t* __restrict__ in, uint32_t len, uint32_t* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < len) out[i] = in[i] - in[0];
}

// Neighbouring split points joined into parts of at most `room` bytes, as few
// as possible.  Empty where not even the offsets of one fit.
std::vector<PairPart> join_greedily(const std::vector<uint2>& points, int rounds, uint64_t room) {
    auto fits = [&](const uint2& a, const uint2& b) {
        return pair_layout(b.y - a.y, b.x - a.x, rounds).bytes <= room;
    };
    std::vector<PairPart> parts;
    for (size_t i = 0; i + 1 < points.size();) {
        size_t j = i + 1;
        while (j + 1 < points.size() && fits(points[i], points[j + 1])) j++;
        const uint2 a = points[i], b = points[j];
        i = j;
        if (a.x == b.x) continue;
        const PairPart p{a.x, b.x, a.y, b.y - a.y, fits(a, b)};
        if (!p.paired && align256((size_t)(p.k1 - p.k0 + 2) * 4) > room) return {};
        parts.push_back(p);
    }
    return parts;
}

// The split points of a call are at most 1 / kPairSteps of a part apart (more
// only where they would be too many).
constexpr uint32_t kPairSteps = 64, kMaxSplitPoints = 4096;

// The same with parts of about equal size: a thread forms its share of a part in
// batches of up to kPairBatch sums, and parts just over a multiple of that have
// many small batches (2^24 points: 83.5 ms per call in full parts and a
// remainder, 82.0 in equal ones; in windows, two at a time, 81.8).
std::vector<PairPart> join_parts(const std::vector<uint2>& points, int rounds, uint64_t room) {
    std::vector<PairPart> parts = join_greedily(points, rounds, room);
    if (parts.size() < 2) return parts;
    const uint64_t n = parts.size();
    const uint64_t even = pair_layout(points.back().y / n, points.back().x / n, rounds).bytes;
    std::vector<PairPart> evened = join_greedily(points, rounds, std::min(room, even + room / kPairSteps));
    return evened.size() == n ? evened : parts;
}

// Rounds and parts of a call's pair sums (no parts: none).  `entries` is an
// upper bound (no zero digits); where it calls for rounds the true number,
// which decides, is read back through `total` (pinned), with the split points
// where the call may not fit one part.
Status plan_pairs(Context* ctx, const Accumulation& all, uint64_t entries, uint64_t threads, uint64_t room,
                  uint32_t* total, int* rounds, std::vector<PairPart>* parts, cudaStream_t st) {
    *rounds = all.quad_blocks ? 0 : pair_rounds(entries, all.keys, threads);
    if (!*rounds || !room) return OK;
    std::vector<uint2> points;
    if (pair_layout(entries, all.keys, *rounds).bytes > room) {
        const uint64_t cost = entries + all.keys;
        const uint64_t step = std::max(room / (kPairSteps * kPairBytes), cost / kMaxSplitPoints) + 1;
        points.resize(cost / step + 1);
        const uint32_t n = (uint32_t)points.size();
        void* d;
        MZK_TRY(ctx->ensure("msm_split_points", n * sizeof(uint2), &d));
        k_part_keys<<<(n + 127) / 128, 128, 0, st>>>(all.offsets, all.keys, step, n, static_cast<uint2*>(d));
        MZK_LAUNCH_CHECK(ctx);
        MZK_CUDA_CHECK(cudaMemcpyAsync(points.data(), d, n * sizeof(uint2), cudaMemcpyDeviceToHost, st));
    } else {
        points.push_back(make_uint2(0, 0));
    }
    MZK_CUDA_CHECK(cudaMemcpyAsync(total, all.offsets + all.keys, 4, cudaMemcpyDeviceToHost, st));
    MZK_CUDA_CHECK(cudaStreamSynchronize(st));
    points.push_back(make_uint2(all.keys, *total));
    *rounds = pair_rounds(*total, all.keys, threads);
    if (*rounds) *parts = join_parts(points, *rounds, room);
    return OK;
}

// The bucket sums of all keys, by rounds of pair sums first where they pay and
// there is memory for them; the same results without.
Status accumulate(Context* ctx, const Accumulation& all, uint64_t entries, uint32_t* total, cudaStream_t st) {
    int per_sm = 0;
    MZK_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pair_sums<true>, kPairThreads, 0));
    const uint32_t blocks = (uint32_t)ctx->num_sms * (uint32_t)std::max(1, per_sm);
    const size_t threads = (size_t)blocks * kPairThreads, fixed = align256(pair_scratch_bytes(threads));
    int rounds = 0;
    std::vector<PairPart> parts;
    MZK_TRY(plan_pairs(ctx, all, entries, threads, ctx->pair_limit > fixed ? ctx->pair_limit - fixed : 0, total,
                       &rounds, &parts, st));
    size_t need = 0;
    for (const PairPart& p : parts)
        need = std::max(need, p.paired ? pair_layout(p.entries, p.k1 - p.k0, rounds).bytes
                                       : align256((size_t)(p.k1 - p.k0 + 2) * 4));
    char* mem = nullptr;
    if (!parts.empty()) mem = static_cast<char*>(ctx->pair_memory(fixed + need));
    if (!mem) {
        rounds = 0;
        parts.assign(1, {0, all.keys, 0, entries, false});
    }
    ctx->last_pair_rounds = rounds;
    ctx->last_pair_parts = mem ? (int)parts.size() : 0;
    const PairScratch scratch = mem ? pair_scratch_at(mem, threads) : PairScratch{};
    MZK_TRY(ctx->phase_begin(PH_ACCUMULATE, st));
    for (const PairPart& p : parts) {
        Accumulation a = all;
        a.keys = p.k1 - p.k0;
        a.buckets = all.buckets + p.k0;
        a.offsets = all.offsets + p.k0;
        if (p.paired) {
            const PairLayout l = pair_layout(p.entries, a.keys, rounds);
            for (int r = 0; r < rounds; r++) {
                uint32_t* off = reinterpret_cast<uint32_t*>(mem + fixed + l.offs[r & 1]);
                Affine* out = reinterpret_cast<Affine*>(mem + fixed + l.sums[r & 1]);
                MZK_TRY(scan_u32<true>(ctx, a.offsets, off, a.keys + 1, st));
                if (r == 0)
                    k_pair_sums<true><<<blocks, kPairThreads, 0, st>>>(a.bases, a.sorted, a.offsets, off, a.keys, out,
                                                                       scratch);
                else
                    k_pair_sums<false><<<blocks, kPairThreads, 0, st>>>(a.bases, nullptr, a.offsets, off, a.keys, out,
                                                                        scratch);
                MZK_LAUNCH_CHECK(ctx);
                a.offsets = off;
                a.bases = out;
            }
        } else if (mem) {
            uint32_t* off = reinterpret_cast<uint32_t*>(mem + fixed);
            k_rebase<<<(a.keys + 1 + 255) / 256, 256, 0, st>>>(a.offsets, a.keys + 1, off);
            MZK_LAUNCH_CHECK(ctx);
            a.offsets = off;
            a.sorted = all.sorted + p.first;
        }
        MZK_CUDA_CHECK(launch_accumulate(a, !p.paired, st));
        if (&p == &parts.back()) {  // one phase each per call, whatever the parts
            MZK_TRY(ctx->phase_end(st));
            MZK_TRY(ctx->phase_begin(PH_FIXUP, st));
        }
        MZK_CUDA_CHECK(launch_fixup(a, st));
        ctx->launches += 4;
    }
    return ctx->phase_end(st);
}

}  // namespace

// Window width by a cost model: W = ceil(256/c) windows of n mixed additions
// (10 Fp mul) plus 2 * 2^(c-1) full additions (14 Fp mul) for the bucket sums.
// The weights are those of an accumulation without pair sums and of running
// sums; the widths were not fitted to today's kernels.
int msm_pick_window(size_t n) {
    double best = 1e300;
    int bc = 8;
    for (int c = 6; c <= 20; c++) {
        const int w = (256 + c - 1) / c;
        const double cost = (double)w * ((double)n * 10.0 + (double)(1u << c) * 14.0 + 2048.0);
        if (cost < best) {
            best = cost;
            bc = c;
        }
    }
    return bc;
}

Status msm_g1_device(Context* ctx, const void* d_scalars, const void* d_bases, size_t n, uint64_t* out18,
                     cudaStream_t st, cudaEvent_t bases_ready) {
    const MsmPart whole{0, n, nullptr, bases_ready};
    return msm_g1_parts(ctx, d_scalars, d_bases, n, out18, st, &whole, 1);
}

// Each part is sorted and accumulated into its own bucket set, in order on
// `st`; the running-sum groups then add the bucket sets key by key.  The sort
// and accumulation scratch (counts, sorted entries, chunk partials) is shared:
// stream order finishes one part's use before the next part's writes.
Status msm_g1_parts(Context* ctx, const void* d_scalars, const void* d_bases, size_t n, uint64_t* out18,
                    cudaStream_t st, const MsmPart* parts, int n_parts) {
    std::memset(out18, 0, 18 * 8);
    if (n == 0) return OK;
    if (n >= 0x80000000ull) {
        set_error("msm: n must be < 2^31");
        return ERR_ARG;
    }
    if (n_parts < 1 || n_parts > kMaxMsmParts || parts[0].begin != 0 || parts[n_parts - 1].end != n) {
        set_error("msm: parts must cover [0, n) in 1.." + std::to_string(kMaxMsmParts) + " pieces");
        return ERR_ARG;
    }
    size_t max_part = 0;
    for (int p = 0; p < n_parts; p++) {
        if (parts[p].end <= parts[p].begin || (p > 0 && parts[p].begin != parts[p - 1].end)) {
            set_error("msm: parts must be non-empty and contiguous");
            return ERR_ARG;
        }
        max_part = std::max(max_part, parts[p].end - parts[p].begin);
    }
    const int c = msm_window_for(ctx, n);
    if (c < 5 || c > 24) {
        set_error("msm: window width must be in [5, 24]");
        return ERR_ARG;
    }
    const MsmShape sh = make_shape(c);
    const size_t entries_cap = (size_t)sh.windows * max_part;
    if (entries_cap >= 0xffffffffull) {
        set_error("msm: n * windows exceeds 2^32 entries");
        return ERR_ARG;
    }
    // accumulate grid: persistent, sized to fill the GPU once
    int acc_blocks_per_sm = 0;
    MZK_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&acc_blocks_per_sm, k_accumulate<true>, kAccThreads, 0));
    if (acc_blocks_per_sm < 1) acc_blocks_per_sm = 1;
    const uint32_t acc_blocks = (uint32_t)(ctx->num_sms * acc_blocks_per_sm);
    const uint32_t acc_threads = acc_blocks * kAccThreads;
    const uint32_t quad_blocks = accumulate_quad_blocks(ctx, entries_cap);

    void *counts, *sorted, *partials, *queue, *arena, *wsum;
    void *offsets[kMaxMsmParts] = {}, *buckets[kMaxMsmParts] = {};
    static const char* const kOffsetNames[kMaxMsmParts] = {"msm_offsets", "msm_offsets2", "msm_offsets3",
                                                            "msm_offsets4"};
    static const char* const kBucketNames[kMaxMsmParts] = {"msm_buckets", "msm_buckets2", "msm_buckets3",
                                                            "msm_buckets4"};
    MZK_TRY(ctx->ensure("msm_counts", ((size_t)sh.keys + 1) * 4, &counts));
    for (int p = 0; p < n_parts; p++) {
        MZK_TRY(ctx->ensure(kOffsetNames[p], ((size_t)sh.keys + 2) * 4, &offsets[p]));
        MZK_TRY(ctx->ensure(kBucketNames[p], (size_t)sh.keys * sizeof(Xyzz), &buckets[p]));
    }
    MZK_TRY(ctx->ensure("msm_sorted", entries_cap * 4, &sorted));
    void* digits;
    MZK_TRY(ctx->ensure("msm_digits", entries_cap * 4, &digits));
    MZK_TRY(ctx->ensure("msm_partials", (size_t)acc_threads * 2 * sizeof(Xyzz), &partials));
    MZK_TRY(ctx->ensure("msm_queue", queue_bytes(acc_threads), &queue));
    std::vector<Window> wins;
    append_windows(sh, 0, sh.windows, wins);
    const ReducePlan plan = plan_reduce(wins, reduce_group_log(sh.keys, (uint32_t)n_parts));
    void* d_tab;
    MZK_TRY(ctx->ensure("msm_wins", plan.table_bytes(), &d_tab));
    MZK_TRY(ctx->ensure("msm_arena", plan.arena * sizeof(Xyzz), &arena));
    MZK_TRY(ctx->ensure("msm_wsum", (size_t)sh.windows * sizeof(Xyzz), &wsum));
    // pinned staging: window sums and the parts' entry counts (read back),
    // then the reduction's tables (uploaded without the sync a pageable copy implies)
    void* host_wsum;
    const size_t tab_off = (size_t)sh.windows * sizeof(Xyzz) + 64;
    MZK_TRY(ctx->ensure_pinned(tab_off + plan.table_bytes(), &host_wsum));
    void* host_tab = static_cast<char*>(host_wsum) + tab_off;
    plan.pack(host_tab);
    uint32_t* host_entries =
        reinterpret_cast<uint32_t*>(static_cast<char*>(host_wsum) + (size_t)sh.windows * sizeof(Xyzz));

    const Fr* sc = static_cast<const Fr*>(d_scalars);
    const Affine* ba = static_cast<const Affine*>(d_bases);
    const int pt_threads = 256;

    MZK_CUDA_CHECK(cudaMemcpyAsync(d_tab, host_tab, plan.table_bytes(), cudaMemcpyHostToDevice, st));
    for (int p = 0; p < n_parts; p++) {
        const MsmPart& part = parts[p];
        const size_t np = part.end - part.begin;
        uint32_t* off = static_cast<uint32_t*>(offsets[p]);
        const uint32_t pt_blocks =
            (uint32_t)std::min<size_t>((np + pt_threads - 1) / pt_threads, (size_t)ctx->num_sms * 16);
        if (part.scalars_ready) MZK_CUDA_CHECK(cudaStreamWaitEvent(st, part.scalars_ready, 0));
        MZK_TRY(ctx->phase_begin(PH_HISTOGRAM, st));
        MZK_CUDA_CHECK(cudaMemsetAsync(counts, 0, ((size_t)sh.keys + 1) * 4, st));
        k_histogram<<<pt_blocks, pt_threads, 0, st>>>(sc + part.begin, np, sh.c, sh.windows, sh.nb,
                                                      (uint32_t*)counts, (uint32_t*)digits);
        MZK_LAUNCH_CHECK(ctx);
        MZK_TRY(ctx->phase_end(st));
        MZK_TRY(ctx->phase_begin(PH_SCAN, st));
        // exclusive scan one place to the right: off[key + 1] = start of key
        MZK_CUDA_CHECK(cudaMemsetAsync(off, 0, 4, st));
        MZK_TRY(scan_u32(ctx, (const uint32_t*)counts, off + 1, sh.keys + 1, st));
        MZK_TRY(ctx->phase_end(st));
        MZK_TRY(ctx->phase_begin(PH_SCATTER, st));
        const uint32_t together = scatter_together((size_t)sh.windows, np);
        for (uint32_t w = 0; w < (uint32_t)sh.windows; w += together) {
            const dim3 grid(pt_blocks, std::min(together, (uint32_t)sh.windows - w));
            k_scatter_window<<<grid, pt_threads, 0, st>>>((const uint32_t*)digits, np, w, off + 1, (uint32_t*)sorted);
            MZK_LAUNCH_CHECK(ctx);
        }
        MZK_TRY(ctx->phase_end(st));
        if (part.bases_ready) MZK_CUDA_CHECK(cudaStreamWaitEvent(st, part.bases_ready, 0));
        const Accumulation acc{ba + part.begin, (const uint32_t*)sorted, off, sh.keys, (Xyzz*)buckets[p],
                               (Xyzz*)partials, queue, acc_blocks, quad_blocks, (uint32_t)ctx->num_sms * 2};
        MZK_TRY(accumulate(ctx, acc, (uint64_t)sh.windows * np, host_entries + p, st));
        MZK_CUDA_CHECK(cudaMemcpyAsync(host_entries + p, off + sh.keys, 4, cudaMemcpyDeviceToHost, st));
    }
    MZK_TRY(ctx->phase_begin(PH_REDUCE, st));
    BucketSets sets{};
    sets.n = (uint32_t)n_parts;
    for (int p = 0; p < n_parts; p++) {
        sets.buckets[p] = (const Xyzz*)buckets[p];
        sets.offsets[p] = (const uint32_t*)offsets[p];
    }
    MZK_CUDA_CHECK(launch_reduce(plan, sets, d_tab, (Xyzz*)arena, (Xyzz*)wsum, &ctx->launches, st));
    MZK_TRY(ctx->phase_end(st));
    MZK_CUDA_CHECK(cudaMemcpyAsync(host_wsum, wsum, (size_t)sh.windows * sizeof(Xyzz), cudaMemcpyDeviceToHost, st));
    MZK_CUDA_CHECK(cudaStreamSynchronize(st));
    ctx->phase_collect();
    ctx->last_c = sh.c;
    ctx->last_windows = sh.windows;
    ctx->last_entries = 0;
    for (int p = 0; p < n_parts; p++) ctx->last_entries += host_entries[p];

    // host: sum_w 2^(c w) S_w by Horner, then normalise
    const host::Xyzz6* hs = static_cast<const host::Xyzz6*>(host_wsum);
    host::combine_windows(hs, sh.windows, sh.c, out18);
    return OK;
}

}  // namespace mzk

namespace mzk {

// ---------------------------------------------------------------------------
// Batched MSMs over one shared device SRS.
//
// Many MSMs (a proof's commitments, or many proofs' commitments) run as one
// MSM of MSMs: every item keeps its own window width, its keys are laid out
// back to back in one key space, so ONE counting sort orders all entries and
// ONE accumulate launch balances the work of all items across the GPU (an
// item of 2^12 points and one of 2^22 share the same chunks).  Only the final
// combination of each item's window sums is per item.  Bases of item m are
// bases[base_offset_m .. base_offset_m + n_m), like commit_many's
// `bases[..size]` prefix of the SRS (proofs/src/poly/kzg/mod.rs:98-103).
// ---------------------------------------------------------------------------
namespace {

struct BatchItemDev {
    const Fr* scalars;
    uint32_t n, point_start, base_offset;
    uint32_t c, windows, nb, key_start;
    uint32_t fixed;  // 1: the windows share one bucket set, window w reads table row w
};

__device__ __forceinline__ uint32_t find_item(const BatchItemDev* items, uint32_t n_items, uint32_t p) {
    uint32_t lo = 0, hi = n_items;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (items[mid].point_start <= p) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Counts per key of every item's digits, and every point's digit per window,
// window-major (digits[w * total_points + p] = key | sign << 31, kNoKey for a
// zero digit or a window past the item's), for the window-by-window scatter.
__global__ void k_digits_batch(const BatchItemDev* __restrict__ items, uint32_t n_items, uint32_t total_points,
                               int max_windows, uint32_t* __restrict__ counts, uint32_t* __restrict__ digits) {
    const uint32_t stride = gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (uint32_t base = blockIdx.x * blockDim.x; base < total_points; base += stride) {
        const uint32_t p = base + threadIdx.x;
        const bool valid = p < total_points;
        BatchItemDev it = items[valid ? find_item(items, n_items, p) : 0];
        const uint32_t local = p - it.point_start;
        Fr s = valid ? fr_from_mont(load_fr(it.scalars, local)) : fr_zero();
        uint32_t carry = 0;
        for (int w = 0; w < max_windows; w++) {
            bool neg = false;
            uint32_t key = kNoKey;
            if (valid && w < (int)it.windows) {
                key = next_digit(s, w, (int)it.c, it.nb, carry, neg);
                if (key != kNoKey) key += it.key_start - (it.fixed ? (uint32_t)w * it.nb : 0u);
            }
            const uint32_t peers = __match_any_sync(0xffffffffu, key);
            if (key != kNoKey && lane == __ffs(peers) - 1) atomicAdd(&counts[key], (uint32_t)__popc(peers));
            if (valid) digits[(size_t)w * total_points + p] = key == kNoKey ? kNoKey : key | (neg ? 0x80000000u : 0u);
        }
    }
}


// The batch scatter of window w of every item from the stored digits: the
// entries land in the items' window-w slices (4 bytes per point of the batch),
// which stay in L2 while the window is scattered.
// table_stride: points per table row (fixed items read window w from row w)
__global__ void k_scatter_window_batch(const uint32_t* __restrict__ digits, const BatchItemDev* __restrict__ items,
                                       uint32_t n_items, uint32_t total_points, uint32_t w0, uint32_t table_stride,
                                       uint32_t* __restrict__ cursor, uint32_t* __restrict__ sorted) {
    const uint32_t w = w0 + blockIdx.y, row_off = w * table_stride;
    const uint32_t* __restrict__ digits_w = digits + (size_t)w * total_points;
    const uint32_t stride = gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    for (uint32_t base = blockIdx.x * blockDim.x; base < total_points; base += stride) {
        const uint32_t p = base + threadIdx.x;
        const uint32_t d = p < total_points ? __ldg(digits_w + p) : kNoKey;
        const uint32_t key = d == kNoKey ? kNoKey : d & 0x7fffffffu;
        const uint32_t peers = __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(peers) - 1;
        uint32_t slot = 0;
        if (key != kNoKey && lane == leader) slot = atomicAdd(&cursor[key], (uint32_t)__popc(peers));
        slot = __shfl_sync(0xffffffffu, slot, leader);
        if (key != kNoKey) {
            const BatchItemDev& it = items[find_item(items, n_items, p)];
            const uint32_t point = it.base_offset + (p - it.point_start) + (it.fixed ? row_off : 0u);
            sorted[slot + (uint32_t)__popc(peers & lt_mask)] = point | (d & 0x80000000u);
        }
    }
}
}  // namespace

namespace {
// row j+1 of a window table from row j: [2^c] P, normalised
__global__ void __launch_bounds__(256) k_window_row(const Affine* __restrict__ prev, Affine* __restrict__ next,
                                                    uint64_t n, int c) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        Xyzz p = xyzz_from_affine(prev[i]);
        for (int b = 0; b < c; b++) p = xyzz_dbl(p);
        next[i] = xyzz_to_affine(p);
    }
}
}  // namespace

uint32_t msm_table_rows(int c) { return (uint32_t)make_shape(c).windows; }

Status msm_window_table(Context* ctx, void* d_table, uint64_t len, int c, uint32_t rows, cudaStream_t st) {
    if (c < 5 || c > 24 || rows < msm_table_rows(c) || len == 0 || (uint64_t)rows * len >= 0x80000000ull) {
        set_error("window table: c in [5, 24], at least msm_table_rows(c) rows, rows x len < 2^31");
        return ERR_ARG;
    }
    Affine* t = static_cast<Affine*>(d_table);
    const uint32_t blocks = (uint32_t)std::min<uint64_t>((len + 255) / 256, (uint64_t)ctx->num_sms * 8);
    for (uint32_t j = 1; j < rows; j++) {
        k_window_row<<<blocks, 256, 0, st>>>(t + (j - 1) * len, t + j * len, len, c);
        MZK_LAUNCH_CHECK(ctx);
    }
    return OK;
}

Status msm_g1_batch_device(Context* ctx, const void* d_bases, size_t bases_len, const BatchItem* items, size_t count,
                           uint64_t* out, cudaStream_t st, const MsmTable* table) {
    if (table) {
        if (table->d_table != d_bases || table->stride != bases_len || table->rows < msm_table_rows(table->c) ||
            table->rows * table->stride >= 0x80000000ull) {
            set_error("msm batch: the window table must start at the bases and cover the windows of its width");
            return ERR_ARG;
        }
    }
    std::memset(out, 0, count * 18 * 8);
    std::vector<BatchItemDev> hi;
    std::vector<Window> hw;
    std::vector<size_t> item_of;  // position in `items` of every device item
    uint64_t points = 0, keys = 0, entries = 0;
    int max_windows = 0;
    auto uses_table = [&](uint64_t n) { return table && n >= table->min_n; };
    for (size_t m = 0; m < count; m++) {
        const BatchItem& it = items[m];
        if (it.n == 0) continue;
        if (!it.d_scalars) {
            set_error("msm batch: null scalars in item " + std::to_string(m));
            return ERR_ARG;
        }
        if (it.base_offset + it.n > bases_len || it.base_offset + it.n >= 0x80000000ull) {
            set_error("msm batch: item " + std::to_string(m) + " reads past the bases");
            return ERR_ARG;
        }
        const bool fixed = uses_table(it.n);
        const int c = fixed ? table->c : msm_window_for(ctx, it.n);
        const MsmShape sh = make_shape(c);
        BatchItemDev d;
        d.scalars = static_cast<const Fr*>(it.d_scalars);
        d.n = (uint32_t)it.n;
        d.point_start = (uint32_t)points;
        d.base_offset = (uint32_t)it.base_offset;
        d.c = (uint32_t)sh.c;
        d.windows = (uint32_t)sh.windows;
        d.nb = sh.nb;
        d.key_start = (uint32_t)keys;
        d.fixed = fixed ? 1u : 0u;
        // fixed: one bucket set, every window's digits land in the same buckets
        append_windows(sh, keys, fixed ? 1 : sh.windows, hw);
        keys += fixed ? sh.nb : sh.keys;
        points += it.n;
        entries += (uint64_t)sh.windows * it.n;
        max_windows = std::max(max_windows, sh.windows);
        hi.push_back(d);
        item_of.push_back(m);
    }
    if (hi.empty()) return OK;
    if (points >= 0xffffffffull || keys >= 0xffffffffull || entries >= 0xffffffffull) {
        set_error("msm batch: more than 2^32 points, keys or entries");
        return ERR_ARG;
    }
    int acc_blocks_per_sm = 0;
    MZK_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&acc_blocks_per_sm, k_accumulate<true>, kAccThreads, 0));
    if (acc_blocks_per_sm < 1) acc_blocks_per_sm = 1;
    const uint32_t acc_blocks = (uint32_t)(ctx->num_sms * acc_blocks_per_sm);
    const uint32_t acc_threads = acc_blocks * kAccThreads;
    const uint32_t quad_blocks = accumulate_quad_blocks(ctx, entries);
    const size_t n_wins = hw.size();
    const ReducePlan plan = plan_reduce(hw, reduce_group_log(keys, 1));
    void *d_items, *d_tab, *counts, *offsets, *sorted, *buckets, *partials, *queue, *arena, *wsum;
    MZK_TRY(ctx->ensure("batch_items", hi.size() * sizeof(BatchItemDev), &d_items));
    MZK_TRY(ctx->ensure("batch_wins", plan.table_bytes(), &d_tab));
    MZK_TRY(ctx->ensure("msm_counts", (keys + 1) * 4, &counts));
    MZK_TRY(ctx->ensure("msm_offsets", (keys + 2) * 4, &offsets));
    MZK_TRY(ctx->ensure("msm_sorted", entries * 4, &sorted));
    void* digits;
    MZK_TRY(ctx->ensure("msm_digits", (size_t)max_windows * points * 4, &digits));
    MZK_TRY(ctx->ensure("msm_buckets", keys * sizeof(Xyzz), &buckets));
    MZK_TRY(ctx->ensure("msm_partials", (size_t)acc_threads * 2 * sizeof(Xyzz), &partials));
    MZK_TRY(ctx->ensure("msm_queue", queue_bytes(acc_threads), &queue));
    MZK_TRY(ctx->ensure("msm_arena", plan.arena * sizeof(Xyzz), &arena));
    MZK_TRY(ctx->ensure("msm_wsum", n_wins * sizeof(Xyzz), &wsum));
    // pinned staging: window sums (read back), then the item table and the reduction's tables
    void* host_wsum;
    const size_t items_off = n_wins * sizeof(Xyzz) + 64;
    const size_t wins_off = items_off + ((hi.size() * sizeof(BatchItemDev) + 255) & ~(size_t)255);
    MZK_TRY(ctx->ensure_pinned(wins_off + plan.table_bytes(), &host_wsum));
    char* staging = static_cast<char*>(host_wsum);
    std::memcpy(staging + items_off, hi.data(), hi.size() * sizeof(BatchItemDev));
    plan.pack(staging + wins_off);
    MZK_CUDA_CHECK(cudaMemcpyAsync(d_items, staging + items_off, hi.size() * sizeof(BatchItemDev),
                                   cudaMemcpyHostToDevice, st));
    MZK_CUDA_CHECK(cudaMemcpyAsync(d_tab, staging + wins_off, plan.table_bytes(), cudaMemcpyHostToDevice, st));

    const uint32_t n_items = (uint32_t)hi.size();
    const int pt_threads = 256;
    const uint32_t pt_blocks =
        (uint32_t)std::min<uint64_t>((points + pt_threads - 1) / pt_threads, (uint64_t)ctx->num_sms * 16);
    MZK_TRY(ctx->phase_begin(PH_HISTOGRAM, st));
    MZK_CUDA_CHECK(cudaMemsetAsync(counts, 0, (keys + 1) * 4, st));
    k_digits_batch<<<pt_blocks, pt_threads, 0, st>>>((const BatchItemDev*)d_items, n_items, (uint32_t)points,
                                                    max_windows, (uint32_t*)counts, (uint32_t*)digits);
    MZK_LAUNCH_CHECK(ctx);
    MZK_TRY(ctx->phase_end(st));
    MZK_TRY(ctx->phase_begin(PH_SCAN, st));
    MZK_CUDA_CHECK(cudaMemsetAsync(offsets, 0, 4, st));
    MZK_TRY(scan_u32(ctx, (const uint32_t*)counts, (uint32_t*)offsets + 1, (uint32_t)keys + 1, st));
    MZK_TRY(ctx->phase_end(st));
    MZK_TRY(ctx->phase_begin(PH_SCATTER, st));
    const uint32_t together = scatter_together((size_t)max_windows, points);
    for (uint32_t w = 0; w < (uint32_t)max_windows; w += together) {
        const dim3 grid(pt_blocks, std::min(together, (uint32_t)max_windows - w));
        k_scatter_window_batch<<<grid, pt_threads, 0, st>>>((const uint32_t*)digits, (const BatchItemDev*)d_items,
                                                            n_items, (uint32_t)points, w,
                                                            table ? (uint32_t)table->stride : 0u,
                                                            (uint32_t*)offsets + 1, (uint32_t*)sorted);
        MZK_LAUNCH_CHECK(ctx);
    }
    MZK_TRY(ctx->phase_end(st));
    const Accumulation acc{static_cast<const Affine*>(d_bases), (const uint32_t*)sorted, (const uint32_t*)offsets,
                           (uint32_t)keys, (Xyzz*)buckets, (Xyzz*)partials, queue, acc_blocks, quad_blocks,
                           (uint32_t)ctx->num_sms * 2};
    MZK_TRY(accumulate(ctx, acc, entries, static_cast<uint32_t*>(host_wsum), st));
    MZK_TRY(ctx->phase_begin(PH_REDUCE, st));
    const BucketSets sets{{(const Xyzz*)buckets}, {(const uint32_t*)offsets}, 1};
    MZK_CUDA_CHECK(launch_reduce(plan, sets, d_tab, (Xyzz*)arena, (Xyzz*)wsum, &ctx->launches, st));
    MZK_TRY(ctx->phase_end(st));
    MZK_CUDA_CHECK(cudaMemcpyAsync(host_wsum, wsum, n_wins * sizeof(Xyzz), cudaMemcpyDeviceToHost, st));
    MZK_CUDA_CHECK(cudaStreamSynchronize(st));
    ctx->phase_collect();
    // host: per item sum_w 2^(c w) S_w by Horner and one inversion (~0.15 ms
    // each, a serial chain of ~250 doublings); items are independent, so a
    // batch spreads them over host threads
    const host::Xyzz6* hs = static_cast<const host::Xyzz6*>(host_wsum);
    std::vector<size_t> first_win(hi.size());
    for (size_t i = 0, w0 = 0; i < hi.size(); w0 += hi[i].fixed ? 1 : hi[i].windows, i++) first_win[i] = w0;
    auto tail = [&](size_t i) {
        // fixed: one window, the table rows already carry the 2^(c w) factors
        host::combine_windows(hs + first_win[i], hi[i].fixed ? 1 : (int)hi[i].windows, (int)hi[i].c,
                              out + 18 * item_of[i]);
    };
    const size_t cores = std::max(1u, std::thread::hardware_concurrency());
    const size_t nthreads = std::min<size_t>({hi.size() / 2, cores / 2, 32});
    if (nthreads <= 1) {
        for (size_t i = 0; i < hi.size(); i++) tail(i);
    } else {
        std::atomic<size_t> next{0};
        auto worker = [&] {
            for (size_t i; (i = next.fetch_add(1)) < hi.size();) tail(i);
        };
        std::vector<std::thread> pool;
        for (size_t t = 1; t < nthreads; t++) pool.emplace_back(worker);
        worker();
        for (std::thread& th : pool) th.join();
    }
    ctx->last_entries = entries;
    return OK;
}

}  // namespace mzk

namespace mzk {

// ---------------------------------------------------------------------------
// Allocation-free MSM for callers that cannot allocate device memory.
//
// Some hosts own every byte of device memory themselves: a framework that
// hands a custom operation its input and output buffers but no workspace, a
// runtime whose memory pool must not be bypassed, or code running where the
// CUDA allocator may not be called.  For them the MSM below takes its scratch
// from one file-scope device array of fixed size instead of cudaMalloc.  It
// serves n <= kNoAllocMaxN points with the window width clamped to [8, 12].
// Every GPU that loads this library holds the array (about 21 MB) until the
// process exits.
// ---------------------------------------------------------------------------
namespace {

constexpr size_t kNoAllocMaxN = size_t(1) << 16;
constexpr int kNoAllocMinC = 8, kNoAllocMaxC = 12;
constexpr uint32_t kNoAllocAccBlocks = 64;  // fixed accumulate grid (64 x 128 threads)
constexpr int kNoAllocMaxDevices = 64;

// largest key count over the allowed widths: c = 12 gives 22 windows x 2048
constexpr size_t kNaKeys = 22 * 2048;
constexpr size_t kNaMaxWindows = 32;  // c = 8
constexpr size_t kNaAccThreads = (size_t)kNoAllocAccBlocks * kAccThreads;
constexpr size_t kNaCountsOff = 0;
constexpr size_t kNaOffsetsOff = kNaCountsOff + align256((kNaKeys + 1) * 4);
constexpr size_t kNaSortedOff = kNaOffsetsOff + align256((kNaKeys + 2) * 4);
constexpr size_t kNaBucketsOff = kNaSortedOff + align256(kNaMaxWindows * kNoAllocMaxN * 4);
constexpr size_t kNaPartialsOff = kNaBucketsOff + align256(kNaKeys * sizeof(Xyzz));
constexpr size_t kNaQueueOff = kNaPartialsOff + align256(kNaAccThreads * 2 * sizeof(Xyzz));
constexpr size_t kNaArenaOff = kNaQueueOff + align256(queue_bytes(kNaAccThreads));
// the reduction tree's values: a node of the first launch's 2^7 buckets (every
// window has as many) leaves 8 values, and up to 16 of those nodes per window
// leave one of at most 12
constexpr size_t kNaArenaPoints = (kNaKeys >> kTreeFirst) * (kTreeFirst + 1) + kNaMaxWindows * 12;
static_assert(kNoAllocMinC - 1 >= (int)kTreeFirst && kNoAllocMaxC - 1 <= (int)kTreeFirst + 4, "two launches of the tree");
constexpr size_t kNaTabBytes = kNaMaxWindows * (4 * sizeof(TreeWin) + sizeof(FinWin));
constexpr size_t kNaWsumOff = kNaArenaOff + align256(kNaArenaPoints * sizeof(Xyzz));
constexpr size_t kNaScanOff = kNaWsumOff + align256(kNaMaxWindows * sizeof(Xyzz));
constexpr size_t kNaWinsOff = kNaScanOff + align256(64 * 4);
constexpr size_t kNaBytes = kNaWinsOff + align256(kNaTabBytes);

// The scratch itself.  Host code must not use this name as a device address:
// on the host it is only a stand-in, so kernels get the pointer obtained from
// cudaGetSymbolAddress below.
__device__ __align__(256) unsigned char g_msm_noalloc_scratch[kNaBytes];

// one lock per device: each device has its own copy of the array
std::mutex g_noalloc_mu[kNoAllocMaxDevices];
void* g_noalloc_ptr[kNoAllocMaxDevices] = {};
int g_noalloc_sms[kNoAllocMaxDevices] = {};

// exclusive scan into caller-provided tile sums (no allocation)
Status scan_u32_noalloc(const uint32_t* in, uint32_t* out, uint32_t len, uint32_t* sums, cudaStream_t st) {
    const uint32_t tiles = (len + kScanTile - 1) / kScanTile;
    k_scan_tiles<false><<<tiles, kScanThreads, 0, st>>>(in, out, len, sums);
    MZK_CUDA_CHECK(cudaGetLastError());
    k_scan_sums<<<1, kScanThreads, 0, st>>>(sums, tiles);
    MZK_CUDA_CHECK(cudaGetLastError());
    k_scan_add<<<tiles, kScanThreads, 0, st>>>(out, len, sums);
    MZK_CUDA_CHECK(cudaGetLastError());
    return OK;
}

Status msm_g1_noalloc_queued(unsigned char* base, int sms, const void* d_scalars, const void* d_bases, size_t n,
                             uint64_t* out18, cudaStream_t st);

Status msm_g1_noalloc(const void* d_scalars, const void* d_bases, size_t n, uint64_t* out18, cudaStream_t st) {
    std::memset(out18, 0, 18 * 8);
    if (n > kNoAllocMaxN) {
        set_error("mzk_msm_g1_noalloc: n = " + std::to_string(n) + " exceeds the fixed scratch limit of " +
                  std::to_string(kNoAllocMaxN) + " points; use mzk_msm_g1_device");
        return ERR_ARG;
    }
    if (n == 0) return OK;
    int dev = 0;
    MZK_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) {
        set_error("mzk_msm_g1_noalloc: device index out of range");
        return ERR_ARG;
    }
    // one lock for this device's array: calls from several host threads take turns
    std::lock_guard<std::mutex> lock(g_noalloc_mu[dev]);
    if (!g_noalloc_ptr[dev]) {
        // set-up, once per device, with that device current
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_msm_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            set_error(std::string("mzk_msm_g1_noalloc: cudaGetSymbolAddress failed: ") + cudaGetErrorString(e));
            return ERR_CUDA;
        }
        int sms = 0;
        MZK_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        g_noalloc_sms[dev] = sms;
        g_noalloc_ptr[dev] = p;
    }
    const Status s = msm_g1_noalloc_queued(static_cast<unsigned char*>(g_noalloc_ptr[dev]), g_noalloc_sms[dev],
                                           d_scalars, d_bases, n, out18, st);
    // a failure after work was queued: let that work finish before the lock
    // is released, so the next call cannot race with it on the array
    if (s != OK) cudaStreamSynchronize(st);
    return s;
}

Status msm_g1_noalloc_queued(unsigned char* base, int sms, const void* d_scalars, const void* d_bases, size_t n,
                             uint64_t* out18, cudaStream_t st) {
    int c = msm_pick_window(n);
    c = c < kNoAllocMinC ? kNoAllocMinC : (c > kNoAllocMaxC ? kNoAllocMaxC : c);
    const MsmShape sh = make_shape(c);
    uint32_t* counts = reinterpret_cast<uint32_t*>(base + kNaCountsOff);
    uint32_t* offsets = reinterpret_cast<uint32_t*>(base + kNaOffsetsOff);
    uint32_t* sorted = reinterpret_cast<uint32_t*>(base + kNaSortedOff);
    Xyzz* buckets = reinterpret_cast<Xyzz*>(base + kNaBucketsOff);
    Xyzz* partials = reinterpret_cast<Xyzz*>(base + kNaPartialsOff);
    void* queue = base + kNaQueueOff;
    Xyzz* arena = reinterpret_cast<Xyzz*>(base + kNaArenaOff);
    Xyzz* wsum = reinterpret_cast<Xyzz*>(base + kNaWsumOff);
    uint32_t* scan_sums = reinterpret_cast<uint32_t*>(base + kNaScanOff);

    const Fr* sc = static_cast<const Fr*>(d_scalars);
    const Affine* ba = static_cast<const Affine*>(d_bases);
    const int pt_threads = 256;
    const uint32_t pt_blocks =
        (uint32_t)std::min<size_t>((n + pt_threads - 1) / pt_threads, (size_t)sms * 16);
    // the array keeps the previous call's contents: zero the counters
    MZK_CUDA_CHECK(cudaMemsetAsync(counts, 0, ((size_t)sh.keys + 1) * 4, st));
    k_histogram<<<pt_blocks, pt_threads, 0, st>>>(sc, n, sh.c, sh.windows, sh.nb, counts, nullptr);
    MZK_CUDA_CHECK(cudaGetLastError());
    MZK_CUDA_CHECK(cudaMemsetAsync(offsets, 0, 4, st));
    MZK_TRY(scan_u32_noalloc(counts, offsets + 1, sh.keys + 1, scan_sums, st));
    k_scatter<<<pt_blocks, pt_threads, 0, st>>>(sc, n, sh.c, sh.windows, sh.nb, offsets + 1, sorted);
    MZK_CUDA_CHECK(cudaGetLastError());
    // (by lanes: the fixed grid of 64 blocks holds 2048 quads only)
    const Accumulation job{ba,       sorted, offsets, sh.keys, buckets, partials, queue, kNoAllocAccBlocks, 0,
                           kNoAllocAccBlocks};
    MZK_CUDA_CHECK(launch_accumulate(job, true, st));
    MZK_CUDA_CHECK(launch_fixup(job, st));
    // the reduction's tables (a copy from pageable memory is staged before the call returns)
    std::vector<Window> wins;
    append_windows(sh, 0, sh.windows, wins);
    const ReducePlan plan = plan_reduce(wins, 0);
    if (plan.arena > kNaArenaPoints || plan.table_bytes() > kNaTabBytes) {
        set_error("mzk_msm_g1_noalloc: the reduction does not fit the fixed scratch");
        return ERR_STATE;
    }
    unsigned char tab[kNaTabBytes];
    plan.pack(tab);
    MZK_CUDA_CHECK(cudaMemcpyAsync(base + kNaWinsOff, tab, plan.table_bytes(), cudaMemcpyHostToDevice, st));
    const BucketSets sets{{buckets}, {offsets}, 1};
    MZK_CUDA_CHECK(launch_reduce(plan, sets, base + kNaWinsOff, arena, wsum, nullptr, st));
    // window sums to host memory owned by this function (no pinned allocation)
    host::Xyzz6 hs[kNaMaxWindows];
    MZK_CUDA_CHECK(cudaMemcpyAsync(hs, wsum, (size_t)sh.windows * sizeof(Xyzz), cudaMemcpyDeviceToHost, st));
    MZK_CUDA_CHECK(cudaStreamSynchronize(st));
    host::combine_windows(hs, sh.windows, sh.c, out18);
    return OK;
}

}  // namespace

}  // namespace mzk

extern "C" int mzk_msm_g1_noalloc(const uint64_t* d_scalars, const uint64_t* d_bases, size_t n, uint64_t out[18],
                                  void* stream) {
    if (!out || (n && (!d_scalars || !d_bases))) {
        mzk::set_error("mzk_msm_g1_noalloc: null pointer");
        return mzk::ERR_ARG;
    }
    return mzk::msm_g1_noalloc(d_scalars, d_bases, n, out, static_cast<cudaStream_t>(stream));
}
