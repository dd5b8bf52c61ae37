// grand.cu — the prover stages around the commitments that are scans over a
// column rather than MSMs or NTTs:
//
//   * batch inversion with ff 0.13 BatchInvert semantics (zeros stay zero),
//     used by both arguments below;
//   * the permutation argument's grand products z of every set
//     (proofs/src/plonk/permutation/prover.rs:81-255);
//   * the logup argument's helper polynomials and running-sum aggregator
//     (proofs/src/plonk/logup/prover.rs:195-300);
//   * eval_polynomial (proofs/src/utils/arithmetic.rs:59-87) and
//     kate_division (arithmetic.rs:106-125), both first-order linear
//     recurrences y_i = c_i + k y_{i+1} solved by one chunked primitive.
//
// Every result is an exact field value, so the parallel orders here give the
// reference's bytes.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/mzk.h"
#include "field.cuh"
#include "grand.hpp"
#include "host_ec.hpp"
#include "inv.cuh"
#include "ntt.hpp"
#include "runtime.hpp"

namespace mzk {

namespace {

constexpr int kThreads = 256;
// elements per thread of a block scan: two serial chains of as many products,
// so fewer where the tiles do not fill the GPU
constexpr uint32_t kScanItemsMin = 2, kScanItemsMax = 8;
constexpr uint32_t kMaxPermSetCols = 8;
constexpr uint32_t kMaxLogupChunks = 8;

__device__ __forceinline__ bool fr_is_zero(const Fr& a) {
    uint32_t acc = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) acc |= a.l[j];
    return acc == 0;
}

Fr to_dev(const host::Fr4& h) {
    Fr r;
    std::memcpy(r.l, h.l, 32);
    return r;
}
host::Fr4 to_host(const uint64_t* p) {
    host::Fr4 r;
    std::memcpy(r.l, p, 32);
    return r;
}

uint32_t grid_for(const Context* ctx, uint64_t items, uint32_t threads) {
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((items + threads - 1) / threads, (uint64_t)ctx->num_sms * 16));
}

// ---- exclusive scans (product or sum) of Fr values ----
template <bool kMul>
__device__ __forceinline__ Fr op(const Fr& a, const Fr& b) {
    return kMul ? fr_mul(a, b) : fr_add(a, b);
}
template <bool kMul>
__device__ __forceinline__ Fr identity() {
    return kMul ? fr_one() : fr_zero();
}

// block-wide exclusive scan of one value per thread (Hillis-Steele in shared
// memory); returns the exclusive prefix, *total the block's total
template <bool kMul>
__device__ Fr block_exclusive(Fr v, Fr* sm, Fr* total) {
    sm[threadIdx.x] = v;
    __syncthreads();
    for (uint32_t off = 1; off < blockDim.x; off <<= 1) {
        Fr o = identity<kMul>();
        if (threadIdx.x >= off) o = sm[threadIdx.x - off];
        __syncthreads();
        if (threadIdx.x >= off) sm[threadIdx.x] = op<kMul>(o, sm[threadIdx.x]);
        __syncthreads();
    }
    *total = sm[blockDim.x - 1];
    const Fr ex = threadIdx.x ? sm[threadIdx.x - 1] : identity<kMul>();
    __syncthreads();
    return ex;
}

// ---- batch inversion (ff BatchInvert: zeros stay zero) ----
//
// A thread multiplies C elements (one from each of C rows of gridDim x
// blockDim, so that loads and stores are coalesced), inverts the product and
// works backward; zeros are left out.  The inversion (inv_divsteps) takes a warp
// the same time for 1 value as for 32, 17 us alone on its scheduler and ~13 us
// for each warp where there are several, so every thread has its own and
// nothing is exchanged: one inversion per block between two scans over its
// threads took 52 us for 2^16 elements and 94 for 2^18.  C weighs the inversions
// against the chain of 3 C products (0.3..0.5 us each): up to 8 keeps the
// elements in registers, 16 reads them twice.
constexpr int kInvThreads = 128;

template <int C>
__global__ void __launch_bounds__(kInvThreads, C > 8 ? 4 : 3) k_batch_invert(Fr* __restrict__ a, uint64_t n) {
    constexpr bool kKeep = C <= 8;
    const uint64_t row = (uint64_t)gridDim.x * kInvThreads, first = (uint64_t)blockIdx.x * kInvThreads + threadIdx.x;
    Fr pre[C], kept[kKeep ? C : 1];
    if (kKeep) {
#pragma unroll
        for (int k = 0; k < C; k++) {
            const uint64_t i = first + (uint64_t)k * row;
            kept[kKeep ? k : 0] = i < n ? a[i] : fr_zero();
        }
    }
    auto element = [&](int k) {
        if (kKeep) return kept[kKeep ? k : 0];
        const uint64_t i = first + (uint64_t)k * row;
        return i < n ? a[i] : fr_zero();
    };
    Fr acc = fr_one();
#pragma unroll
    for (int k = 0; k < C; k++) {
        const Fr v = element(k);
        pre[k] = acc;
        if (!fr_is_zero(v)) acc = fr_mul(acc, v);
    }
    Fr inv = fr_invert(acc);
#pragma unroll
    for (int k = C - 1; k >= 0; k--) {
        const Fr v = element(k);
        if (!fr_is_zero(v)) {
            a[first + (uint64_t)k * row] = fr_mul(pre[k], inv);
            inv = fr_mul(inv, v);
        }
    }
}

Status batch_invert(Context* ctx, Fr* a, uint64_t n, cudaStream_t st) {
    if (n == 0) return OK;
    // one warp per scheduler up to C = 8 (2^17 elements), two at 2^18
    const uint64_t wave = (uint64_t)ctx->num_sms * kInvThreads;
    const uint64_t per = (n + wave - 1) / wave;
    const int C = per <= 1 ? 1 : per <= 2 ? 2 : per <= 4 ? 4 : per <= 16 ? 8 : 16;
    const uint64_t blocks = (n + (uint64_t)kInvThreads * C - 1) / ((uint64_t)kInvThreads * C);
    if (blocks > 0x7fffffffull) {
        set_error("batch_invert: too many elements");
        return ERR_ARG;
    }
    const uint32_t g = (uint32_t)blocks;
    switch (C) {
        case 1: k_batch_invert<1><<<g, kInvThreads, 0, st>>>(a, n); break;
        case 2: k_batch_invert<2><<<g, kInvThreads, 0, st>>>(a, n); break;
        case 4: k_batch_invert<4><<<g, kInvThreads, 0, st>>>(a, n); break;
        case 8: k_batch_invert<8><<<g, kInvThreads, 0, st>>>(a, n); break;
        default: k_batch_invert<16><<<g, kInvThreads, 0, st>>>(a, n); break;
    }
    MZK_LAUNCH_CHECK(ctx);
    return OK;
}

// pass 1: out = exclusive scan within each tile of kThreads * kItems, sums[tile] = tile total
template <bool kMul, uint32_t kItems>
__global__ void __launch_bounds__(kThreads) k_scan_tile(const Fr* in, Fr* out, uint64_t n, Fr* __restrict__ sums) {
    __shared__ Fr sm[kThreads];
    const uint64_t base = ((uint64_t)blockIdx.x * kThreads + threadIdx.x) * kItems;
    Fr v[kItems];
    Fr acc = identity<kMul>();
#pragma unroll
    for (uint32_t j = 0; j < kItems; j++) {
        v[j] = base + j < n ? in[base + j] : identity<kMul>();
        acc = op<kMul>(acc, v[j]);
    }
    Fr total;
    Fr pre = block_exclusive<kMul>(acc, sm, &total);
#pragma unroll
    for (uint32_t j = 0; j < kItems; j++) {
        if (base + j < n) out[base + j] = pre;
        pre = op<kMul>(pre, v[j]);
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// pass 3: out[i] = prefix[tile] (op) out[i]
template <bool kMul>
__global__ void k_scan_apply(Fr* __restrict__ out, uint64_t n, const Fr* __restrict__ prefix, uint64_t tile) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint64_t t = i / tile;
        if (t) out[i] = op<kMul>(prefix[t], out[i]);
    }
}

// out[i] = in[0] (op) ... (op) in[i-1] (the identity for i = 0); in and out may alias
template <bool kMul>
Status scan_exclusive(Context* ctx, const Fr* in, Fr* out, uint64_t n, cudaStream_t st, int depth = 0) {
    if (n == 0) return OK;
    uint32_t items = kScanItemsMin;
    while (items < kScanItemsMax && n / (kThreads * items * 2) >= (uint64_t)ctx->num_sms * 2) items *= 2;
    const uint64_t tile = (uint64_t)kThreads * items;
    const uint64_t tiles = (n + tile - 1) / tile;
    void* sums;
    MZK_TRY(ctx->ensure(("grand_scan_" + std::to_string(depth)).c_str(), (tiles + 1) * sizeof(Fr), &sums));
    if (items == 2) k_scan_tile<kMul, 2><<<(uint32_t)tiles, kThreads, 0, st>>>(in, out, n, (Fr*)sums);
    else if (items == 4) k_scan_tile<kMul, 4><<<(uint32_t)tiles, kThreads, 0, st>>>(in, out, n, (Fr*)sums);
    else k_scan_tile<kMul, 8><<<(uint32_t)tiles, kThreads, 0, st>>>(in, out, n, (Fr*)sums);
    MZK_LAUNCH_CHECK(ctx);
    if (tiles > 1) {
        // exclusive scan of the tile totals (recursively), then fold it in
        MZK_TRY(scan_exclusive<kMul>(ctx, (const Fr*)sums, (Fr*)sums, tiles, st, depth + 1));
        k_scan_apply<kMul><<<grid_for(ctx, n, kThreads), kThreads, 0, st>>>(out, n, (const Fr*)sums, tile);
        MZK_LAUNCH_CHECK(ctx);
    }
    return OK;
}

// ---- first-order linear recurrences from the top: y_i = c_i + k y_{i+1},
// y_n = 0, for T tasks of one length (blockIdx.y: the task) ----
//
// A block takes kThreads x K consecutive elements, a thread K of them.  The
// chain of K products gives a thread its y with a zero carry-in, a scan over
// the block (log2 kThreads products, the factors k^(K 2^l) alike for every
// thread) the carry from the threads above, and the same chain started from
// the true carry the outputs.  Between blocks the values at the block starts
// solve the same recurrence with the factor k^(kThreads K): k_rec_totals leaves
// them, this function solves them, and k_rec_solve starts from the results.
// The products of a thread are a serial chain and small inputs are bound by it:
// K is 4 unless the blocks already fill the GPU.
constexpr uint32_t kRecItemsMin = 4, kRecItemsMax = 16;
constexpr uint32_t kRecBatch = 32;
constexpr uint32_t kRecLevels = 8;  // log2 kThreads
static_assert((1 << kRecLevels) == kThreads, "one scan level per bit of the thread index");

struct RecTasks {
    const Fr* c[kRecBatch];
    Fr* y[kRecBatch];
    Fr k[kRecBatch];
    Fr kk[kRecBatch][kRecLevels];  // k^(K 2^l)
};

// the thread's y at its first element with a zero carry-in
template <uint32_t K>
__device__ __forceinline__ Fr rec_chain(const Fr* __restrict__ c, uint64_t lo, uint64_t n, const Fr& k) {
    Fr acc = fr_zero();
#pragma unroll
    for (int i = (int)K - 1; i >= 0; i--) {
        const Fr v = lo + (uint64_t)i < n ? c[lo + (uint64_t)i] : fr_zero();
        acc = fr_add(v, fr_mul(k, acc));
    }
    return acc;
}

// v <- sum_{u >= t} k^(K (u - t)) v_u over the block's threads (sm: kThreads);
// live: threads from there on hold zero
__device__ __forceinline__ Fr rec_scan(Fr v, const Fr* __restrict__ kk, Fr* sm, uint32_t live) {
    sm[threadIdx.x] = v;
    __syncthreads();
#pragma unroll 1
    for (uint32_t l = 0; l < kRecLevels && (1u << l) < live; l++) {
        const uint32_t off = 1u << l;
        const bool on = threadIdx.x + off < (uint32_t)kThreads;
        if (on) v = fr_add(v, fr_mul(kk[l], sm[threadIdx.x + off]));
        __syncthreads();
        sm[threadIdx.x] = v;
        __syncthreads();
    }
    return v;
}

// threads of the block with elements below n, all of them where a carry comes in
template <uint32_t K>
__device__ __forceinline__ uint32_t rec_live(uint64_t n) {
    const uint64_t first = (uint64_t)blockIdx.x * kThreads * K;
    return (uint32_t)min((uint64_t)kThreads, (n - first + K - 1) / K);
}

// starts[task * stride + block] = the block's y at its first element with a zero carry-in
template <uint32_t K>
__global__ void __launch_bounds__(kThreads) k_rec_totals(const RecTasks t, uint64_t n, Fr* __restrict__ starts,
                                                         uint64_t stride) {
    __shared__ Fr sm[kThreads];
    const uint32_t j = blockIdx.y;
    const uint64_t lo = ((uint64_t)blockIdx.x * kThreads + threadIdx.x) * K;
    const Fr v = rec_scan(rec_chain<K>(t.c[j], lo, n, t.k[j]), t.kk[j], sm, rec_live<K>(n));
    if (threadIdx.x == 0) starts[j * stride + blockIdx.x] = v;
}

// every y, the block's carry-in carry[task * stride + block + 1] (none for the last)
template <uint32_t K>
__global__ void __launch_bounds__(kThreads) k_rec_solve(const RecTasks t, uint64_t n, const Fr* __restrict__ carry,
                                                        uint64_t stride) {
    __shared__ Fr sm[kThreads];
    const uint32_t j = blockIdx.y;
    const Fr* __restrict__ c = t.c[j];
    Fr* __restrict__ y = t.y[j];
    const Fr k = t.k[j];
    const uint64_t lo = ((uint64_t)blockIdx.x * kThreads + threadIdx.x) * K;
    Fr v = rec_chain<K>(c, lo, n, k);
    const bool has_carry = blockIdx.x + 1 < gridDim.x;
    Fr in = fr_zero();
    if (has_carry) in = carry[j * stride + blockIdx.x + 1];
    // the carry enters as the value above the last thread's chunk
    if (has_carry && threadIdx.x == kThreads - 1) v = fr_add(v, fr_mul(t.kk[j][0], in));
    rec_scan(v, t.kk[j], sm, rec_live<K>(n));
    Fr acc = threadIdx.x + 1 < (uint32_t)kThreads ? sm[threadIdx.x + 1] : in;
#pragma unroll
    for (int i = (int)K - 1; i >= 0; i--) {
        if (lo + (uint64_t)i < n) {
            acc = fr_add(c[lo + (uint64_t)i], fr_mul(k, acc));
            y[lo + (uint64_t)i] = acc;
        }
    }
}

template <uint32_t K>
cudaError_t launch_rec(const RecTasks& t, uint64_t n, uint64_t blocks, uint32_t T, Fr* starts, const Fr* carry,
                       uint64_t stride, cudaStream_t st) {
    const dim3 grid((uint32_t)blocks, T);
    if (starts) k_rec_totals<K><<<grid, kThreads, 0, st>>>(t, n, starts, stride);
    else k_rec_solve<K><<<grid, kThreads, 0, st>>>(t, n, carry, stride);
    return cudaGetLastError();
}

// y[j] (n) from c[j] (n) with factor k[j]; in and out may not alias.
// first_only (one task): y[0] receives its first value alone (y[0][0]).
Status linrec_suffix_batch(Context* ctx, const Fr* const* c, Fr* const* y, const host::Fr4* k, uint32_t T, uint64_t n,
                           cudaStream_t st, bool first_only = false, int depth = 0) {
    if (n == 0 || T == 0) return OK;
    // four elements per thread until the tasks' blocks are four per SM
    uint32_t K = kRecItemsMin;
    while (K < kRecItemsMax && n * std::min(T, kRecBatch) / ((uint64_t)kThreads * K * 2) >= (uint64_t)ctx->num_sms * 4)
        K *= 2;
    const uint64_t blocks = (n + (uint64_t)kThreads * K - 1) / ((uint64_t)kThreads * K);
    auto launch = [&](const RecTasks& t, uint32_t tb, Fr* starts, const Fr* carry) {
        return K == 4   ? launch_rec<4>(t, n, blocks, tb, starts, carry, 2 * blocks, st)
               : K == 8 ? launch_rec<8>(t, n, blocks, tb, starts, carry, 2 * blocks, st)
                        : launch_rec<16>(t, n, blocks, tb, starts, carry, 2 * blocks, st);
    };
    for (uint32_t j0 = 0; j0 < T; j0 += kRecBatch) {
        const uint32_t tb = std::min(kRecBatch, T - j0);
        RecTasks t;
        std::vector<host::Fr4> kblock(tb);
        for (uint32_t j = 0; j < tb; j++) {
            t.c[j] = c[j0 + j];
            t.y[j] = y[j0 + j];
            t.k[j] = to_dev(k[j0 + j]);
            host::Fr4 p = k[j0 + j];
            for (uint32_t b = 1; b < K; b <<= 1) p = host::fr_mul(p, p);
            for (uint32_t l = 0; l < kRecLevels; l++) {
                t.kk[j][l] = to_dev(p);
                p = host::fr_mul(p, p);
            }
            kblock[j] = p;  // k^(kThreads K)
        }
        Fr* starts = nullptr;
        if (blocks > 1) {
            // task j's block values at 2 blocks j, the solved ones after them
            void* buf;
            MZK_TRY(ctx->ensure(("grand_rec_" + std::to_string(depth)).c_str(), 2 * blocks * tb * sizeof(Fr), &buf));
            starts = static_cast<Fr*>(buf);
            MZK_CUDA_CHECK(launch(t, tb, starts, nullptr));
            ctx->launches++;
            std::vector<const Fr*> sc(tb);
            std::vector<Fr*> sy(tb);
            for (uint32_t j = 0; j < tb; j++) {
                sc[j] = starts + 2 * blocks * j;
                sy[j] = first_only ? t.y[j] : starts + 2 * blocks * j + blocks;
            }
            MZK_TRY(linrec_suffix_batch(ctx, sc.data(), sy.data(), kblock.data(), tb, blocks, st, first_only, depth + 1));
            if (first_only) continue;
        } else if (first_only) {  // its start is the first value
            MZK_CUDA_CHECK(launch(t, 1, t.y[0], nullptr));
            ctx->launches++;
            continue;
        }
        MZK_CUDA_CHECK(launch(t, tb, nullptr, starts ? starts + blocks : nullptr));
        ctx->launches++;
    }
    return OK;
}

Status linrec_suffix(Context* ctx, const Fr* c, Fr* y, uint64_t n, const host::Fr4& k, cudaStream_t st,
                     bool first_only = false) {
    return linrec_suffix_batch(ctx, &c, &y, &k, 1, n, st, first_only);
}

// ---- permutation argument ----
struct PermCols {
    const Fr* values[kMaxPermSetCols];
    const Fr* sigmas[kMaxPermSetCols];
    Fr delta_pow[kMaxPermSetCols];  // delta^(set chunk_len + j)
    uint32_t cols;
};

// den[i] = prod_j (beta s_j[i] + gamma + p_j[i])
__global__ void k_perm_den(PermCols pc, Fr beta, Fr gamma, Fr* __restrict__ den, uint32_t n) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        Fr acc = fr_one();
        for (uint32_t j = 0; j < pc.cols; j++)
            acc = fr_mul(acc, fr_add(fr_add(fr_mul(beta, pc.sigmas[j][i]), gamma), pc.values[j][i]));
        den[i] = acc;
    }
}
// mv[i] *= prod_j (delta^(..+j) w^i beta + gamma + p_j[i]); w^i from the split tables
__global__ void k_perm_num(PermCols pc, Fr beta, Fr gamma, const Fr* __restrict__ wlo, const Fr* __restrict__ whi,
                           Fr* __restrict__ mv, uint32_t n) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const Fr wb = fr_mul(fr_mul(wlo[i & 4095u], whi[i >> 12]), beta);
        Fr acc = mv[i];
        for (uint32_t j = 0; j < pc.cols; j++)
            acc = fr_mul(acc, fr_add(fr_add(fr_mul(pc.delta_pow[j], wb), gamma), pc.values[j][i]));
        mv[i] = acc;
    }
}
constexpr uint32_t kMaxPermSets = 16;
struct SetPtrs {
    Fr* z[kMaxPermSets];
};
// corr[0] = 1, corr[s] = corr[s-1] * z_{s-1}[n - bf - 1] (the uncorrected last
// products, read before any set is corrected); one thread, sets in order
__global__ void k_perm_corrections(SetPtrs sp, uint32_t sets, uint32_t last, Fr* __restrict__ corr) {
    Fr c = fr_one();
    for (uint32_t s = 0; s < sets; s++) {
        corr[s] = c;
        c = fr_mul(c, sp.z[s][last]);
    }
}
// z[i] = (i < n - bf ? z[i] : blinds[i - (n - bf)]) * corr (multiplying by
// one where the reference skips the product leaves the value unchanged)
__global__ void k_perm_finish(Fr* __restrict__ z, uint32_t n, uint32_t bf, const Fr* __restrict__ blinds,
                              const Fr* __restrict__ corr) {
    const Fr c = *corr;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const Fr v = i < n - bf ? z[i] : blinds[i - (n - bf)];
        z[i] = fr_mul(v, c);
    }
}

// ---- logup argument ----
// out[i] = beta + v[i]
__global__ void k_add_const(const Fr* __restrict__ v, Fr beta, Fr* __restrict__ out, uint32_t n) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = fr_add(beta, v[i]);
}
// h[i] = sum of the chunk's inverted columns (cols consecutive arrays of n)
__global__ void k_sum_cols(const Fr* __restrict__ inv, uint32_t cols, Fr* __restrict__ h, uint32_t n) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        Fr acc = fr_zero();
        for (uint32_t j = 0; j < cols; j++) acc = fr_add(acc, inv[(size_t)j * n + i]);
        h[i] = acc;
    }
}
// ld[i] = sel[i] * sum_c h_c[i] - m[i] * tden[i]
struct HelperPtrs {
    Fr* h[kMaxLogupChunks];
    uint32_t chunks;
};
__global__ void k_logderivative(HelperPtrs hp, const Fr* __restrict__ sel, const Fr* __restrict__ m,
                                const Fr* __restrict__ tden, Fr* __restrict__ ld, uint32_t n) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        Fr s = fr_zero();
        for (uint32_t c = 0; c < hp.chunks; c++) s = fr_add(s, hp.h[c][i]);
        ld[i] = fr_sub(fr_mul(sel[i], s), fr_mul(m[i], tden[i]));
    }
}
// z[n - bf + b] = blinds[b]
__global__ void k_set_tail(Fr* __restrict__ z, uint32_t n, uint32_t bf, const Fr* __restrict__ blinds) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < bf) z[n - bf + b] = blinds[b];
}

}  // namespace

Status permutation_z_device(Context* ctx, const Domain* d, const mzk_permutation_desc* desc, cudaStream_t st) {
    const uint32_t n = 1u << d->k, bf = desc->blinding_factors;
    if (desc->chunk_len == 0 || desc->chunk_len > kMaxPermSetCols || bf + 1 >= n || desc->n_cols == 0 ||
        !desc->values || !desc->sigmas || !desc->z_out || (bf && !desc->blinds)) {
        set_error("permutation_z: need 1..8 columns per set, blinding_factors < n - 1 and non-null arrays");
        return ERR_ARG;
    }
    const uint32_t sets = (desc->n_cols + desc->chunk_len - 1) / desc->chunk_len;
    if (sets > kMaxPermSets) {
        set_error("permutation_z: at most 16 sets");
        return ERR_ARG;
    }
    void *mv_buf, *dbl, *corr;
    MZK_TRY(ctx->ensure("perm_mv", (size_t)n * sizeof(Fr), &mv_buf));
    MZK_TRY(ctx->ensure("perm_blinds", ((size_t)sets * bf + 1) * sizeof(Fr), &dbl));
    MZK_TRY(ctx->ensure("perm_corr", (size_t)sets * sizeof(Fr), &corr));
    if (bf)
        MZK_CUDA_CHECK(cudaMemcpyAsync(dbl, desc->blinds, (size_t)sets * bf * sizeof(Fr), cudaMemcpyHostToDevice, st));
    Fr* mv = (Fr*)mv_buf;
    const Fr beta = to_dev(to_host(desc->beta)), gamma = to_dev(to_host(desc->gamma));
    const host::Fr4 delta = to_host(host::FR_DELTA4);
    const uint32_t grid = grid_for(ctx, n, kThreads);
    for (uint32_t s = 0; s < sets; s++) {
        PermCols pc;
        pc.cols = std::min(desc->chunk_len, desc->n_cols - s * desc->chunk_len);
        const uint64_t e0 = (uint64_t)s * desc->chunk_len;
        host::Fr4 dp = host::fr_pow(delta, &e0, 1);
        for (uint32_t j = 0; j < pc.cols; j++) {
            const uint32_t c = s * desc->chunk_len + j;
            if (!desc->values[c] || !desc->sigmas[c] || !desc->z_out[s]) {
                set_error("permutation_z: null column");
                return ERR_ARG;
            }
            pc.values[j] = reinterpret_cast<const Fr*>(desc->values[c]);
            pc.sigmas[j] = reinterpret_cast<const Fr*>(desc->sigmas[c]);
            pc.delta_pow[j] = to_dev(dp);
            dp = host::fr_mul(dp, delta);
        }
        k_perm_den<<<grid, kThreads, 0, st>>>(pc, beta, gamma, mv, n);
        MZK_LAUNCH_CHECK(ctx);
        MZK_TRY(batch_invert(ctx, mv, n, st));
        k_perm_num<<<grid, kThreads, 0, st>>>(pc, beta, gamma, d->lo[0], d->hi[0], mv, n);
        MZK_LAUNCH_CHECK(ctx);
        Fr* z = reinterpret_cast<Fr*>(desc->z_out[s]);
        MZK_TRY(scan_exclusive<true>(ctx, mv, z, n, st));
    }
    // corrections from the uncorrected last products z_s[n - bf - 1], on the
    // device (no host round trip), then blinds and corrections per set
    SetPtrs sp;
    for (uint32_t s = 0; s < sets; s++) sp.z[s] = reinterpret_cast<Fr*>(desc->z_out[s]);
    k_perm_corrections<<<1, 1, 0, st>>>(sp, sets, n - bf - 1, (Fr*)corr);
    MZK_LAUNCH_CHECK(ctx);
    for (uint32_t s = 0; s < sets; s++) {
        k_perm_finish<<<grid, kThreads, 0, st>>>(sp.z[s], n, bf, (const Fr*)dbl + (size_t)s * bf, (const Fr*)corr + s);
        MZK_LAUNCH_CHECK(ctx);
    }
    return OK;
}

Status logup_device(Context* ctx, const Domain* d, const mzk_logup_desc* desc, cudaStream_t st) {
    const uint32_t n = 1u << d->k, bf = desc->blinding_factors;
    if (desc->n_chunks == 0 || desc->n_chunks > kMaxLogupChunks || bf + 1 >= n || !desc->chunk_cols ||
        !desc->inputs || !desc->table || !desc->selector || !desc->multiplicities || !desc->helpers_out ||
        !desc->aggregator_out || (bf && !desc->blinds)) {
        set_error("logup: need 1..8 chunks, blinding_factors < n - 1 and non-null arrays");
        return ERR_ARG;
    }
    uint32_t total_cols = 0;
    for (uint32_t c = 0; c < desc->n_chunks; c++) total_cols += desc->chunk_cols[c];
    void *cols_buf, *ld_buf, *dbl;
    // the table's column, then the inputs', inverted together
    MZK_TRY(ctx->ensure("logup_cols", ((size_t)total_cols + 1) * n * sizeof(Fr), &cols_buf));
    MZK_TRY(ctx->ensure("logup_ld", (size_t)n * sizeof(Fr), &ld_buf));
    MZK_TRY(ctx->ensure("logup_blinds", ((size_t)bf + 1) * sizeof(Fr), &dbl));
    if (bf) MZK_CUDA_CHECK(cudaMemcpyAsync(dbl, desc->blinds, (size_t)bf * sizeof(Fr), cudaMemcpyHostToDevice, st));
    Fr *tden = (Fr*)cols_buf, *cols = tden + n, *ld = (Fr*)ld_buf;
    const Fr beta = to_dev(to_host(desc->beta));
    const uint32_t grid = grid_for(ctx, n, kThreads);
    // T = 1 / (t + beta) and, for every input column, 1 / (f + beta) (inverting
    // them together gives the same field values)
    k_add_const<<<grid, kThreads, 0, st>>>(reinterpret_cast<const Fr*>(desc->table), beta, tden, n);
    MZK_LAUNCH_CHECK(ctx);
    for (uint32_t j = 0; j < total_cols; j++) {
        if (!desc->inputs[j]) {
            set_error("logup: null input column");
            return ERR_ARG;
        }
        k_add_const<<<grid, kThreads, 0, st>>>(reinterpret_cast<const Fr*>(desc->inputs[j]), beta,
                                               cols + (size_t)j * n, n);
        MZK_LAUNCH_CHECK(ctx);
    }
    MZK_TRY(batch_invert(ctx, tden, ((uint64_t)total_cols + 1) * n, st));
    HelperPtrs hp;
    hp.chunks = desc->n_chunks;
    for (uint32_t c = 0, j = 0; c < desc->n_chunks; j += desc->chunk_cols[c], c++) {
        if (!desc->helpers_out[c]) {
            set_error("logup: null helper output");
            return ERR_ARG;
        }
        hp.h[c] = reinterpret_cast<Fr*>(desc->helpers_out[c]);
        k_sum_cols<<<grid, kThreads, 0, st>>>(cols + (size_t)j * n, desc->chunk_cols[c], hp.h[c], n);
        MZK_LAUNCH_CHECK(ctx);
    }
    k_logderivative<<<grid, kThreads, 0, st>>>(hp, reinterpret_cast<const Fr*>(desc->selector),
                                               reinterpret_cast<const Fr*>(desc->multiplicities), tden, ld, n);
    MZK_LAUNCH_CHECK(ctx);
    // aggregator: exclusive running sum over the first n - bf rows, then the blinds
    Fr* agg = reinterpret_cast<Fr*>(desc->aggregator_out);
    MZK_TRY(scan_exclusive<false>(ctx, ld, agg, n - bf, st));
    if (bf) {
        k_set_tail<<<1, 64, 0, st>>>(agg, n, bf, (const Fr*)dbl);
        MZK_LAUNCH_CHECK(ctx);
    }
    return OK;
}

namespace {
// out[i] = sum_p s_p polys[p][i] (i < len_p), polys and lengths in device tables
__global__ void k_inner_product(const Fr* const* __restrict__ polys, const uint64_t* __restrict__ lens,
                                const Fr* __restrict__ scalars, uint32_t m, Fr* __restrict__ out, uint64_t out_len) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < out_len; i += stride) {
        Fr acc = fr_zero();
        for (uint32_t p = 0; p < m; p++)
            if (i < lens[p]) acc = fr_add(acc, fr_mul(polys[p][i], scalars[p]));
        out[i] = acc;
    }
}
}  // namespace

Status poly_inner_product_device(Context* ctx, const uint64_t* const* polys, const uint64_t* lens, uint32_t m,
                                 const uint64_t* scalars, void* out, uint64_t out_len, cudaStream_t st) {
    if (out_len == 0) return OK;
    // one device table: m pointers, m lengths, m scalars (staged through pinned memory)
    const size_t bytes = (size_t)m * (8 + 8 + 32);
    void *d_tab, *h_tab;
    MZK_TRY(ctx->ensure("grand_ip_tab", bytes + 64, &d_tab));
    MZK_TRY(ctx->ensure_pinned(bytes + 64, &h_tab));
    char* h = static_cast<char*>(h_tab);
    std::memcpy(h, polys, (size_t)m * 8);
    std::memcpy(h + (size_t)m * 8, lens, (size_t)m * 8);
    std::memcpy(h + (size_t)m * 16, scalars, (size_t)m * 32);
    MZK_CUDA_CHECK(cudaMemcpyAsync(d_tab, h_tab, bytes, cudaMemcpyHostToDevice, st));
    const char* d = static_cast<const char*>(d_tab);
    k_inner_product<<<grid_for(ctx, out_len, kThreads), kThreads, 0, st>>>(
        reinterpret_cast<const Fr* const*>(d), reinterpret_cast<const uint64_t*>(d + (size_t)m * 8),
        reinterpret_cast<const Fr*>(d + (size_t)m * 16), m, static_cast<Fr*>(out), out_len);
    MZK_LAUNCH_CHECK(ctx);
    // the pinned table is reused by the next call: finish this one first
    MZK_CUDA_CHECK(cudaStreamSynchronize(st));
    return OK;
}

namespace {
__global__ void k_fill(Fr* __restrict__ out, uint64_t n, Fr v) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = v;
}
}  // namespace

Status fr_powers_device(Context* ctx, const uint64_t s[4], uint64_t n, void* out, cudaStream_t st) {
    if (n == 0) return OK;
    k_fill<<<grid_for(ctx, n, kThreads), kThreads, 0, st>>>(static_cast<Fr*>(out), n, to_dev(to_host(s)));
    MZK_LAUNCH_CHECK(ctx);
    return scan_exclusive<true>(ctx, static_cast<const Fr*>(out), static_cast<Fr*>(out), n, st);
}

Status batch_invert_device(Context* ctx, void* a, uint64_t n, cudaStream_t st) {
    return batch_invert(ctx, static_cast<Fr*>(a), n, st);
}

Status eval_polynomial_device(Context* ctx, const void* poly, uint64_t n, const uint64_t point[4], uint64_t out[4],
                              cudaStream_t st) {
    std::memset(out, 0, 32);
    if (n == 0) return OK;
    void* y;
    MZK_TRY(ctx->ensure("grand_eval", sizeof(Fr), &y));
    MZK_TRY(linrec_suffix(ctx, static_cast<const Fr*>(poly), (Fr*)y, n, to_host(point), st, true));
    MZK_CUDA_CHECK(cudaMemcpyAsync(out, y, 32, cudaMemcpyDeviceToHost, st));
    MZK_CUDA_CHECK(cudaStreamSynchronize(st));
    return OK;
}

Status kate_division_device(Context* ctx, const void* a, uint64_t n, const uint64_t b[4], void* q, cudaStream_t st) {
    if (n < 2) return OK;
    // q_i = a_{i+1} + b q_{i+1}, q_{n-1} = 0
    return linrec_suffix(ctx, static_cast<const Fr*>(a) + 1, static_cast<Fr*>(q), n - 1, to_host(b), st);
}

Status kate_division_batch(Context* ctx, const void* const* a, void* const* q, const host::Fr4* b, uint32_t T,
                           uint64_t n, cudaStream_t st) {
    if (n < 2 || T == 0) return OK;
    std::vector<const Fr*> c(T);
    for (uint32_t j = 0; j < T; j++) c[j] = static_cast<const Fr*>(a[j]) + 1;
    return linrec_suffix_batch(ctx, c.data(), reinterpret_cast<Fr* const*>(q), b, T, n - 1, st);
}

}  // namespace mzk
