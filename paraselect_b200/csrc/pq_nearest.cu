// Nearest codeword of every sub-vector: a tcgen05 product that filters, exact distances that decide.  PQ encoding and the assignment of the
// codebook trainer.
//
// Semantics follow the reference encoder and trainer: argmin of squared L2 with strict '<', so that the lowest index wins ties
// (src/quantization/pq/pq_encode.cuh:24-40, src/clustering/kmeans/kmeans_utils.cu:359-413).
//
// Per (row, sub-quantiser) all k codewords have to be compared; evaluated one by one in the reference encoder's arithmetic (sub,
// mul, add per dimension, compare, select) that is 13 instructions for each of n * m * k pairs and the whole cost.  Here
// w = x.c - |c|^2 / 2 (largest for the nearest codeword) comes from the tensor cores with the operands split into two bf16 terms each and the
// norm into three,
//     K slots  [ xh  xh  xl  1 1 1 ] . [ ch  cl  ch  -n0 -n1 -n2 ],   3 D + 3 <= 16 * KS,
// which is within E of the true value; only groups of eight codewords that hold a value >= max - 2E are evaluated exactly.
//   E: bf16 splits 3.1 * 2^-18 |x||c|; accumulation and norm split (16 KS) 2^-22 (|x||c| + |c|^2 / 2); rounding of the exact fp32
//   distance (2 D + 2) 2^-24 (|x| + |c|)^2: together 2E <= 2^-15 |x| cmax + (KS + 1) 2^-18 (|x| + cmax)^2, and where products
//   are subnormal or vanish, 2^-126 for each of the 16 KS products and three norm terms: 2 (16 KS + 3) 2^-126 <= 2^-118.
// The nearest codeword in the exact arithmetic and all its ties are among the evaluated ones; the lowest index wins a tie.
// kTrain: the evaluated ones are compared by |c|^2 - 2 x.c in fused multiply-adds, as the trainer's Lloyd iterations always have (the
// reference's trainer assigns with a TF32 GEMM: src/quantization/pq/pq_trainer.cu:97-170); its rounding is within the same bound.
//
// One accumulator = 128 rows x 256 codewords of one sub-quantiser, K = 16 KS: a row's scores lie in one thread's lane of tensor memory, so
// their maxima need no exchange between lanes.  A 128-byte operand row holds the K steps of SPA = 4 / KS sub-quantisers ("an atom"); B (the
// codebook) is built once per item of up to kMaxTiles row tiles.
//   warps 0-2    producers: B and the fp32 codewords of an item (ring of 2; the next item's a part at a time between the tiles), the fp32
//                sub-vectors of a row tile (ring of kRingX, copied kAhead tiles ahead) and A (ring of kRingA)
//   warp 3       issues the products, each into the next of two accumulators (the whole tensor memory)
//   warps 4-15   three groups of four: maxima of the accumulators, evaluation, codes; a group takes every third tile, all its sub-quantisers
// What bounds it: the groups' dependent steps on an accumulator (read 800 cycles, threshold 480, evaluation 800) at three warps per scheduler;
// the maxima alone (one three-input maximum per two scores, a two-cycle instruction) would take 0.23 ms of the first case below.  Accumulators of
// half the codewords, two groups, or one product warp per group were slower.  Against mma.sync, whose 8 cycles per 128 scores and SM quarter, one
// comparison per score and hit queue this replaces: 1M rows, 128 dimensions, m = 32 2,037 -> 1,100 us; 96, 48 5,367 -> 1,640; 128, 16
// 1,823 -> 790; 32,768 x 96, m = 24 80.6 -> 47; 1,000 x 128, m = 32 19.5 -> 19.
#include <cuda_bf16.h>
#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "kernels.h"
#include "tc_ptx.cuh"

namespace psb {

using namespace tc;

namespace {

constexpr int kTile = 128;         // rows of a tile (M of the product)
constexpr int kCodes = 256;        // codewords, those past k far away
constexpr int kGroups = 3;
constexpr int kRingA = 4, kRingX = 8;   // row tiles in flight as operands, and as fp32 sub-vectors
constexpr int kAhead = 2;          // tiles whose sub-vectors are on their way while one is converted
constexpr int kAcc = 2;            // accumulators: all of the tensor memory
constexpr int kProducerWarps = 3, kProducerThreads = kProducerWarps * 32;
constexpr int kWarpIssue = 3;      // warps 0-2: producers, 3: issuer, 4-15: groups
constexpr int kThreads = (kWarpIssue + 1 + 4 * kGroups) * 32;   // sixteen warps: 128 registers each
constexpr int kMaxTiles = 15;      // row tiles of an item at most, whole turns of the groups: building B takes a twentieth of the work on them
constexpr float kTiny = 3.1e-36f;  // above 2^-118
constexpr float kFarNorm = 3.0e38f;   // in place of |c|^2 / 2 for codewords past k: below every score a threshold is taken from
constexpr uint32_t kTmemCols = 512;
constexpr int kNearWaitLimit = 1 << 18;   // polls before a wait gives up

template <int D> struct Near {
    static constexpr int KS = (3 * D + 3 + 15) / 16;
    static constexpr int SPA = KS == 1 ? 4 : (KS == 2 ? 2 : 1);
    // A row's sub-vectors in shared memory: an odd number of vector loads apart, or four with their places exchanged from row to row, so that a
    // warp's rows spread over the banks.
    static constexpr int V = D % 4 == 0 ? 4 : (D % 2 == 0 ? 2 : 1);
    static constexpr bool TURN = V == 4 && SPA * D == 16;
    static constexpr int PITCH = TURN ? 16 : ((SPA * D / V) | 1) * V;
    static __device__ __forceinline__ int place(int row, int d) { return row * PITCH + (TURN ? d ^ (((row >> 1) & 3) << 2) : d); }   // d: a multiple of V
    static constexpr size_t B = (size_t)kCodes * 128, A = (size_t)kTile * 128, CB = (size_t)SPA * kCodes * D * 4, X = (size_t)kTile * PITCH * 4;
    static constexpr size_t SMEM = 1024 + 2 * (B + CB) + kRingA * A + kRingX * X;
};

__device__ __forceinline__ uint32_t bf16_word(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
template <int D>
__device__ __forceinline__ void load_vec(float (&v)[D], const float* __restrict__ x) {   // a sub-vector from shared memory
    if constexpr (D % 4 == 0) {
#pragma unroll
        for (int d = 0; d < D; d += 4) { const float4 w = *reinterpret_cast<const float4*>(x + d); v[d] = w.x; v[d + 1] = w.y; v[d + 2] = w.z; v[d + 3] = w.w; }
    } else if constexpr (D % 2 == 0) {
#pragma unroll
        for (int d = 0; d < D; d += 2) { const float2 w = *reinterpret_cast<const float2*>(x + d); v[d] = w.x; v[d + 1] = w.y; }
    } else {
#pragma unroll
        for (int d = 0; d < D; ++d) v[d] = x[d];
    }
}
template <int D>
__device__ __forceinline__ void load_row(float (&v)[D], const float* __restrict__ x, int row, int sub) {   // a sub-vector of a row tile
    using P = Near<D>;
    if constexpr (P::TURN) {
#pragma unroll
        for (int d = 0; d < D; d += 4) {
            const float4 w = *reinterpret_cast<const float4*>(x + P::place(row, sub * D + d));
            v[d] = w.x; v[d + 1] = w.y; v[d + 2] = w.z; v[d + 3] = w.w;
        }
    } else {
        load_vec<D>(v, x + row * P::PITCH + sub * D);
    }
}
template <int D>
__device__ __forceinline__ void store_vec(float* __restrict__ x, const float (&v)[D]) {
    if constexpr (D % 4 == 0) {
#pragma unroll
        for (int d = 0; d < D; d += 4) *reinterpret_cast<float4*>(x + d) = make_float4(v[d], v[d + 1], v[d + 2], v[d + 3]);
    } else if constexpr (D % 2 == 0) {
#pragma unroll
        for (int d = 0; d < D; d += 2) *reinterpret_cast<float2*>(x + d) = make_float2(v[d], v[d + 1]);
    } else {
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = v[d];
    }
}
// The K slots of one sub-quantiser as 2 KS chunks of eight bf16 in an operand row (128-byte swizzle): first, second, third D slots from
// (hi, hi, lo) of a row or (hi, lo, hi) of a codeword, then three more.
template <int D, bool kRow>
__device__ __forceinline__ void store_slots(unsigned char* __restrict__ operand, int row, int sub, const float (&v)[D], float t0, float t1, float t2) {
    constexpr int KS = Near<D>::KS;
    uint32_t word[KS * 8];
#pragma unroll
    for (int w = 0; w < KS * 8; ++w) word[w] = 0u;
    if constexpr (D % 2 == 0) {
#pragma unroll
        for (int d = 0; d < D; d += 2) {
            const uint32_t h = bf16_word(v[d], v[d + 1]);
            const uint32_t l = bf16_word(v[d] - __uint_as_float(h << 16), v[d + 1] - __uint_as_float(h & 0xFFFF0000u));
            word[d / 2] = h; word[(D + d) / 2] = kRow ? h : l; word[(2 * D + d) / 2] = kRow ? l : h;
        }
        word[3 * D / 2] = bf16_word(t0, t1); word[3 * D / 2 + 1] = bf16_word(t2, 0.0f);
    } else {
        float slot[KS * 16];
#pragma unroll
        for (int s = 0; s < KS * 16; ++s) slot[s] = 0.0f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const float h = bf16_round(v[d]), l = v[d] - h;
            slot[d] = h; slot[D + d] = kRow ? h : l; slot[2 * D + d] = kRow ? l : h;
        }
        slot[3 * D] = t0; slot[3 * D + 1] = t1; slot[3 * D + 2] = t2;
#pragma unroll
        for (int w = 0; w < KS * 8; ++w) word[w] = bf16_word(slot[2 * w], slot[2 * w + 1]);
    }
    unsigned char* base = operand + (size_t)row * 128;
#pragma unroll
    for (int c = 0; c < 2 * KS; ++c)
        *reinterpret_cast<uint4*>(base + (((uint32_t)(sub * 2 * KS + c) ^ ((uint32_t)row & 7u)) << 4)) =
            make_uint4(word[4 * c], word[4 * c + 1], word[4 * c + 2], word[4 * c + 3]);
}
// Global to shared memory behind the thread's back, N bytes (4, 8, 16), zeros where there is nothing to read.
template <int N>
__device__ __forceinline__ void copy_behind(float* dst, const float* src, bool live) {
    if constexpr (N == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(live ? N : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(dst)), "l"(src), "n"(N), "r"(live ? N : 0) : "memory");
}
// The exact distance that decides.
template <int D, bool kTrain>
__device__ __forceinline__ float near_dist(const float (&x)[D], const float (&c)[D]) {
    float dist = 0.0f;
    if constexpr (kTrain) {
#pragma unroll
        for (int d = 0; d < D; ++d) dist = fmaf(c[d], c[d], dist);
#pragma unroll
        for (int d = 0; d < D; ++d) dist = fmaf(x[d], -2.0f * c[d], dist);
    } else {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const float diff = __fsub_rn(x[d], c[d]);
            dist = __fadd_rn(dist, __fmul_rn(diff, diff));
        }
    }
    return dist;
}

// Not below the square root: the approximation is good to a few units in the last place.
__device__ __forceinline__ float near_root(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r * 1.00001f;
}
__device__ __forceinline__ bool near_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    for (int i = 0; i < kNearWaitLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255) == 255 && *abort_flag) return false;
    }
    return false;
}
__device__ __forceinline__ bool near_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(0xffffffffu, near_wait(bar, parity, abort_flag));
}
__device__ __forceinline__ void near_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }

struct NearArgs {
    const float* data;       // [n][dim]
    const float* codebook;   // [m][k][D]
    uint8_t* codes;          // [n][m]
    long long n;
    int dim, m, k;
    int atoms;               // ranges of SPA sub-quantisers
    long long tiles;         // of kTile rows
    int per;                 // tiles of an item at most
    long long items;         // atoms x ranges of tiles, the atom running fastest: CTAs at work together read neighbouring parts of the rows
    int vec;                 // sub-vectors may be loaded V floats at a time
    int step_atom;           // from one item of a CTA to its next: atoms, and tiles
    long long step_tiles;
    long long issued;        // the items below this one get their products: all, or fewer in the test of the time-out path
    int* gave_up;            // the test's count of CTAs that gave up, or null
};

// The items of a CTA in order; every role walks them on its own.
struct NearItem {
    long long id, tile;      // tile: the first of its row tiles
    int atom;
    uint32_t it = 0, t = 0;  // running numbers of the item and of its first tile
    __device__ __forceinline__ explicit NearItem(const NearArgs& g) : id(blockIdx.x) {
        const unsigned c = blockIdx.x / (unsigned)g.atoms;
        atom = (int)(blockIdx.x - c * (unsigned)g.atoms);
        tile = (long long)c * g.per;
    }
    __device__ __forceinline__ bool live(const NearArgs& g) const { return id < g.items; }
    __device__ __forceinline__ int tiles(const NearArgs& g) const { return (int)min((long long)g.per, g.tiles - tile); }
    template <int SPA> __device__ __forceinline__ int subs(const NearArgs& g) const { return min(SPA, g.m - atom * SPA); }
    __device__ __forceinline__ void next(const NearArgs& g) {
        t += (uint32_t)tiles(g); ++it; id += gridDim.x;
        atom += g.step_atom; tile += g.step_tiles;
        if (atom >= g.atoms) { atom -= g.atoms; tile += g.per; }
    }
};

// Codewords e0 .. e1 (256 to a sub-quantiser) of an item, every `stride`-th from this thread's on: operand, fp32 copy and largest norms.  A function of
// its own: inlined at both of its places it made the kernel 8 % slower, whose roles share the instruction cache.
template <int D>
__device__ __noinline__ void near_build(const float* __restrict__ codebook, int k, int sub0, int e0, int e1, int stride, unsigned char* __restrict__ operand,
                                        float* __restrict__ cb, float* __restrict__ cmax) {
    for (int e = e0; e < e1; e += stride) {   // a warp's codewords belong to one sub-quantiser
        const int sub = e / kCodes, c = e % kCodes;
        float v[D], n2 = 0.0f;
        const float* src = codebook + ((size_t)(sub0 + sub) * k + c) * D;
#pragma unroll
        for (int d = 0; d < D; ++d) v[d] = c < k ? __ldg(src + d) : 0.0f;
#pragma unroll
        for (int d = 0; d < D; ++d) n2 = fmaf(v[d], v[d], n2);
        float rest = c < k ? 0.5f * n2 : kFarNorm, n[3];   // codewords past k are never near
#pragma unroll
        for (int i = 0; i < 3; ++i) { n[i] = bf16_round(rest); rest -= n[i]; }
        store_slots<D, false>(operand, c, sub, v, -n[0], -n[1], -n[2]);
#pragma unroll
        for (int d = 0; d < D; ++d) v[d] = c < k ? v[d] : __int_as_float(0x7f800000);   // no distance to them is a finite number
        store_vec<D>(cb + (size_t)e * D, v);
        const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(n2) & 0x7fffffffu);   // bits: what is not a number comes first
        if ((threadIdx.x & 31) == 0) cmax[e >> 5] = __uint_as_float(top);
    }
}

template <int D, bool kTrain>
__global__ void __launch_bounds__(kThreads, 1) k_pq_nearest(const NearArgs g) {
    using P = Near<D>;
    constexpr int KS = P::KS, SPA = P::SPA, PITCH = P::PITCH;
    extern __shared__ __align__(1024) unsigned char s_raw[];
    unsigned char* s_b = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(s_raw) + 1023) & ~uintptr_t(1023));   // [2] operand of an atom's codewords
    unsigned char* s_a = s_b + 2 * P::B;                                   // [kRingA] operand of a row tile
    float* s_cb = reinterpret_cast<float*>(s_a + kRingA * P::A);            // [2][SPA][kCodes][D] the codewords
    float* s_x = s_cb + 2 * P::CB / 4;                                     // [kRingX][kTile][PITCH]
    __shared__ __align__(8) uint64_t b_full[2], b_empty[2], a_full[kRingX], a_empty[kRingA], x_empty[kRingX], acc_full[kGroups][kAcc], acc_empty[kAcc], drained;
    __shared__ __align__(16) float s_cmax[2][SPA][kCodes / 32];   // largest |c|^2 of every 32 codewords
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    volatile int* abort_flag = &s_abort;

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) { mbar_init(&b_full[i], kProducerThreads); mbar_init(&b_empty[i], 1 + 4 * kGroups); }
        for (int i = 0; i < kRingX; ++i) { mbar_init(&a_full[i], kProducerThreads); mbar_init(&x_empty[i], 4); }
        for (int i = 0; i < kRingA; ++i) mbar_init(&a_empty[i], 1);
        for (int i = 0; i < kAcc; ++i) {
            for (int p = 0; p < kGroups; ++p) mbar_init(&acc_full[p][i], 1);
            mbar_init(&acc_empty[i], 4);
        }
        mbar_init(&drained, 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(&s_tmem, kTmemCols);
    {   // the first item's, by all warps
        const NearItem o(g);
        if (o.live(g)) near_build<D>(g.codebook, g.k, o.atom * SPA, tid, o.subs<SPA>(g) * kCodes, kThreads, s_b, s_cb, &s_cmax[0][0][0]);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // operand stores -> visible to the tensor core
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    bool failed = false;

    if (warp < kProducerWarps) {
        // ---- producers ----
        constexpr int TASKS = SPA * kTile, EACH = (TASKS + kProducerThreads - 1) / kProducerThreads;
        // Sub-vectors of a tile, (row, sub) number i * 96 + tid with the sub-quantiser running fastest: a thread converts what it copied.
        NearItem ao(g);   // the tile copied next
        int ak = 0;
        auto copy = [&]() {
            if (ao.live(g)) {
                const uint32_t t = ao.t + (uint32_t)ak;
                if (!near_wait_warp(&x_empty[t % kRingX], ((t / kRingX) & 1u) ^ 1u, abort_flag)) return false;
                float* to = s_x + (size_t)(t % kRingX) * kTile * PITCH;
                const int nsub = ao.subs<SPA>(g);
#pragma unroll 1
                for (int i = 0; i < EACH; ++i) {
                    const int e = i * kProducerThreads + tid, sub = e % SPA;
                    if (e >= TASKS) break;
                    const long long row = (ao.tile + ak) * kTile + e / SPA;
                    const bool live = row < g.n && sub < nsub;
                    const float* src = live ? g.data + (size_t)row * g.dim + (size_t)(ao.atom * SPA + sub) * D : g.data;
                    const int at = e / SPA;
                    if (P::V == 4 && g.vec) {
#pragma unroll
                        for (int d = 0; d < D; d += 4) copy_behind<16>(to + P::place(at, sub * D + d), src + d, live);
                    } else if (P::V == 2 && g.vec) {
#pragma unroll
                        for (int d = 0; d < D; d += 2) copy_behind<8>(to + P::place(at, sub * D + d), src + d, live);
                    } else {
#pragma unroll
                        for (int d = 0; d < D; ++d) copy_behind<4>(to + P::place(at, (sub * D + d) / P::V * P::V) + (sub * D + d) % P::V, src + d, live);
                    }
                }
                if (++ak == ao.tiles(g)) { ak = 0; ao.next(g); }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            return true;
        };
        for (int i = 0; i < kAhead && !failed; ++i) failed = !copy();
        auto built = [&](const NearItem& o) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // operand stores -> visible to the tensor core
            near_arrive(&b_full[o.it & 1u]);
        };
        NearItem o(g);
        if (!failed && o.live(g)) built(o);
        while (o.live(g) && !failed) {
            const int ntiles = o.tiles(g);
            NearItem then = o;
            then.next(g);
            const int todo = then.live(g) ? then.subs<SPA>(g) * kCodes : 0;
            int done = 0;
            for (int k = 0; k < ntiles; ++k) {
                const uint32_t t = o.t + (uint32_t)k, slot = t % kRingA;
                if (!copy()) { failed = true; break; }
                asm volatile("cp.async.wait_group %0;" ::"n"(kAhead) : "memory");   // this tile's sub-vectors are there
                if (!near_wait_warp(&a_empty[slot], ((t / kRingA) & 1u) ^ 1u, abort_flag)) { failed = true; break; }
#pragma unroll 2
                for (int i = 0; i < EACH; ++i) {
                    const int e = i * kProducerThreads + tid, sub = e % SPA, row = e / SPA;
                    if (e >= TASKS) break;
                    float v[D];
                    load_row<D>(v, s_x + (size_t)(t % kRingX) * kTile * PITCH, row, sub);
                    store_slots<D, true>(s_a + slot * P::A, row, sub, v, 1.0f, 1.0f, 1.0f);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                near_arrive(&a_full[t % kRingX]);
                // The next item's codewords, a part of them behind each tile.  (The first tiles may still be ahead of the groups' last ones of the item before, whose codewords are in the place.)
                if (done < todo && (k >= kRingA || k + 1 == ntiles)) {
                    if (done == 0 && !near_wait_warp(&b_empty[then.it & 1u], ((then.it >> 1) & 1u) ^ 1u, abort_flag)) { failed = true; break; }
                    const int upto = k + 1 == ntiles ? todo : min(todo, done + kProducerThreads);
                    const uint32_t bs = then.it & 1u;
                    near_build<D>(g.codebook, g.k, then.atom * SPA, done + tid, upto, kProducerThreads, s_b + bs * P::B, s_cb + bs * (P::CB / 4), &s_cmax[bs][0][0]);
                    done = upto;
                }
            }
            if (todo > 0 && !failed) built(then);
            o = then;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp != kWarpIssue) {
        // ---- scores -> codes: one row per thread ----
        const int group = (warp - kWarpIssue - 1) >> 2, quad = warp & 3, row = quad * 32 + lane;   // the tensor-memory lanes this warp may read
        const uint32_t col0 = tmem + ((uint32_t)(quad * 32) << 16);
        const bool words = SPA == 4 && g.m % 4 == 0 && (reinterpret_cast<uintptr_t>(g.codes) & 3) == 0;
        uint32_t seq0 = 0, phase = 0;   // accumulators before this turn; bit a: the phase of this group's barrier of accumulator a
        for (NearItem o(g); o.live(g) && !failed; o.next(g)) {
            const int bs = (int)(o.it & 1u), nsub = o.subs<SPA>(g), ntiles = o.tiles(g);
            if (!near_wait_warp(&b_full[bs], (o.it >> 1) & 1u, abort_flag)) { failed = true; break; }
            for (int k0 = 0; k0 < ntiles && !failed; k0 += kGroups) {   // a turn: a tile for each group
                const int turn = min(kGroups, ntiles - k0), k = k0 + group;
                const uint32_t t = o.t + (uint32_t)k, slot = t % kRingX;
                if (group >= turn) { seq0 += (uint32_t)(turn * nsub); continue; }
                if (!near_wait_warp(&a_full[slot], (t / kRingX) & 1u, abort_flag)) { failed = true; break; }
                const long long at = (o.tile + k) * kTile + row;
                const bool live = at < g.n;
                const float* xtile = s_x + (size_t)slot * kTile * PITCH;
                uint32_t packed = 0;
#pragma unroll 1
                for (int sub = 0; sub < nsub; ++sub) {
                    const uint32_t acc = (seq0 + (uint32_t)(sub * turn + group)) % kAcc, col = col0 + acc * kCodes;   // in the issuer's order
                    // A barrier per group and accumulator: by the accumulator's own a group could come to wait two phases early, by the group's
                    // own (where other groups have no tile left) two phases late.
                    if (!near_wait_warp(&acc_full[group][acc], (phase >> acc) & 1u, abort_flag)) { failed = true; break; }
                    phase ^= 1u << acc;
                    tc_fence_after();
                    float gm[32];   // the largest score of every eight codewords
                    auto fold = [&](const uint32_t (&v)[32], int b) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t* w = v + 8 * i;
                            const float a = fmaxf(fmaxf(__uint_as_float(w[0]), __uint_as_float(w[1])), __uint_as_float(w[2]));
                            const float c = fmaxf(fmaxf(__uint_as_float(w[3]), __uint_as_float(w[4])), __uint_as_float(w[5]));
                            const float e = fmaxf(fmaxf(__uint_as_float(w[6]), __uint_as_float(w[7])), a);
                            gm[4 * b + i] = fmaxf(e, c);
                        }
                    };
                    uint32_t va[32], vb[32];
                    tmem_ld32(col, va);
#pragma unroll
                    for (int b = 0; b < 8; b += 2) {   // two loads in flight: the next 32 columns arrive while these are folded
                        tmem_ld_wait();
                        tmem_ld32(col + 32 * (b + 1), vb);
                        fold(va, b);
                        tmem_ld_wait();
                        if (b + 2 < 8) tmem_ld32(col + 32 * (b + 2), va);
                        else { tc_fence_before(); __syncwarp(); if (lane == 0) near_arrive(&acc_empty[acc]); }   // all scores are in registers
                        fold(vb, b + 1);
                    }
                    float x[D], xn = 0.0f;
                    load_row<D>(x, xtile, row, sub);
#pragma unroll
                    for (int d = 0; d < D; ++d) xn = fmaf(x[d], x[d], xn);
                    float part[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        part[i] = fmaxf(fmaxf(gm[8 * i], gm[8 * i + 1]), gm[8 * i + 2]);
                        part[i] = fmaxf(fmaxf(gm[8 * i + 3], gm[8 * i + 4]), part[i]);
                        part[i] = fmaxf(fmaxf(gm[8 * i + 5], gm[8 * i + 6]), part[i]);
                    }
                    const float mx = fmaxf(fmaxf(fmaxf(fmaxf(part[0], gm[7]), part[1]), fmaxf(fmaxf(gm[15], part[2]), gm[23])), fmaxf(part[3], gm[31]));
                    unsigned top = 0;
#pragma unroll
                    for (int i = 0; i < kCodes / 32; ++i) top = max(top, __float_as_uint(s_cmax[bs][sub][i]));
                    const float cmax = near_root(__uint_as_float(top)), nx = near_root(xn), both = nx + cmax;
                    const float thr = mx - (3.0517578125e-5f * nx * cmax + (float)(KS + 1) * 3.814697265625e-6f * both * both + kTiny);
                    uint32_t below[4] = {0, 0, 0, 0};   // bit 31 - u of all: group u lies below the threshold
#pragma unroll
                    for (int u = 0; u < 8; ++u)
#pragma unroll
                        for (int i = 0; i < 4; ++i) below[i] = __funnelshift_l(__float_as_uint(gm[8 * i + u] - thr), below[i], 1);
                    uint32_t hit = ~((below[0] << 24) | (below[1] << 16) | (below[2] << 8) | below[3]);
                    if (!(fabsf(thr) <= 0.9f * kFarNorm)) hit = 0xffffffffu;   // a product or a norm overflowed or is not a number, or the codewords past k came first: evaluate everything
                    if (!live) hit = 0u;
                    const float* cb = s_cb + (size_t)(bs * SPA + sub) * kCodes * D;
                    float best = FLT_MAX;
                    int code = 0;
                    while (hit) {
                        const int u = __clz((int)hit);
                        hit &= ~(0x80000000u >> u);
                        // a lane's order is its own: the eight lanes of a request read eight different sixteenths of the banks
                        float dist[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            float c[D];
                            load_vec<D>(c, cb + ((8 * u + (lane & 7)) ^ j) * D);
                            dist[j] = near_dist<D, kTrain>(x, c);
                        }
                        const float near = fminf(fminf(fminf(fminf(dist[0], dist[1]), dist[2]), fminf(fminf(dist[3], dist[4]), dist[5])), fminf(dist[6], dist[7]));
                        int first = 7;
#pragma unroll
                        for (int j = 0; j < 8; ++j) first = min(first, dist[j] == near ? (lane & 7) ^ j : 7);
                        if (near < best) { best = near; code = 8 * u + first; }
                    }
                    __syncwarp();
                    if (words) packed |= (uint32_t)code << (8 * sub);
                    else if (live) g.codes[(size_t)at * g.m + o.atom * SPA + sub] = (uint8_t)code;
                }
                if (failed) break;
                seq0 += (uint32_t)(turn * nsub);
                if (lane == 0) near_arrive(&x_empty[slot]);
                if (words && live) *reinterpret_cast<uint32_t*>(g.codes + (size_t)at * g.m + o.atom * SPA) = packed;
            }
            if (failed) break;
            __syncwarp();
            if (lane == 0) near_arrive(&b_empty[bs]);
        }
    } else {
        // ---- issuer (the whole warp keeps step, one lane issues: what is the same for all lanes stays in uniform registers): the sub-quantisers of a turn's tiles one after the other, each product into the next accumulator ----
        const bool elected = elect_one();
        const uint32_t idesc = idesc_bf16(kTile, kCodes);
        const uint64_t da0 = make_sw128_desc(smem_u32(s_a)), db0 = make_sw128_desc(smem_u32(s_b));   // the address field counts 16-byte units
        uint32_t seq = 0;
        for (NearItem o(g); o.id < g.issued && !failed; o.next(g)) {
            const int nsub = o.subs<SPA>(g), ntiles = o.tiles(g);
            const uint32_t bs = o.it & 1u;
            if (!near_wait_warp(&b_full[bs], (o.it >> 1) & 1u, abort_flag)) { failed = true; break; }
            for (int k0 = 0; k0 < ntiles && !failed; k0 += kGroups) {
                const int turn = min(kGroups, ntiles - k0);
                for (int sub = 0; sub < nsub && !failed; ++sub)
                    for (int p = 0; p < turn; ++p, ++seq) {
                        const uint32_t t = o.t + (uint32_t)(k0 + p), slot = t % kRingA, acc = seq % kAcc;
                        if ((sub == 0 && !near_wait_warp(&a_full[t % kRingX], (t / kRingX) & 1u, abort_flag)) || !near_wait_warp(&acc_empty[acc], ((seq / kAcc) & 1u) ^ 1u, abort_flag)) { failed = true; break; }
                        tc_fence_after();
                        if (elected) {
#pragma unroll
                            for (int ks = 0; ks < KS; ++ks) {
                                const uint64_t off = (uint64_t)(sub * KS + ks) * 2;   // a K step is 32 bytes
                                umma_bf16(tmem + acc * kCodes, da0 + slot * (P::A / 16) + off, db0 + bs * (P::B / 16) + off, idesc, ks ? 1u : 0u);
                            }
                            umma_commit(&acc_full[p][acc]);
                            if (sub + 1 == nsub) umma_commit(&a_empty[slot]);
                        }
                        __syncwarp();
                    }
            }
            if (!failed && elected) umma_commit(&b_empty[bs]);
            __syncwarp();
        }
        // Whether or not a wait gave up: the products issued are done before the tensor memory that they write and the operands that they read go to
        // someone else.  No other role has a part in this wait, so the flag does not end it.
        if (elected) umma_commit(&drained);
        __syncwarp();
        if (!__all_sync(0xffffffffu, mbar_wait(&drained, 0, kNearWaitLimit))) failed = true;
    }
    if (failed) *abort_flag = 1;
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kTmemCols);
    if (!s_abort) return;
    // A bounded wait gave up: the CTA's items are evaluated one codeword after the other.
    if (g.gave_up && tid == 0) atomicAdd(g.gave_up, 1);
    for (long long id = blockIdx.x; id < g.items; id += gridDim.x) {
        const int atom = (int)(id % g.atoms), nsub = min(SPA, g.m - atom * SPA);
        const long long r0 = id / g.atoms * g.per * kTile, r1 = min(g.n, r0 + (long long)g.per * kTile);
        for (long long e = tid; e < (r1 - r0) * nsub; e += kThreads) {
            const long long row = r0 + e / nsub;
            const int sub = atom * SPA + (int)(e % nsub);
            float x[D], c[D], best = FLT_MAX;
            int code = 0;
            for (int d = 0; d < D; ++d) x[d] = g.data[(size_t)row * g.dim + (size_t)sub * D + d];
            for (int j = 0; j < g.k; ++j) {
                for (int d = 0; d < D; ++d) c[d] = g.codebook[((size_t)sub * g.k + j) * D + d];
                const float dist = near_dist<D, kTrain>(x, c);
                if (dist < best) { best = dist; code = j; }
            }
            g.codes[(size_t)row * g.m + sub] = (uint8_t)code;
        }
    }
}

template <int D, bool kTrain>
psb_status run_nearest(const float* d_data, long long n, int dim, const float* d_codebook, int m, int k, uint8_t* d_codes, int sm_count, cudaStream_t s,
                       const NearTest& test) {
    using P = Near<D>;
    NearArgs g;
    g.data = d_data; g.codebook = d_codebook; g.codes = d_codes; g.n = n; g.dim = dim; g.m = m; g.k = k;
    g.atoms = (m + P::SPA - 1) / P::SPA;
    g.tiles = (n + kTile - 1) / kTile;
    // Items as large as leave every SM one, up to kMaxTiles tiles; more than one turn: whole turns.
    g.per = (int)std::max<long long>(1, std::min<long long>(kMaxTiles, (g.tiles * g.atoms + sm_count - 1) / sm_count));
    if (g.per > kGroups) {
        // Of the whole turns those that end soonest: rounds of items over the SMs, each its tiles and three quarters of one for its codewords.  150,000 rows, sub-vectors of
        // 4, two atoms: items of fifteen are 158 for 148 SMs, 81 us, of nine 53.
        double least = 0.0;
        for (int per = kGroups; per <= kMaxTiles; per += kGroups) {
            const long long rounds = ((g.tiles + per - 1) / per * g.atoms + sm_count - 1) / sm_count;
            const double cost = (double)rounds * (per + 0.75);
            if (least == 0.0 || cost <= least) { least = cost; g.per = per; }
        }
    }
    g.items = (g.tiles + g.per - 1) / g.per * g.atoms;
    const unsigned grid = (unsigned)std::min<long long>(g.items, sm_count);
    g.step_atom = (int)(grid % (unsigned)g.atoms); g.step_tiles = (long long)(grid / (unsigned)g.atoms) * g.per;
    g.issued = test.items >= 0 ? std::min<long long>(test.items, g.items) : g.items; g.gave_up = test.gave_up;
    g.vec = dim % P::V == 0 && reinterpret_cast<uintptr_t>(d_data) % (4 * P::V) == 0 ? 1 : 0;
    PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_pq_nearest<D, kTrain>), P::SMEM));
    k_pq_nearest<D, kTrain><<<grid, kThreads, P::SMEM, s>>>(g);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

}  // namespace

// The filter's operands hold 16 dimensions at most, and it pays from about 32 codewords on.
bool pq_nearest_supported(int dsub, int k, bool train) {
    if (k <= 32 || k > kCodes) return false;
    if (train) return dsub == 2 || dsub == 4 || dsub == 8;
    return (dsub >= 2 && dsub <= 6) || dsub == 8 || dsub == 10 || dsub == 12 || dsub == 16;
}

psb_status launch_pq_nearest(const float* d_data, long long n, int dim, const float* d_codebook, int m, int k, bool train, uint8_t* d_codes, int sm_count,
                             cudaStream_t s, const NearTest& test) {
    if (n <= 0) return PSB_OK;
    if (train) {
        switch (dim / m) {
            case 2: return run_nearest<2, true>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            case 4: return run_nearest<4, true>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            case 8: return run_nearest<8, true>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            default: break;
        }
    } else {
        switch (dim / m) {
            case 2: return run_nearest<2, false>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            case 3: return run_nearest<3, false>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            case 4: return run_nearest<4, false>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            case 5: return run_nearest<5, false>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            case 6: return run_nearest<6, false>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            case 8: return run_nearest<8, false>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            case 10: return run_nearest<10, false>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            case 12: return run_nearest<12, false>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            case 16: return run_nearest<16, false>(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s, test);
            default: break;
        }
    }
    return fail(PSB_INTERNAL, "sub-vector length without a filter");
}

}  // namespace psb
