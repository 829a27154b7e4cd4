// Coarse stage, tensor-core part: a bf16 tcgen05 GEMM (queries x centroids, fp32 accumulators in tensor memory,
// operands staged in shared memory by TMA) whose epilogue folds in the centroid norms and filters - it never
// writes the distance matrix.  Two passes over the same GEMM:
//   pass 1  epilogue keeps, per query and per group of G consecutive centroids, the minimum approximate distance
//           a = |c'|^2 - 2 q'.c'  (q', c' = inputs minus the mean centroid, rounded to bf16).  The nprobe-th smallest
//           group minimum T is an upper bound of the nprobe-th smallest approximate distance.
//   pass 2  epilogue appends every centroid with a <= T + 2E to the query's candidate list, E >= |a - exact|.
//           Every centroid of the exact top-nprobe is then a candidate: the nprobe approximately-nearest have exact
//           distance <= T + E, so the exact nprobe-th distance is <= T + E and its members have a <= T + 2E.
// E comes from the rounding that happened, not from the format's worst case: with qb, cb the bf16 operands,
//     |q'.c' - qb.cb| <= |q' - qb| |c'| + |qb| |c' - cb|,   E = 2 (|q' - qb| max|c'| + |qb| max|c' - cb|) plus fp32 slack,
// four to five times below 2^-7 |q'| max|c'|.
// k_coarse_refine re-scores the candidates (typically 1.1-1.3 x nprobe) in the CPU path's arithmetic (sequential
// non-fused fp32, reference src/cpu/utils/cpu_distance.h:74-81) and sorts by (distance, id): results are bit-identical
// to the exact kernels in coarse.cu.  A query whose list overflowed is redone by k_coarse_exact_query.
//
// Reference counterpart: the fused fp16 GEMM + threshold admission + exact top-nprobe of
// src/search/kernels/coarse/runtime/kernels/wmma_body.cuh:45-248 and coarse_runtime.cu:121-149 (wmma, SM 12.0 only).
//
// Every wait on an mbarrier is bounded: after kWaitLimit polls the CTA raises a status word, releases its tensor
// memory and returns, and the host reports PSB_TIMEOUT.
#include <cuda.h>
#include <cuda_bf16.h>

#include "common.cuh"
#include "kernels.h"
#include "tc_ptx.cuh"

namespace psb {
namespace {

using namespace tc;

constexpr int TQ = 128;          // queries per tile  (UMMA M)
constexpr int TCOL = 256;        // centroids per tile (UMMA N)
constexpr int KATOM = 64;        // bf16 elements per 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int kCandCap = 2048;

// kind::f16 instruction descriptor: D fp32, A and B bf16, both K-major, M = 128, N = 256.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TCOL >> 3) << 17) | ((uint32_t)(TQ >> 4) << 24);

// Per group of G consecutive values of a 32-value chunk: out = -2 * max(w), i.e. the minimum of a = -2 w.
template <int G>
__device__ __forceinline__ void group_mins(const float (&v)[32], float* __restrict__ out, size_t stride) {
#pragma unroll
    for (int g = 0; g < 32 / G; ++g) {
        float t[G];
#pragma unroll
        for (int j = 0; j < G; ++j) t[j] = v[g * G + j];
#pragma unroll
        for (int w = G / 2; w >= 1; w >>= 1)  // pairwise tree: short dependency chains
#pragma unroll
            for (int j = 0; j < w; ++j) t[j] = fmaxf(t[j], t[j + w]);
        out[g * stride] = -2.0f * t[0];
    }
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float m;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    return m;
}
template <int FROM>
__device__ __forceinline__ float max8(const float (&v)[32]) {   // of eight values
    return fmaxf(max3(max3(v[FROM], v[FROM + 1], v[FROM + 2]), v[FROM + 3], v[FROM + 4]), max3(v[FROM + 5], v[FROM + 6], v[FROM + 7]));
}

__device__ __forceinline__ void add_f32x2(float& o0, float& o1, float a0, float a1, float b0, float b1) {
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(o0), "=f"(o1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

struct TcArgs {
    const int* nq_dev;      // when set: the number of rows is min(*nq_dev, nq), known on the device only
    int nq, nlist, katoms;  // katoms = padded dim / 64
    int ntiles;             // centroid tiles of TCOL
    int group;              // G: centroids per minimum in pass 1 (power of two <= 32)
    int lg_group;           // log2(G)
    int ngroups;            // minima per query row = ntiles * (TCOL / G)
    int nprobe;
    const float* cn2;       // [ntiles * TCOL] |c'|^2, +inf beyond nlist
    const float2* qnorm;    // [nq] |q'| and |q' - qb|
    const float* cmax;      // [2] max |c'| and max |c' - cb|
    float* gmin;            // pass 1 out: the minimum of row q and group g at [q * gmin_q + g * gmin_g]
    int gmin_q, gmin_g;
    const float* seltop;    // pass 2 in: [nq][nprobe] ascending group minima (T = last)
    uint32_t* mask;         // pass 2 out: [nq][mwords] one bit per centroid (zeroed before the launch; only non-zero words are written)
    int mwords;             // ntiles * TCOL / 32
    int* status;            // [1] != 0 after a bounded wait gave up
    int cblocks, qtiles;    // work = cblocks (512 centroids each) x qtiles (128 queries each) tile pairs
    int* cand_cnt;          // pass 2, list form (nearest-centroid assignment with a known bound): [nq] candidates found so far
    int* cand_list;         //   [nq][cand_cap] their ids; null: the bit mask above is written instead
    int cand_cap;
    float band;             // pass 2: cut = T + band * E; 2, or 1 when T bounds the exact distance itself (a previous assignment)
    int wait_limit;         // polls before a wait gives up (0: kWaitLimit)
    uint32_t load_tiles;    // query tiles a CTA loads before its producer gives up: all, or fewer in the test of the time-out path (0: no load at all)
};

// Work split: the (centroid block, query tile) pairs are numbered block-major and CTA b takes the contiguous range
// [total * b / grid, total * (b + 1) / grid), so every CTA gets the same number of tile pairs (+-1) and reloads its
// resident centroid block at most once or twice.  A range is walked as segments of one centroid block each.
__device__ __forceinline__ void cta_range(const TcArgs& a, long long& l0, long long& l1) {
    const long long total = (long long)a.cblocks * a.qtiles;
    l0 = total * blockIdx.x / gridDim.x;
    l1 = total * (blockIdx.x + 1) / gridDim.x;
}
__device__ __forceinline__ int seg_count(const TcArgs& a, long long l0, long long l1) {
    return l1 > l0 && a.qtiles > 0 ? (int)((l1 - 1) / a.qtiles - l0 / a.qtiles) + 1 : 0;
}
__device__ __forceinline__ void seg_get(const TcArgs& a, long long l0, long long l1, int i, int& cblock, int& t0, int& t1) {
    cblock = (int)(l0 / a.qtiles) + i;
    const long long b = (long long)cblock * a.qtiles;
    t0 = (int)((l0 > b ? l0 : b) - b);
    t1 = (int)((l1 < b + a.qtiles ? l1 : b + a.qtiles) - b);
}

// Persistent, warp-specialised kernel.  A work unit = one segment of the CTA's range: (block of 512 centroids, range of query tiles).  The unit's
// two centroid tiles (B operands) stay in shared memory while query tiles (A operand, 128 rows) stream through a
// two-stage ring; each query tile is multiplied against both centroid tiles into two tensor-memory accumulators, so
// the epilogue of one accumulator overlaps the MMAs of the other.
//   warps 0-15 epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. +31 (one query row per thread) and the 64
//              columns (w / 4) * 64 .. +63 of each accumulator, 32 columns per tcgen05.ld; folds |c'|^2 in;
//              pass 1: group minima -> gmin, pass 2: compare with the row's cut-off -> candidate list.
//              Sixteen warps because the epilogue (2+ instructions per matrix element), not the MMA, sets the pace.
//   warp 16    TMA producer (one lane)
//   warp 17    MMA issuer (one lane): 2 x katoms x 4 tcgen05.mma per query tile, tcgen05.commit -> mbarriers
constexpr int kStagesA = 2;
constexpr int kEpiWarps = 16;
constexpr int kEpiThreads = kEpiWarps * 32;
constexpr int kTcThreadsV2 = kEpiThreads + 64;
constexpr int kBlockCols = 2 * TCOL;  // centroids per work unit

// kAug: the operands carry 3 extra K slots (ones on the query side, minus the three-term bf16 split of |c'|^2 / 2 on the
// centroid side), so the accumulator already holds w = q'.c' - |c'|^2 / 2 and the epilogue needs no norm arithmetic.
template <bool kSecondPass, bool kAug>
__global__ void __launch_bounds__(kTcThreadsV2, 1)
k_coarse_tc(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_c, const TcArgs args) {
    TcArgs a = args;
    if (a.nq_dev) { a.nq = min(*a.nq_dev, a.nq); a.qtiles = (a.nq + TQ - 1) / TQ; }
    extern __shared__ __align__(1024) unsigned char s_tc[];
    unsigned char* s_base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(s_tc) + 1023) & ~uintptr_t(1023));
    const size_t a_bytes = (size_t)a.katoms * TQ * 128, b_bytes = (size_t)a.katoms * TCOL * 128;
    unsigned char* s_a = s_base;                         // [kStagesA][katoms][TQ][128 B]
    unsigned char* s_b = s_base + kStagesA * a_bytes;    // [2][katoms][TCOL][128 B]
    __shared__ __align__(8) uint64_t a_full[kStagesA], a_empty[kStagesA], b_full, b_empty, acc_full[2], acc_empty[2], drained;
    __shared__ uint32_t s_tmem;
    __shared__ __align__(16) float s_cn2[kBlockCols];
    __shared__ __align__(16) float s_top[kBlockCols / 8];   // the largest s_cn2 of every eight columns
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int i = 0; i < kStagesA; ++i) { mbar_init(&a_full[i], 1); mbar_init(&a_empty[i], 1); }
        mbar_init(&b_full, 1); mbar_init(&b_empty, 1); mbar_init(&drained, 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], kEpiWarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(&s_tmem, 2 * TCOL);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    long long l0, l1;
    cta_range(a, l0, l1);
    const int nunits = seg_count(a, l0, l1);
    const int wl = a.wait_limit > 0 ? a.wait_limit : kWaitLimit;
    int failed = 0;

    if (warp == kEpiWarps) {
        if (lane == 0 && a.load_tiles) {
            uint32_t it = 0, un = 0;  // query tiles issued, units issued
            while ((int)un < nunits && !failed) {
                int cblock, t0, t1;
                seg_get(a, l0, l1, (int)un, cblock, t0, t1);
                if (!mbar_wait(&b_empty, (un & 1u) ^ 1u, wl)) { failed = 1; break; }
                mbar_expect_tx(&b_full, (uint32_t)(2 * b_bytes));
                for (int h = 0; h < 2; ++h)
                    for (int ka = 0; ka < a.katoms; ++ka)
                        tma_load_2d(s_b + h * b_bytes + (size_t)ka * TCOL * 128, &map_c, ka * KATOM, cblock * kBlockCols + h * TCOL, &b_full);
                ++un;
                for (int t = t0; t < t1; ++t, ++it) {
                    const uint32_t st = it % kStagesA;
                    if (it >= a.load_tiles || !mbar_wait(&a_empty[st], ((it / kStagesA) & 1u) ^ 1u, wl)) { failed = 1; break; }
                    mbar_expect_tx(&a_full[st], (uint32_t)a_bytes);
                    for (int ka = 0; ka < a.katoms; ++ka)
                        tma_load_2d(s_a + st * a_bytes + (size_t)ka * TQ * 128, &map_q, ka * KATOM, t * TQ, &a_full[st]);
                }
            }
            // Whether or not a wait gave up: the loads issued have landed before the CTA gives back the memory they write to.  (A barrier's phase is
            // never more than one behind its last load.)
            if (un && !mbar_wait(&b_full, (un - 1) & 1u)) failed = 1;
            for (uint32_t st = 0; st < kStagesA; ++st)
                if (it > st && !mbar_wait(&a_full[st], ((it - st - 1) / kStagesA) & 1u)) failed = 1;
        }
    } else if (warp == kEpiWarps + 1) {
        if (lane == 0) {
            uint32_t it = 0, un = 0, nacc[2] = {0, 0};
            for (; (int)un < nunits && !failed; ++un) {
                int cblock, t0, t1;
                seg_get(a, l0, l1, (int)un, cblock, t0, t1);
                (void)cblock;
                if (!mbar_wait(&b_full, un & 1u, wl)) { failed = 1; break; }
                for (int t = t0; t < t1 && !failed; ++t, ++it) {
                    const uint32_t st = it % kStagesA;
                    if (!mbar_wait(&a_full[st], (it / kStagesA) & 1u, wl)) { failed = 1; break; }
                    for (int h = 0; h < 2; ++h) {
                        if (!mbar_wait(&acc_empty[h], (nacc[h] & 1u) ^ 1u, wl)) { failed = 1; break; }
                        tc_fence_after();
                        const uint32_t sa = smem_u32(s_a + st * a_bytes), sb = smem_u32(s_b + h * b_bytes);
                        for (int ka = 0; ka < a.katoms; ++ka)
                            for (int kk = 0; kk < KATOM / UMMA_K; ++kk)
                                umma_bf16(tmem + (uint32_t)(h * TCOL), make_sw128_desc(sa + ka * TQ * 128 + kk * UMMA_K * 2),
                                          make_sw128_desc(sb + ka * TCOL * 128 + kk * UMMA_K * 2), kIdesc, (ka | kk) ? 1u : 0u);
                        umma_commit(&acc_full[h]);
                        ++nacc[h];
                    }
                    umma_commit(&a_empty[st]);  // stage reusable once both MMAs have read it
                }
                umma_commit(&b_empty);
            }
            // So it is with the products and the tensor memory.
            umma_commit(&drained);
            if (!mbar_wait(&drained, 0)) failed = 1;
        }
    } else {
        // epilogue warps
        uint32_t nacc[2] = {0, 0};
        const int quad = warp & 3, part = warp >> 2;
        const int row = quad * 32 + lane;  // tensor-memory lane = row of the current query tile
        const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32) << 16);
        for (int u = 0; u < nunits; ++u) {  // every thread passes both barriers of every unit, failed or not
            int cblock, t0, t1;
            seg_get(a, l0, l1, u, cblock, t0, t1);
            asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");  // previous unit's readers of s_cn2 are done
            for (int i = tid; i < kBlockCols; i += kEpiThreads) {
                const float n = -0.5f * a.cn2[(size_t)cblock * kBlockCols + i];
                s_cn2[i] = n;
                float top = n;
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
                if ((i & 7) == 0) s_top[i >> 3] = top;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
            for (int t = t0; t < t1 && !failed; ++t) {
                const int q = t * TQ + row;
                float cut = 0.0f;
                if (kSecondPass && q < a.nq) {
                    const float T = a.seltop[(size_t)q * a.nprobe + a.nprobe - 1];
                    const float2 qn = a.qnorm[q];
                    const float cm = a.cmax[0], ce = a.cmax[1];
                    const float E = 2.0001f * (qn.y * cm + (qn.x + qn.y) * ce);
                    cut = -0.5f * (T + a.band * E + 6e-5f * (qn.x + cm) * (qn.x + cm));  // candidates: w >= cut
                }
                const bool partial = (cblock + 1) * kBlockCols > a.nlist;  // block reaches past the last centroid
                for (int h = 0; h < 2; ++h) {
                    if (!mbar_wait(&acc_full[h], nacc[h] & 1u, wl)) { failed = 1; break; }
                    ++nacc[h];
                    tc_fence_after();
                    uint32_t r0[32], r1[32];
                    const int cb0 = part * 64;
                    __syncwarp();
                    tmem_ld32(lane_addr + (uint32_t)(h * TCOL + cb0), r0);
                    tmem_ld32(lane_addr + (uint32_t)(h * TCOL + cb0 + 32), r1);
                    tmem_ld_wait();
                    // the accumulators are in registers: hand the tensor memory back before the arithmetic
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[h])) : "memory");
                    if (q < a.nq) {
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            const int cb = cb0 + half * 32;
                            const int c0 = cblock * kBlockCols + h * TCOL + cb;
                            float v[32];  // w = q'.c' - |c'|^2 / 2 = -a / 2; -inf beyond the last centroid
                            const uint32_t* rr = half ? r1 : r0;
                            if (kAug || kSecondPass) {   // second pass without the extra slots: the norms come in below
#pragma unroll
                                for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(rr[j]);
                                if (kAug && partial) {
#pragma unroll
                                    for (int j = 0; j < 32; ++j) if (c0 + j >= a.nlist) v[j] = __int_as_float(0xff800000);
                                }
                            } else {
#pragma unroll
                                for (int j = 0; j < 32; j += 4) {   // s_cn2 holds -|c'|^2 / 2
                                    const float4 n4 = *reinterpret_cast<const float4*>(&s_cn2[h * TCOL + cb + j]);
                                    add_f32x2(v[j], v[j + 1], __uint_as_float(rr[j]), __uint_as_float(rr[j + 1]), n4.x, n4.y);
                                    add_f32x2(v[j + 2], v[j + 3], __uint_as_float(rr[j + 2]), __uint_as_float(rr[j + 3]), n4.z, n4.w);
                                }
                            }
                            if (!kSecondPass) {
                                float* out = a.gmin + (size_t)q * a.gmin_q + (size_t)(c0 >> a.lg_group) * a.gmin_g;
                                switch (a.lg_group) {  // uniform
                                    case 5: out[0] = -2.0f * fmaxf(max3(max8<0>(v), max8<8>(v), max8<16>(v)), max8<24>(v)); break;
                                    case 4: group_mins<16>(v, out, a.gmin_g); break;
                                    case 3: group_mins<8>(v, out, a.gmin_g); break;
                                    case 2: group_mins<4>(v, out, a.gmin_g); break;
                                    case 1: group_mins<2>(v, out, a.gmin_g); break;
                                    default: group_mins<1>(v, out, a.gmin_g); break;
                                }
                            } else {
                                // one bit per centroid of this 32-column chunk; most chunks hold none, which their maximum tells in a
                                // quarter of the instructions the bits take, and so it is with the eighths of a chunk that does
                                // (without the extra slots: their largest sum q'.c' and largest norm term bound it from above;
                                // six iterations over 400,000 x 8,192 x 128 took 5,042 us when every sum got its norm first, 4,593 so)
                                float m[4] = {max8<0>(v), max8<8>(v), max8<16>(v), max8<24>(v)};
                                if (!kAug) {
                                    const float4 top = *reinterpret_cast<const float4*>(&s_top[(h * TCOL + cb) >> 3]);
                                    m[0] += top.x; m[1] += top.y; m[2] += top.z; m[3] += top.w;
                                }
                                if (fmaxf(max3(m[0], m[1], m[2]), m[3]) >= cut) {
                                    uint32_t bits = 0;
#pragma unroll
                                    for (int g = 0; g < 4; ++g) {
                                        if (m[g] < cut) continue;
#pragma unroll
                                        for (int j = 8 * g; j < 8 * g + 8; ++j) bits |= ((kAug ? v[j] : v[j] + s_cn2[h * TCOL + cb + j]) >= cut ? 1u : 0u) << j;
                                    }
                                    if (!kAug && !bits) continue;
                                    if (a.cand_list) {   // a handful of candidates per row: a short list instead of a mask to scan
                                        while (bits) {
                                            const int j = __ffs((int)bits) - 1;
                                            bits &= bits - 1;
                                            const int pos = atomicAdd(&a.cand_cnt[q], 1);
                                            if (pos < a.cand_cap) a.cand_list[(size_t)q * a.cand_cap + pos] = c0 + j;
                                        }
                                    } else {
                                        a.mask[(size_t)q * a.mwords + (c0 >> 5)] = bits;
                                    }
                                }
                            }
                        }
                    }
                }
            }
        }
    }
    if (failed) atomicExch(a.status, 1);
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    if (warp == 0) tmem_dealloc(tmem, 2 * TCOL);
}

// q' = q - mu as bf16 rows padded with zeros to dimp, |q'|^2 (sq), |q'| with the rounding error |q' - qb| (norm), and the largest of
// each over all rows (maxima [2], zeroed by the caller).
// aug: 0 = no extra slots, 1 = query rows (slots dim..dim+2 hold 1), 2 = centroid rows (slots hold minus the bf16
// three-term split of |c'|^2 / 2).
__global__ void k_tc_prep_rows(const float* __restrict__ x, long long n, int dim, int dimp, const float* __restrict__ mu,
                               __nv_bfloat16* __restrict__ out, float2* __restrict__ norm, float* __restrict__ sq, float* __restrict__ maxima, int aug) {
    const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= n) return;
    float s = 0.0f, e = 0.0f;
    for (int d = lane; d < dimp; d += 32) {
        float v = 0.0f;
        if (d < dim) v = x[(size_t)row * dim + d] - mu[d];
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        if (!(aug && d >= dim && d < dim + 3)) out[(size_t)row * dimp + d] = h;
        const float r = v - __bfloat162float(h);
        s += v * v;
        e += r * r;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { s += __shfl_xor_sync(0xffffffffu, s, o); e += __shfl_xor_sync(0xffffffffu, e, o); }
    if (lane == 0) {
        const float nrm = sqrtf(s), err = sqrtf(e) * 1.0001f;
        if (norm) norm[row] = make_float2(nrm, err);
        if (sq) sq[row] = s;
        if (maxima) {   // non-negative floats order like their bits
            atomicMax(reinterpret_cast<int*>(maxima), __float_as_int(nrm * 1.0001f));
            atomicMax(reinterpret_cast<int*>(maxima) + 1, __float_as_int(err));
        }
        if (aug == 1) {
            for (int i = 0; i < 3; ++i) out[(size_t)row * dimp + dim + i] = __float2bfloat16_rn(1.0f);
        } else if (aug == 2) {
            float rest = 0.5f * s;
            for (int i = 0; i < 3; ++i) {
                const __nv_bfloat16 h = __float2bfloat16_rn(rest);
                out[(size_t)row * dimp + dim + i] = __hneg(h);
                rest -= __bfloat162float(h);
            }
        }
    }
}

// Mean of n rows, one CTA per 32 dimensions, a warp per 32nd row: the point the operands are centred on.
__global__ void __launch_bounds__(1024) k_mean_row(const float* __restrict__ x, int n, int dim, float* __restrict__ mu) {
    __shared__ double s_part[32][33];
    const int d = blockIdx.x * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
    double acc = 0.0;
    if (d < dim) for (int r = w; r < n; r += 32) acc += (double)x[(size_t)r * dim + d];
    s_part[w][threadIdx.x & 31] = acc;
    __syncthreads();
    if (w == 0 && d < dim) {
        for (int i = 1; i < 32; ++i) acc += s_part[i][threadIdx.x & 31];
        mu[d] = (float)(acc / n);
    }
}

__global__ void k_fill_inf(float* p, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = __int_as_float(0x7f800000);
}

// Per query row a value that at least k of its n <= 2048 values do not exceed - the k-th smallest or a little more - written to
// out[q * out_stride + out_stride - 1].  One warp per row, the values in registers; bisection between the row's extremes that ends
// when exactly k values lie below or after kKthRounds rounds: the filter's cut may be a little high, never low, and a
// 2^14th of the row's range is far below the band E that is added to it.  (An exact k-th smallest took 32 rounds.)
constexpr int kKthPerLane = 64, kKthRounds = 14;
// The values of a query lie `pitch` apart (pass 1 stores 32 queries' minima of a group side by side; one query's side by side made
// every 4-byte store a memory sector of its own, and those, not the products, set pass 1's pace: 298 us for 20,000 x 65,536 x 96),
// so a CTA takes eight queries, a sector, and turns them over in shared memory.
// The rounds are arithmetic at a fifth of the memory's rate, so pass 2's candidate masks (nlist bits a query, 164 MB for 20,000 x 65,536) are cleared
// by these warps meanwhile instead of by a fill of their own between the passes: 20,000 x 65,536 x 96 962 -> 945 us, 3,601 x 15,175 x 120 116 -> 112.
constexpr int kKthQueries = 8;
__global__ void __launch_bounds__(kKthQueries * 32)
k_kth_smallest(const float* __restrict__ vals, int nq, int pitch, int n, int k, float* __restrict__ out, int out_stride, uint32_t* __restrict__ mask, int mwords) {
    extern __shared__ __align__(16) float s_vals[];   // [kKthQueries][n]
    const int q0 = blockIdx.x * kKthQueries, w = threadIdx.x >> 5, lane = threadIdx.x & 31, q = q0 + w;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += kKthQueries * 32) {
        const float4* src = reinterpret_cast<const float4*>(vals + (size_t)i * pitch + q0);   // pitch is a multiple of 8
        const float4 a = __ldg(src), b = __ldg(src + 1);
        s_vals[i] = a.x; s_vals[n + i] = a.y; s_vals[2 * n + i] = a.z; s_vals[3 * n + i] = a.w;
        s_vals[4 * n + i] = b.x; s_vals[5 * n + i] = b.y; s_vals[6 * n + i] = b.z; s_vals[7 * n + i] = b.w;
    }
    __syncthreads();
    if (q >= nq) return;
    uint4* m4 = reinterpret_cast<uint4*>(mask + (size_t)q * mwords);   // mwords is a multiple of 8
    for (int i = lane; i < mwords / 4; i += 32) m4[i] = make_uint4(0u, 0u, 0u, 0u);
    float v[kKthPerLane];
    const float inf = __int_as_float(0x7f800000);
    float mn = inf, mx = -inf;
#pragma unroll
    for (int j = 0; j < kKthPerLane; ++j) {
        const int i = j * 32 + lane;
        v[j] = i < n ? s_vals[w * n + i] : inf;
        mn = fminf(mn, v[j]);
        if (v[j] < inf) mx = fmaxf(mx, v[j]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    float lo = mn, hi = mx;   // at most k values <= lo is not known yet; all finite values <= hi
    for (int it = 0; it < kKthRounds; ++it) {
        const float mid = lo + 0.5f * (hi - lo);
        int c = 0;
#pragma unroll
        for (int j = 0; j < kKthPerLane; ++j) c += v[j] <= mid ? 1 : 0;
        c = __reduce_add_sync(0xffffffffu, c);
        if (c >= k) hi = mid; else lo = mid;
        if (c == k) break;
    }
    // fewer than k finite values: no cut at all
    int c = 0;
#pragma unroll
    for (int j = 0; j < kKthPerLane; ++j) c += v[j] <= hi ? 1 : 0;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) out[(size_t)q * out_stride + out_stride - 1] = c >= k ? hi : inf;
}

// k = 1: the minimum of any number of values per query, `pitch` apart; a CTA takes 32 queries, each warp every eighth value of them.
__global__ void __launch_bounds__(256) k_row_min(const float* __restrict__ vals, int nq, const int* __restrict__ nq_dev, int pitch, int n, float* __restrict__ out) {
    __shared__ float s_min[8][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, q = blockIdx.x * 32 + lane;
    if (nq_dev) nq = min(nq, *nq_dev);
    if (blockIdx.x * 32 >= nq) return;   // uniform
    float mn = __int_as_float(0x7f800000);
    if (q < nq) {
#pragma unroll 4
        for (int i = w; i < n; i += 8) mn = fminf(mn, __ldg(vals + (size_t)i * pitch + q));
    }
    s_min[w][lane] = mn;
    __syncthreads();
    if (w == 0 && q < nq) {
        for (int i = 1; i < 8; ++i) mn = fminf(mn, s_min[i][lane]);
        out[q] = mn;
    }
}

// Distance of a centroid row to a query in the CPU path's arithmetic (sequential, non-fused); both rows 16-byte aligned when vec.
__device__ __forceinline__ float l2_sequential(const float* q, const float* c, int dim, bool vec) {
    float sum = 0.0f;
    if (vec) {
        const float4* c4 = reinterpret_cast<const float4*>(c);
        const float4* q4 = reinterpret_cast<const float4*>(q);
#pragma unroll 8
        for (int d = 0; d < dim / 4; ++d) {
            const float4 x = c4[d];
            const float4 y = q4[d];
            float diff = __fsub_rn(y.x, x.x); sum = __fadd_rn(sum, __fmul_rn(diff, diff));
            diff = __fsub_rn(y.y, x.y); sum = __fadd_rn(sum, __fmul_rn(diff, diff));
            diff = __fsub_rn(y.z, x.z); sum = __fadd_rn(sum, __fmul_rn(diff, diff));
            diff = __fsub_rn(y.w, x.w); sum = __fadd_rn(sum, __fmul_rn(diff, diff));
        }
    } else {
        for (int d = 0; d < dim; ++d) {
            const float diff = __fsub_rn(q[d], c[d]);
            sum = __fadd_rn(sum, __fmul_rn(diff, diff));
        }
    }
    return sum;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// Exact re-scoring of a query's candidates in the CPU path's arithmetic, sort by (distance, id), first nprobe out.
// 128 threads per query.  The candidates' rows come through shared memory, kRefineTile at a time, loaded whole by warps; a thread
// then walks its own row (a row per thread straight from L2 read each 32-byte sector four times over: 600 us for 20,000 queries
// x 65,536 centroids x 96, top 64).
constexpr int kRefineThreads = 128;
constexpr int kRefineTile = 64;
constexpr int kRefineFew = 2 * kRefineThreads;   // with at most this many candidates their keys leave room for more rows at a time
__host__ __device__ __forceinline__ int refine_pitch(int dim) { return (dim + 3) / 4 * 4 + 4; }   // rows spread over the banks
__global__ void __launch_bounds__(kRefineThreads)
k_coarse_refine(const float* __restrict__ queries, const float* __restrict__ centroids, int dim, int nlist, int nprobe,
                const uint32_t* __restrict__ mask, int mwords, int* __restrict__ out_ids,
                float* __restrict__ out_dist, int* __restrict__ fail_list, int* __restrict__ n_fail) {
    extern __shared__ __align__(16) unsigned char s_ref[];
    const int pitch = refine_pitch(dim);
    uint64_t* s_keys = reinterpret_cast<uint64_t*>(s_ref);                        // [kCandCap]; the low words hold the ids first
    float* s_q = reinterpret_cast<float*>(s_ref + (size_t)kCandCap * 8) + kRefineTile * pitch;   // [pitch]
    __shared__ int s_n;
    const int q = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) s_n = 0;
    for (int d = threadIdx.x; d < dim; d += kRefineThreads) s_q[d] = queries[(size_t)q * dim + d];
    __syncthreads();
    const uint4* m4 = reinterpret_cast<const uint4*>(mask + (size_t)q * mwords);   // mwords is a multiple of 16
    // the candidate bits of this query -> list of centroid ids; four loads in flight per thread
    for (int w0 = threadIdx.x; w0 < mwords / 4; w0 += 4 * kRefineThreads) {
        uint4 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = w0 + i * kRefineThreads < mwords / 4 ? __ldg(m4 + w0 + i * kRefineThreads) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t words[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
            if ((words[0] | words[1] | words[2] | words[3]) == 0u) continue;
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                uint32_t bits = words[h];
                while (bits) {
                    const int j = __ffs((int)bits) - 1;
                    bits &= bits - 1;
                    const int pos = atomicAdd(&s_n, 1);
                    if (pos < kCandCap) s_keys[pos] = (uint64_t)((w0 + i * kRefineThreads) * 128 + h * 32 + j);
                }
            }
        }
    }
    __syncthreads();
    const int n = s_n;
    if (n > kCandCap || n < nprobe) {
        if (threadIdx.x == 0) {
            fail_list[atomicAdd(n_fail, 1)] = q;
            atomicAdd(n_fail + 3, 1);  // cumulative count of queries sent to the exact per-query kernel
        }
        return;
    }
    const bool vec = (dim & 3) == 0 && (reinterpret_cast<uintptr_t>(centroids) & 15) == 0;
    // [tile][pitch]: all the candidates at once as a rule, since every tile costs a memory latency and a chain of dim additions
    float* s_row = reinterpret_cast<float*>(s_ref + (size_t)(n <= kRefineFew ? kRefineFew : kCandCap) * 8);
    const int tile = n <= kRefineFew ? min(kRefineThreads, kRefineTile + (kCandCap - kRefineFew) * 2 / pitch) : kRefineTile;
    for (int t0 = 0; t0 < n; t0 += tile) {
        const int cnt = min(tile, n - t0);
        if (vec) {
            const int n4 = dim >> 2;
            for (int i = warp; i < cnt; i += kRefineThreads / 32) {
                const float4* src = reinterpret_cast<const float4*>(centroids + (size_t)(uint32_t)s_keys[t0 + i] * dim);
                for (int d = lane; d < n4; d += 32) cp_async16(s_row + i * pitch + d * 4, src + d);   // all rows in flight at once
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        } else {
            for (int i = warp; i < cnt; i += kRefineThreads / 32) {
                const float* src = centroids + (size_t)(uint32_t)s_keys[t0 + i] * dim;
                for (int d = lane; d < dim; d += 32) s_row[i * pitch + d] = __ldg(src + d);
            }
        }
        __syncthreads();
        if (threadIdx.x < cnt) {
            const uint32_t c = (uint32_t)s_keys[t0 + threadIdx.x];
            s_keys[t0 + threadIdx.x] = make_key(l2_sequential(s_q, s_row + threadIdx.x * pitch, dim, vec), c);
        }
        __syncthreads();
    }
    if (n <= kRefineFew) {   // a key's place is the number of smaller ones: no barriers, a third of the sort's instructions
        const uint64_t k0 = threadIdx.x < n ? s_keys[threadIdx.x] : KEY_MAX;
        const uint64_t k1 = threadIdx.x + kRefineThreads < n ? s_keys[threadIdx.x + kRefineThreads] : KEY_MAX;
        int rank0 = 0, rank1 = 0;
        if (n > kRefineThreads) {
            for (int j = 0; j < n; ++j) { const uint64_t o = s_keys[j]; rank0 += o < k0 ? 1 : 0; rank1 += o < k1 ? 1 : 0; }
        } else if ((threadIdx.x & ~31) < n) {
#pragma unroll 4
            for (int j = 0; j < n; ++j) rank0 += s_keys[j] < k0 ? 1 : 0;
        }
        if (threadIdx.x < n && rank0 < nprobe) {
            out_ids[(size_t)q * nprobe + rank0] = (int)key_idx(k0);
            if (out_dist) out_dist[(size_t)q * nprobe + rank0] = key_dist(k0);
        }
        if (threadIdx.x + kRefineThreads < n && rank1 < nprobe) {
            out_ids[(size_t)q * nprobe + rank1] = (int)key_idx(k1);
            if (out_dist) out_dist[(size_t)q * nprobe + rank1] = key_dist(k1);
        }
        return;
    }
    const int np = next_pow2(n);
    for (int i = n + threadIdx.x; i < np; i += kRefineThreads) s_keys[i] = KEY_MAX;
    __syncthreads();
    block_bitonic_sort(s_keys, np);
    for (int i = threadIdx.x; i < nprobe; i += kRefineThreads) {
        out_ids[(size_t)q * nprobe + i] = (int)key_idx(s_keys[i]);
        if (out_dist) out_dist[(size_t)q * nprobe + i] = key_dist(s_keys[i]);
    }
}

// ---- nearest-centroid assignment with a bound known beforehand (Lloyd iterations after the first) -------------------------
// A row's distance to the centroid it was assigned to in the previous iteration, at that centroid's NEW position, bounds its
// distance to the nearest centroid from above.  With that bound in place of pass 1's group minimum the GEMM runs once: the
// candidates (every centroid whose bf16 estimate is within the bound plus the rounding slack - the nearest one and all its
// ties among them) go to a short per-row list, and k_coarse_refine1 picks the exact nearest in the CPU path's arithmetic.
constexpr int kAssignCap = 32;   // candidates kept per row; more: the exact per-row kernel
// seltop[row] = (bound on the squared distance) - |q'|^2, the quantity pass 2 compares a = |c'|^2 - 2 q'.c' against.  A warp takes four
// rows, so that their loads, each behind the row's previous id, are in flight together.
__global__ void __launch_bounds__(256) k_prev_bound(const float* __restrict__ rows, int n, int dim, const float* __restrict__ centroids, int nlist,
                                                    const int* __restrict__ prev, const float2* __restrict__ qnorm, float* __restrict__ seltop) {
    const int r0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 4, lane = threadIdx.x & 31;
    if (r0 >= n) return;
    const bool vec = (dim & 3) == 0 && ((reinterpret_cast<uintptr_t>(centroids) | reinterpret_cast<uintptr_t>(rows)) & 15) == 0;
    int mine = -1;
    float qn = 0.0f;
    if (lane < 4 && r0 + lane < n) { mine = prev[r0 + lane]; qn = qnorm[r0 + lane].x; if (mine < 0 || mine >= nlist) mine = -1; }
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    int c[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = __shfl_sync(0xffffffffu, mine, i);
    if (vec) {
        for (int d = lane; d < dim >> 2; d += 32) {
            float4 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (c[i] >= 0) {
                    a[i] = __ldg(reinterpret_cast<const float4*>(rows + (size_t)(r0 + i) * dim) + d);
                    b[i] = __ldg(reinterpret_cast<const float4*>(centroids + (size_t)c[i] * dim) + d);
                }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (c[i] >= 0) {
                    float diff = a[i].x - b[i].x; acc[i] = fmaf(diff, diff, acc[i]);
                    diff = a[i].y - b[i].y; acc[i] = fmaf(diff, diff, acc[i]);
                    diff = a[i].z - b[i].z; acc[i] = fmaf(diff, diff, acc[i]);
                    diff = a[i].w - b[i].w; acc[i] = fmaf(diff, diff, acc[i]);
                }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (c[i] >= 0)
                for (int d = lane; d < dim; d += 32) {
                    const float diff = __ldg(rows + (size_t)(r0 + i) * dim + d) - __ldg(centroids + (size_t)c[i] * dim + d);
                    acc[i] = fmaf(diff, diff, acc[i]);
                }
    }
    float bound = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
        if (lane == i) bound = acc[i];
    }
    // a bound, not a result: one part in 1e5 covers the different summation order
    if (lane < 4 && r0 + lane < n) seltop[r0 + lane] = mine >= 0 ? bound * (1.0f + 1e-5f) - qn * qn : __int_as_float(0x7f800000);
}
// A warp per 32 rows: their candidates (one or two each as a rule), a lane apiece, exactly (sequential non-fused fp32, the CPU path's
// arithmetic), each row's smallest (distance, id).  The lanes take the candidates of all 32 rows one after the other: with
// candidate i of every row in round i, rounds after the first kept a few lanes busy (400,000 rows x 8,192 x 128, six iterations: 1,036 -> 715 us).  The rows and the candidates' centroids pass through shared memory 32 dimensions at a time, a row's 128 bytes
// loaded by eight lanes: every line is fetched once (32 rows walked by 32 threads straight from L1 took 1.7 times as long, a warp
// per row left 30 of 32 lanes without a candidate).  No candidate or too many: the row goes on the fail list.
// index: the rows' numbers when the candidates belong to a gathered subset (*n_dev of them, at most n).
constexpr int kR1Warps = 4, kR1Pitch = 36;
__global__ void __launch_bounds__(kR1Warps * 32)
k_coarse_refine1(const float* __restrict__ rows, const float* __restrict__ centroids, int dim, int n, const int* __restrict__ n_dev,
                 const int* __restrict__ index, const int* __restrict__ cand_cnt, const int* __restrict__ cand_list,
                 int* __restrict__ out_ids, float* __restrict__ out_dist, int* __restrict__ fail_list, int* __restrict__ n_fail,
                 int* __restrict__ fail_total) {
    __shared__ __align__(16) float s_tile[kR1Warps][2][32 * kR1Pitch];
    __shared__ unsigned long long s_best[kR1Warps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (n_dev) n = min(n, *n_dev);
    const int at = (blockIdx.x * kR1Warps + warp) * 32 + lane;
    if (at - lane >= n) return;
    int r = -1, cnt = 0;
    if (at < n) {
        r = index ? index[at] : at;
        cnt = cand_cnt[at];
        if (cnt <= 0 || cnt > kAssignCap) {
            fail_list[atomicAdd(n_fail, 1)] = r;
            if (fail_total) atomicAdd(fail_total, 1);
            cnt = 0;
        }
    }
    const bool vec = (dim & 3) == 0 && ((reinterpret_cast<uintptr_t>(centroids) | reinterpret_cast<uintptr_t>(rows)) & 15) == 0;
    float* xs = s_tile[warp][0];
    float* cs = s_tile[warp][1];
    int upto = cnt;   // candidates of the rows up to this one
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
    }
    const int total = __shfl_sync(0xffffffffu, upto, 31);
    s_best[warp][lane] = KEY_MAX;
    __syncwarp();
    for (int p0 = 0; p0 < total; p0 += 32) {
        const int p = p0 + lane;
        int owner = 0;   // the row of candidate p: as many rows end at or before it
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            if (__shfl_sync(0xffffffffu, upto, owner + o - 1) <= p) owner += o;
        owner = min(owner, 31);
        const int first = __shfl_sync(0xffffffffu, upto - cnt, owner), mine = __shfl_sync(0xffffffffu, r, owner);
        const int c = p < total ? cand_list[(size_t)(at - lane + owner) * kAssignCap + p - first] : -1;
        float sum = 0.0f;
        for (int d0 = 0; d0 < dim; d0 += 32) {
            const int w = min(32, dim - d0);
            if (vec) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {   // four rows and their centroids per step, eight lanes each
                    const int o = j * 4 + (lane >> 3), v = (lane & 7) * 4;
                    const int ro = __shfl_sync(0xffffffffu, mine, o), co = __shfl_sync(0xffffffffu, c, o);
                    if (co >= 0 && v < w) {
                        *reinterpret_cast<float4*>(xs + o * kR1Pitch + v) = __ldg(reinterpret_cast<const float4*>(rows + (size_t)ro * dim + d0 + v));
                        *reinterpret_cast<float4*>(cs + o * kR1Pitch + v) = __ldg(reinterpret_cast<const float4*>(centroids + (size_t)co * dim + d0 + v));
                    }
                }
            } else {
                for (int o = 0; o < 32; ++o) {
                    const int ro = __shfl_sync(0xffffffffu, mine, o), co = __shfl_sync(0xffffffffu, c, o);
                    if (co >= 0 && lane < w) {
                        xs[o * kR1Pitch + lane] = __ldg(rows + (size_t)ro * dim + d0 + lane);
                        cs[o * kR1Pitch + lane] = __ldg(centroids + (size_t)co * dim + d0 + lane);
                    }
                }
            }
            __syncwarp();
            if (c >= 0) {
                const float* x = xs + lane * kR1Pitch;
                const float* y = cs + lane * kR1Pitch;
                if (w == 32) {
#pragma unroll
                    for (int d = 0; d < 32; d += 4) {
                        const float4 a = *reinterpret_cast<const float4*>(x + d), b = *reinterpret_cast<const float4*>(y + d);
                        float diff = __fsub_rn(a.x, b.x); sum = __fadd_rn(sum, __fmul_rn(diff, diff));
                        diff = __fsub_rn(a.y, b.y); sum = __fadd_rn(sum, __fmul_rn(diff, diff));
                        diff = __fsub_rn(a.z, b.z); sum = __fadd_rn(sum, __fmul_rn(diff, diff));
                        diff = __fsub_rn(a.w, b.w); sum = __fadd_rn(sum, __fmul_rn(diff, diff));
                    }
                } else {
                    for (int d = 0; d < w; ++d) { const float diff = __fsub_rn(x[d], y[d]); sum = __fadd_rn(sum, __fmul_rn(diff, diff)); }
                }
            }
            __syncwarp();
        }
        if (c >= 0) atomicMin(&s_best[warp][owner], (unsigned long long)make_key(sum, (uint32_t)c));
    }
    __syncwarp();
    const uint64_t key = s_best[warp][lane];
    if (cnt > 0) {
        out_ids[r] = (int)key_idx(key);
        if (out_dist) out_dist[r] = key_dist(key);
    }
}

// The operands of the rows on the fail list, gathered for a two-pass search of their own; rows beyond `cap` go straight to `rest`.
__global__ void k_gather_failed(const int* __restrict__ fail_list, const int* __restrict__ n_fail, int cap, const uint4* __restrict__ qb,
                                const float2* __restrict__ qnorm, int row16, uint4* __restrict__ qb_out, float2* __restrict__ qnorm_out,
                                int* __restrict__ rest, int* __restrict__ n_rest) {
    const int n = *n_fail, lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
        const int r = fail_list[i];
        if (i >= cap) { if (lane == 0) rest[atomicAdd(n_rest, 1)] = r; continue; }
        if (lane < row16) qb_out[(size_t)i * row16 + lane] = qb[(size_t)r * row16 + lane];
        if (lane == 0) qnorm_out[i] = qnorm[r];
    }
}

// Whole-row exact coarse search for the queries on the fail list: running cut-off buffer, one CTA per query.
constexpr int kExactThreads = 1024;
__global__ void __launch_bounds__(kExactThreads)
k_coarse_exact_query(const float* __restrict__ queries, const float* __restrict__ centroids, int dim, int nlist,
                     int nprobe, int buf_n, const int* __restrict__ fail_list, const int* __restrict__ n_fail,
                     int* __restrict__ cursor, int* __restrict__ out_ids, float* __restrict__ out_dist) {
    extern __shared__ __align__(16) unsigned char s_ex[];
    uint64_t* s_keys = reinterpret_cast<uint64_t*>(s_ex);                 // [buf_n]
    float* s_q = reinterpret_cast<float*>(s_ex + (size_t)buf_n * 8);     // [dim]
    __shared__ int s_cnt, s_idx;
    __shared__ uint64_t s_cut;
    const int nf = *n_fail;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_idx = atomicAdd(cursor, 1);
        __syncthreads();
        if (s_idx >= nf) return;
        const int q = fail_list[s_idx];
        for (int d = threadIdx.x; d < dim; d += blockDim.x) s_q[d] = queries[(size_t)q * dim + d];
        if (threadIdx.x == 0) { s_cnt = 0; s_cut = KEY_MAX; }
        __syncthreads();
        for (int base = 0; base < nlist; base += blockDim.x) {
            const int c_now = s_cnt;
            __syncthreads();
            if (c_now + (int)blockDim.x > buf_n) {  // uniform
                for (int i = c_now + threadIdx.x; i < buf_n; i += blockDim.x) s_keys[i] = KEY_MAX;
                __syncthreads();
                block_bitonic_sort(s_keys, buf_n);
                if (threadIdx.x == 0) { s_cnt = nprobe; s_cut = s_keys[nprobe - 1]; }  // c_now >= nprobe here
                __syncthreads();
            }
            const int c = base + threadIdx.x;
            if (c < nlist) {
                const float* cp = centroids + (size_t)c * dim;
                float sum = 0.0f;
                for (int d = 0; d < dim; ++d) {
                    const float diff = __fsub_rn(s_q[d], __ldg(cp + d));
                    sum = __fadd_rn(sum, __fmul_rn(diff, diff));
                }
                const uint64_t key = make_key(sum, (uint32_t)c);
                if (key < s_cut) s_keys[atomicAdd(&s_cnt, 1)] = key;
            }
            __syncthreads();
        }
        const int c = s_cnt;
        for (int i = c + threadIdx.x; i < buf_n; i += blockDim.x) s_keys[i] = KEY_MAX;
        __syncthreads();
        block_bitonic_sort(s_keys, buf_n);
        for (int i = threadIdx.x; i < nprobe; i += blockDim.x) {
            const uint64_t key = s_keys[i];
            const bool ok = key != KEY_MAX;
            out_ids[(size_t)q * nprobe + i] = ok ? (int)key_idx(key) : -1;
            if (out_dist) out_dist[(size_t)q * nprobe + i] = ok ? key_dist(key) : FLT_MAX;
        }
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

psb_status encode_rows_map(CUtensorMap* map, const void* base, long long rows, int dimp, int box_rows) {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        PSB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres));
        if (!p || qres != cudaDriverEntryPointSuccess) return fail(PSB_CUDA_ERROR, "cuTensorMapEncodeTiled is not available");
        fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    const cuuint64_t gdim[2] = {(cuuint64_t)dimp, (cuuint64_t)rows};
    const cuuint64_t gstride[1] = {(cuuint64_t)dimp * 2};
    const cuuint32_t box[2] = {(cuuint32_t)KATOM, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), gdim, gstride, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(PSB_CUDA_ERROR, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
    return PSB_OK;
}

}  // namespace

int coarse_tc_padded_dim(int dim) { return (dim + KATOM - 1) / KATOM * KATOM; }
int coarse_tc_tiles(int nlist) { return (nlist + kBlockCols - 1) / kBlockCols * 2; }  // whole 512-centroid blocks
int coarse_tc_list_cap() { return kAssignCap; }
int coarse_tc_retry_rows() { return 65536; }
int coarse_tc_pitch(int nq) { return (nq + 7) / 8 * 8; }
int coarse_tc_mask_words(int nlist) { return coarse_tc_tiles(nlist) * TCOL / 32; }

int coarse_tc_group(int nlist, int nprobe) {
    int g = 32;
    while (g > 1 && nlist / g < 4 * nprobe) g >>= 1;
    return g;
}

bool coarse_tc_supported(int nq, int nlist, int dim, int nprobe) {
    const int dimp = coarse_tc_padded_dim(dim);
    return nq >= 64 && nlist >= 1024 && dimp <= 128 && nprobe <= 512 && nlist >= 8 * nprobe &&
           nlist / coarse_tc_group(nlist, nprobe) >= 4 * nprobe;
}

psb_status launch_mean_row(const float* d_rows, int n, int dim, float* d_mu, cudaStream_t s) {
    k_mean_row<<<(dim + 31) / 32, 1024, 0, s>>>(d_rows, n, dim, d_mu);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_tc_prep_centroids(const float* d_centroids, int nlist, int dim, const float* d_mu, void* d_cb,
                                    float* d_cn2, float* d_maxima, cudaStream_t s) {
    const int dimp = coarse_tc_padded_dim(dim);
    const long long padded = (long long)coarse_tc_tiles(nlist) * TCOL;
    if (padded > nlist) {
        k_fill_inf<<<(unsigned)((padded - nlist + 255) / 256), 256, 0, s>>>(d_cn2 + nlist, padded - nlist);
        count_launch();
        PSB_LAUNCH_CHECK();
    }
    PSB_CUDA(cudaMemsetAsync(d_maxima, 0, 2 * sizeof(float), s));
    k_tc_prep_rows<<<(unsigned)(((long long)nlist * 32 + 255) / 256), 256, 0, s>>>(d_centroids, nlist, dim, dimp, d_mu,
                                                            static_cast<__nv_bfloat16*>(d_cb), nullptr, d_cn2, d_maxima,
                                                            dimp - dim >= 3 ? 2 : 0);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_tc_prep_queries(const CoarseTcIndex& ix, const float* d_rows, long long n, void* d_qb, void* d_qnorm, cudaStream_t s) {
    const int dimp = coarse_tc_padded_dim(ix.dim);
    k_tc_prep_rows<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(d_rows, n, ix.dim, dimp, ix.mu, static_cast<__nv_bfloat16*>(d_qb),
                                                                     static_cast<float2*>(d_qnorm), nullptr, nullptr, dimp - ix.dim >= 3 ? 1 : 0);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

namespace {
// The kernel arguments both entry points share, the tensor maps and the launch shape.
struct TcPlan {
    TcArgs a;
    CUtensorMap map_q, map_c;
    size_t smem;
    unsigned grid;
    bool aug;
};
psb_status plan_tc(const CoarseTcIndex& ix, const CoarseTcWorkspace& ws, int nq, int nprobe, int group, int sm_count, TcPlan* pl) {
    const int dimp = coarse_tc_padded_dim(ix.dim);
    TcArgs& a = pl->a;
    a.nq_dev = nullptr; a.nq = nq; a.nlist = ix.nlist; a.katoms = dimp / KATOM; a.ntiles = coarse_tc_tiles(ix.nlist);
    a.group = group; a.ngroups = a.ntiles * (TCOL / group);
    a.lg_group = 0;
    while ((1 << a.lg_group) < group) ++a.lg_group;
    a.nprobe = nprobe; a.cn2 = ix.cn2; a.qnorm = static_cast<const float2*>(ws.qnorm); a.cmax = ix.cmax; a.gmin = ws.gmin; a.seltop = ws.seltop;
    a.mwords = coarse_tc_mask_words(ix.nlist); a.status = ws.status;
    a.mask = nullptr; a.cand_cnt = nullptr; a.cand_list = nullptr; a.cand_cap = 0; a.band = 2.0f;
    a.wait_limit = ws.test_wait_limit; a.load_tiles = ws.test_load_tiles >= 0 ? (uint32_t)ws.test_load_tiles : 0xffffffffu;
    a.gmin_q = 1; a.gmin_g = coarse_tc_pitch(nq);
    a.qtiles = (nq + TQ - 1) / TQ;
    a.cblocks = a.ntiles / 2;
    pl->aug = dimp - ix.dim >= 3;
    pl->smem = (size_t)a.katoms * (kStagesA * TQ + 2 * TCOL) * 128 + 1024;
    const long long pairs = (long long)a.cblocks * a.qtiles;
    pl->grid = (unsigned)(pairs < sm_count ? pairs : sm_count);
    PSB_TRY(encode_rows_map(&pl->map_q, ws.qb, nq, dimp, TQ));
    return encode_rows_map(&pl->map_c, ix.cb, ix.nlist, dimp, TCOL);
}
template <bool kSecondPass>
psb_status run_tc(const TcPlan& pl, cudaEvent_t begin, cudaEvent_t end, cudaStream_t s) {
    auto go = [&](auto kernel) -> psb_status {
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(kernel), pl.smem));
        if (begin) PSB_CUDA(cudaEventRecord(begin, s));
        kernel<<<pl.grid, kTcThreadsV2, pl.smem, s>>>(pl.map_q, pl.map_c, pl.a);
        if (end) PSB_CUDA(cudaEventRecord(end, s));
        return PSB_OK;
    };
    if (pl.aug) PSB_TRY(go(k_coarse_tc<kSecondPass, true>));
    else PSB_TRY(go(k_coarse_tc<kSecondPass, false>));
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}
// Queries whose candidates overflowed, one CTA each.
psb_status run_exact_queries(const CoarseTcIndex& ix, const CoarseTcWorkspace& ws, const float* d_queries, int nprobe, int* d_ids, float* d_dist,
                             int sm_count, cudaStream_t s) {
    int buf_n = 2048;
    while (buf_n < nprobe + kExactThreads) buf_n <<= 1;
    const size_t esmem = (size_t)buf_n * 8 + (size_t)ix.dim * sizeof(float);
    if (esmem > 32 * 1024)
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_coarse_exact_query), esmem));
    k_coarse_exact_query<<<sm_count, kExactThreads, esmem, s>>>(d_queries, ix.centroids, ix.dim, ix.nlist, nprobe, buf_n,
                                                                ws.fail_list, ws.n_fail, ws.fail_cursor ? ws.fail_cursor : ws.n_fail + 1, d_ids, d_dist);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}
psb_status run_refine1(const CoarseTcIndex& ix, const CoarseTcWorkspace& ws, const float* d_rows, int n, const int* n_dev, const int* index,
                       int* d_ids, float* d_dist, int* fail_list, int* n_fail, int* fail_total, cudaStream_t s) {
    k_coarse_refine1<<<(unsigned)((n + kR1Warps * 32 - 1) / (kR1Warps * 32)), kR1Warps * 32, 0, s>>>(
        d_rows, ix.centroids, ix.dim, n, n_dev, index, ws.cand_cnt, ws.cand, d_ids, d_dist, fail_list, n_fail, fail_total);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}
// Pass 2 with short candidate lists, one or two per row, and the exact nearest of each row (nprobe 1).
psb_status nearest_by_lists(const CoarseTcIndex& ix, const CoarseTcWorkspace& ws, TcPlan& pl, const float* d_rows, int nq, float band, int* d_ids,
                            float* d_dist, int* fail_total, cudaStream_t s) {
    pl.a.cand_cnt = ws.cand_cnt; pl.a.cand_list = ws.cand; pl.a.cand_cap = kAssignCap; pl.a.band = band;
    PSB_CUDA(cudaMemsetAsync(ws.cand_cnt, 0, sizeof(int) * (size_t)nq, s));
    PSB_TRY(run_tc<true>(pl, ws.ev[2], ws.ev[3], s));
    return run_refine1(ix, ws, d_rows, nq, nullptr, nullptr, d_ids, d_dist, ws.fail_list, ws.n_fail, fail_total, s);
}
}  // namespace

psb_status launch_coarse_tc(const CoarseTcIndex& ix, const CoarseTcWorkspace& ws, const float* d_queries, int nq,
                            int nprobe, int* d_ids, float* d_dist, int sm_count, cudaStream_t s) {
    if (nq <= 0) return PSB_OK;
    // query side: centre, round to bf16, norms
    if (!ws.queries_ready) PSB_TRY(launch_tc_prep_queries(ix, d_queries, nq, ws.qb, ws.qnorm, s));
    TcPlan pl;
    PSB_TRY(plan_tc(ix, ws, nq, nprobe, coarse_tc_group(ix.nlist, nprobe), sm_count, &pl));
    PSB_CUDA(cudaMemsetAsync(ws.n_fail, 0, 2 * sizeof(int), s));  // n_fail, cursor
    const int ngroups = pl.a.ngroups;
    const bool own_kth = ngroups <= kKthPerLane * 32;
    if (nprobe > 1 && !own_kth) { pl.a.gmin_q = ngroups; pl.a.gmin_g = 1; }   // the general row selection wants rows
    PSB_TRY(run_tc<false>(pl, ws.ev[0], ws.ev[1], s));
    // pass 2 needs only T = an upper bound of the nprobe-th smallest group minimum of each query
    if (nprobe == 1) {
        k_row_min<<<(unsigned)((nq + 31) / 32), 256, 0, s>>>(ws.gmin, nq, nullptr, pl.a.gmin_g, ngroups, ws.seltop);
        count_launch();
        PSB_LAUNCH_CHECK();
        PSB_TRY(nearest_by_lists(ix, ws, pl, d_queries, nq, 2.0f, d_ids, d_dist, ws.n_fail + 3, s));
        return run_exact_queries(ix, ws, d_queries, 1, d_ids, d_dist, sm_count, s);
    }
    uint32_t* mask = reinterpret_cast<uint32_t*>(ws.cand);
    if (own_kth) {
        const size_t ksmem = (size_t)kKthQueries * ngroups * sizeof(float);
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_kth_smallest), ksmem));
        k_kth_smallest<<<(unsigned)((nq + kKthQueries - 1) / kKthQueries), kKthQueries * 32, ksmem, s>>>(ws.gmin, nq, pl.a.gmin_g, ngroups, nprobe, ws.seltop, nprobe,
                                                                                                                  mask, pl.a.mwords);
        count_launch();
        PSB_LAUNCH_CHECK();
    } else {
        PSB_TRY(launch_select_rows(ws.gmin, nq, ngroups, nprobe, ws.selids, ws.seltop, s));
        PSB_CUDA(cudaMemsetAsync(mask, 0, sizeof(uint32_t) * (size_t)nq * pl.a.mwords, s));
    }
    pl.a.mask = mask;
    PSB_TRY(run_tc<true>(pl, ws.ev[2], ws.ev[3], s));
    const size_t rsmem = (size_t)kCandCap * 8 + (size_t)(kRefineTile + 1) * refine_pitch(ix.dim) * sizeof(float);
    PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_coarse_refine), rsmem));
    k_coarse_refine<<<nq, kRefineThreads, rsmem, s>>>(d_queries, ix.centroids, ix.dim, ix.nlist, nprobe, pl.a.mask, pl.a.mwords, d_ids, d_dist,
                                                      ws.fail_list, ws.n_fail);
    count_launch();
    PSB_LAUNCH_CHECK();
    return run_exact_queries(ix, ws, d_queries, nprobe, d_ids, d_dist, sm_count, s);
}

// Nearest centroid of every row when a previous assignment is known (d_prev [nq], may alias d_ids): ONE GEMM pass.
psb_status launch_coarse_tc_assign(const CoarseTcIndex& ix, const CoarseTcWorkspace& ws, const float* d_rows, int nq, const int* d_prev,
                                   int* d_ids, float* d_dist, int sm_count, cudaStream_t s) {
    if (nq <= 0) return PSB_OK;
    if (!ws.queries_ready) PSB_TRY(launch_tc_prep_queries(ix, d_rows, nq, ws.qb, ws.qnorm, s));
    k_prev_bound<<<(unsigned)((nq + 31) / 32), 256, 0, s>>>(d_rows, nq, ix.dim, ix.centroids, ix.nlist, d_prev,
                                                                              static_cast<const float2*>(ws.qnorm), ws.seltop);
    count_launch();
    PSB_LAUNCH_CHECK();
    TcPlan pl;
    PSB_TRY(plan_tc(ix, ws, nq, 1, 32, sm_count, &pl));
    PSB_CUDA(cudaMemsetAsync(ws.n_fail, 0, 2 * sizeof(int), s));  // n_fail, cursor
    PSB_CUDA(cudaMemsetAsync(ws.n_fail2, 0, sizeof(int), s));
    PSB_TRY(nearest_by_lists(ix, ws, pl, d_rows, nq, 1.0f, d_ids, d_dist, nullptr, s));
    // Rows whose bound was too loose (their centroid has moved far away: the second iteration of a training, rows of clusters that
    // had drawn no initial centroid) are gathered and get the two passes of a row without a bound; how many they are is known on
    // the device only.  Searched one CTA per row, 13 % of 400,000 rows took 10 ms.
    const int cap = nq < coarse_tc_retry_rows() ? nq : coarse_tc_retry_rows();
    const int row16 = coarse_tc_padded_dim(ix.dim) / 8;
    k_gather_failed<<<sm_count * 4, 256, 0, s>>>(ws.fail_list, ws.n_fail, cap, static_cast<const uint4*>(ws.qb), static_cast<const float2*>(ws.qnorm),
                                                 row16, static_cast<uint4*>(ws.retry_qb), static_cast<float2*>(ws.retry_qnorm), ws.fail_list2, ws.n_fail2);
    count_launch();
    PSB_LAUNCH_CHECK();
    CoarseTcWorkspace w2 = ws;
    w2.qb = ws.retry_qb; w2.qnorm = ws.retry_qnorm;
    TcPlan p2;
    PSB_TRY(plan_tc(ix, w2, cap, 1, 32, sm_count, &p2));
    p2.a.nq_dev = ws.n_fail;
    PSB_TRY(run_tc<false>(p2, nullptr, nullptr, s));
    k_row_min<<<(unsigned)((cap + 31) / 32), 256, 0, s>>>(ws.gmin, cap, ws.n_fail, p2.a.gmin_g, p2.a.ngroups, ws.seltop);
    count_launch();
    PSB_LAUNCH_CHECK();
    p2.a.cand_cnt = ws.cand_cnt; p2.a.cand_list = ws.cand; p2.a.cand_cap = kAssignCap;
    PSB_CUDA(cudaMemsetAsync(ws.cand_cnt, 0, sizeof(int) * (size_t)cap, s));
    PSB_TRY(run_tc<true>(p2, nullptr, nullptr, s));
    PSB_TRY(run_refine1(ix, ws, d_rows, cap, ws.n_fail, ws.fail_list, d_ids, d_dist, ws.fail_list2, ws.n_fail2, nullptr, s));
    CoarseTcWorkspace w3 = ws;
    w3.fail_list = ws.fail_list2; w3.n_fail = ws.n_fail2; w3.fail_cursor = ws.n_fail + 1;
    return run_exact_queries(ix, w3, d_rows, 1, d_ids, d_dist, sm_count, s);
}

}  // namespace psb
