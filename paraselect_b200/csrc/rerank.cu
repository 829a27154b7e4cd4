// Exact rerank of the ADC candidates, id mapping and the multi-shard candidate merge.
//
// Rows in device memory, and the rows of a small batch, are scored where they lie.  The rows of a large batch in host memory cross
// PCIe once each, whatever the number of queries that ask for them (a third of the requests of a 10,000-query batch over 1M
// rows, two thirds and more on skewed lists, name a row another query has asked for):
//   k_mark_rows, k_count_rows, k_place_rows   every row the candidates name gets a slot of the staging buffer, in the order of the rows
//   k_gather_unique   copies the claimed rows - host memory mapped into the device address space, read over PCIe - to their
//                     slots; a warp keeps eight rows in flight.  Host threads fill a range of the slots instead or besides.
//   k_rerank_score*   eight lanes (half-warps, for rows that are not whole 16-byte units) score rows - from the slots or from where they lie - in the accumulation order of the CPU kernel
//                     the reference uses (four 16-lane FMA accumulators, pairwise combine, halving tree:
//                     src/cpu/distance/fp32_l2_avx512.h:16-53); rows not held here score +inf
//   k_topk_select     one CTA per query: the topk smallest (distance,row), duplicate rows once (reference semantics:
//                     src/search/ivf_common/ivf_host_rerank.cpp:152-177, src/search/ivf_common/ivf_exact_topk.h:12-22)
//   k_release_rows    the claims of a batch are taken back
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "select.cuh"

namespace psb {
namespace {

__device__ __forceinline__ int cand_count(const int* counts, int q, int candidate_count) {
    if (!counts) return candidate_count;
    const int c = counts[q];
    return c < 0 ? 0 : (c > candidate_count ? candidate_count : c);
}

// Global (index-wide, list-contiguous) row -> row of this session's exact store, or -1 when not held here.
__device__ __forceinline__ long long local_row(const RowMap& mp, long long r) {
    if (r < 0) return -1;
    if (!mp.global_begin) {
        const long long l = r - mp.base;
        return (l >= 0 && l < mp.count) ? l : -1;
    }
    int lo = 0, hi = mp.nlist;  // largest list with global_begin[list] <= r
    if (r < mp.global_begin[0]) return -1;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (mp.global_begin[mid] <= r) lo = mid; else hi = mid;
    }
    const long long l = mp.local_offsets[lo] + (r - mp.global_begin[lo]);
    return l < mp.local_offsets[lo + 1] ? l : -1;
}

// The claim of a part of a batch: k_mark_rows sets the bit of every row the part names and no earlier part has a slot for, k_count_rows counts the
// bits of each stretch of rows, k_place_rows gives the marked rows the next slots in the order of their numbers.  The order is what makes the fetch
// fast: rows read over PCIe at random places of a large array are bound by the translation of their addresses, in ascending order by the link.  A
// million rows of 384 bytes on 16 SMs: from an array of 0.8 GB 50.8 GB/s in random order, 50.9 sorted; of 4.6 GB 18.9 and 51.0; of 20 GB 12.9 and
// 51.0 (one large copy: 55.5).  The bits, count / 8 bytes of them (12.5 MB for 100M rows), are read by k_count_rows and by k_place_rows, which also
// clears as many of the claim before, for every part of a batch.
// Up to kSelfCountWords words each CTA counts the marks before its stretch itself, and k_count_rows is not launched (27,000 requests of 510,000
// rows: 10 us less per call).  The other CTAs read a CTA's words while it places them: the marks of the claim before are what it takes back.
constexpr int kPlaceThreads = 1024;                // words of 32 rows a CTA places: each warp 32 of them, one row per lane at a time
constexpr long long kSelfCountWords = 65536;
__global__ void __launch_bounds__(256) k_mark_rows(RowMap mp, const int* __restrict__ cand, int nq, int candidate_count, int candidate_stride,
                                                   const int* __restrict__ counts, const int* __restrict__ slot_of, unsigned* __restrict__ bits) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nq * candidate_count) return;
    const int q = (int)(i / candidate_count), c = (int)(i - (long long)q * candidate_count);
    if (c >= cand_count(counts, q, candidate_count)) return;
    const long long row = local_row(mp, cand[(size_t)q * candidate_stride + c]);
    if (row < 0 || slot_of[row] >= 0) return;
    const unsigned bit = 1u << (row & 31);
    if (!(*(volatile unsigned*)(bits + (row >> 5)) & bit)) atomicOr(bits + (row >> 5), bit);
}

__global__ void __launch_bounds__(kPlaceThreads) k_count_rows(const unsigned* __restrict__ bits, long long words, int* __restrict__ sums) {
    __shared__ int s_warp[32];
    const long long w = (long long)blockIdx.x * kPlaceThreads + threadIdx.x;
    int n = w < words ? __popc(bits[w]) : 0;
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x < 32) {
        n = __reduce_add_sync(0xffffffffu, s_warp[threadIdx.x]);
        if (threadIdx.x == 0) sums[blockIdx.x] = n;
    }
}

// *begin: the first slot of the part.  The last CTA notes the end, and with it the number of slots so far.  sums null: not counted.
__global__ void __launch_bounds__(kPlaceThreads) k_place_rows(const unsigned* __restrict__ bits, unsigned* __restrict__ old_bits, long long words,
                                                              const int* __restrict__ sums,
                                                              const int* __restrict__ begin, int* __restrict__ end, int* __restrict__ n_unique,
                                                              int* __restrict__ slot_of, int* __restrict__ unique) {
    __shared__ int s_warp[33], s_before[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * kPlaceThreads + threadIdx.x;
    const unsigned word = w < words ? bits[w] : 0u;
    int before = 0;   // marked rows of the stretches before this one
    if (sums) {
        for (int b = threadIdx.x; b < (int)blockIdx.x; b += kPlaceThreads) before += sums[b];
    } else {
#pragma unroll 8
        for (int b = 0; b < (int)blockIdx.x; ++b) before += __popc(bits[b * kPlaceThreads + threadIdx.x]);
    }
    if (w < words) old_bits[w] = 0u;
    before = __reduce_add_sync(0xffffffffu, before);
    const int mine = __popc(word), all = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) { s_before[warp] = before; s_warp[warp] = all; }
    __syncthreads();
    if (warp == 0) {
        const int v = s_warp[lane];
        int in = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int up = __shfl_up_sync(0xffffffffu, in, o); if (lane >= o) in += up; }
        const int base = *begin + __reduce_add_sync(0xffffffffu, s_before[lane]);
        s_warp[lane] = base + in - v;
        if (lane == 31) {
            s_warp[32] = base + in;
            if (blockIdx.x == gridDim.x - 1) { *end = base + in; *n_unique = base + in; }
        }
    }
    __syncthreads();
    int slot = s_warp[warp];   // of the warp's next word
    unsigned live = __ballot_sync(0xffffffffu, word != 0u);
    const int row0 = (int)((w - lane) * 32);
    while (live) {
        const int l = __ffs((int)live) - 1;
        live &= live - 1;
        const unsigned x = __shfl_sync(0xffffffffu, word, l);
        if ((x >> lane) & 1u) {
            const int at = slot + __popc(x & ((1u << lane) - 1u)), row = row0 + l * 32 + lane;
            unique[at] = row;
            slot_of[row] = at;
        }
        slot += __popc(x);
    }
}

// A copy to the host behind the last kernel took 3 us of copy engine and 8 of waiting for it.
__global__ void k_call_tail(const unsigned long long* __restrict__ words, const int* __restrict__ coarse, CallTail* tail) {
    behind();
    mark_start(&tail->end);
    if (threadIdx.x < 16) tail->c[threadIdx.x] = words[threadIdx.x];
    if (coarse && threadIdx.x < 8) tail->tc[threadIdx.x] = coarse[threadIdx.x];
}

// *fetched grows by the number of rows.
__global__ void k_release_rows(const int* __restrict__ unique, const int* __restrict__ n_unique, int* __restrict__ slot_of, unsigned long long* __restrict__ fetched) {
    const int n = *n_unique;
    if ((blockIdx.x | threadIdx.x) == 0) *fetched += (unsigned long long)n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) slot_of[unique[i]] = -1;
}

// Copies the rows of slots [*begin, *end), from the end of the host threads' share (host_pct) on, into the staging buffer; a warp takes eight slots
// at a time, all eight rows' loads issued before the first store.
__device__ __forceinline__ void gather_unique_body(const unsigned char* __restrict__ src, int row_bytes, const int* __restrict__ unique,
                                                   const int* __restrict__ begin, const int* __restrict__ end, int host_pct,
                                                   unsigned char* __restrict__ stage) {
    constexpr int U = 8;
    const int lane = threadIdx.x & 31;
    const int warp0 = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5), nwarps = (int)(((long long)gridDim.x * blockDim.x) >> 5);
    const int e = *end, b = host_share_end(*begin, e, host_pct);
    const uintptr_t both = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(stage);
    const bool vec16 = (row_bytes % 16) == 0 && (both % 16) == 0, vec4 = (row_bytes % 4) == 0 && (both % 4) == 0;
    for (int s0 = b + warp0 * U; s0 < e; s0 += nwarps * U) {
        const int mine = lane < U && s0 + lane < e ? unique[s0 + lane] : -1;
        if (vec16) {
            for (int j0 = 0; j0 < row_bytes / 16; j0 += 32) {
                const int j = j0 + lane;
                uint4 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int r = __shfl_sync(0xffffffffu, mine, u);
                    if (r >= 0 && j < row_bytes / 16) v[u] = reinterpret_cast<const uint4*>(src + (size_t)r * row_bytes)[j];
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (__shfl_sync(0xffffffffu, mine, u) >= 0 && j < row_bytes / 16) reinterpret_cast<uint4*>(stage + (size_t)(s0 + u) * row_bytes)[j] = v[u];
            }
        } else if (vec4) {
            for (int j0 = 0; j0 < row_bytes / 4; j0 += 32) {
                const int j = j0 + lane;
                uint32_t v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int r = __shfl_sync(0xffffffffu, mine, u);
                    if (r >= 0 && j < row_bytes / 4) v[u] = reinterpret_cast<const uint32_t*>(src + (size_t)r * row_bytes)[j];
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (__shfl_sync(0xffffffffu, mine, u) >= 0 && j < row_bytes / 4) reinterpret_cast<uint32_t*>(stage + (size_t)(s0 + u) * row_bytes)[j] = v[u];
            }
        } else {
            for (int u = 0; u < U; ++u) {
                const int r = __shfl_sync(0xffffffffu, mine, u);
                if (r < 0) continue;
                for (int j = lane; j < row_bytes; j += 32) stage[(size_t)(s0 + u) * row_bytes + j] = src[(size_t)r * row_bytes + j];
            }
        }
    }
}

__global__ void __launch_bounds__(256) k_gather_unique(const unsigned char* __restrict__ src, int row_bytes, const int* __restrict__ unique,
                                                       const int* __restrict__ begin, const int* __restrict__ end, int host_pct,
                                                       unsigned char* __restrict__ stage) {
    gather_unique_body(src, row_bytes, unique, begin, end, host_pct, stage);
}
// The same gather built to sit BESIDE a scan kernel that owns nearly a whole SM (one 576-thread CTA with ~55K registers and
// ~200 KB of shared memory): 128-thread CTAs capped at 40 registers and no shared memory, two of which fit into what the
// scan leaves of every SM.
__global__ void __launch_bounds__(256, 6) k_gather_unique_beside(const unsigned char* __restrict__ src, int row_bytes, const int* __restrict__ unique,
                                                                 const int* __restrict__ begin, const int* __restrict__ end, int host_pct,
                                                                 unsigned char* __restrict__ stage) {
    gather_unique_body(src, row_bytes, unique, begin, end, host_pct, stage);
}
// The same gather on SMs of its own: CTAs of 1,024 threads that also claim (without using it) nearly all the shared memory of
// an SM, so that no kernel with a shared-memory footprint - the scan, the cutoff sampling, the selections - shares an SM with
// them.  Reads of host memory stay in flight for microseconds; next to another kernel's warps they held up that kernel's own
// memory traffic (its stages ran at half speed), on separate SMs they do not.
__global__ void __launch_bounds__(1024, 1) k_gather_unique_owned(const unsigned char* __restrict__ src, int row_bytes, const int* __restrict__ unique,
                                                                 const int* __restrict__ begin, const int* __restrict__ end, int host_pct,
                                                                 unsigned char* __restrict__ stage) {
    gather_unique_body(src, row_bytes, unique, begin, end, host_pct, stage);
}

// fp32 squared L2 by a half-warp (16 lanes), bit-identical to the AVX-512 kernel's order.
// All 16 lanes of the half-warp must call it together; hmask names exactly those lanes.
__device__ __forceinline__ float l2_halfwarp(const float* __restrict__ q, const float* __restrict__ v, int dim, int j,
                                             unsigned hmask) {
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
    int i = 0;
    for (; i + 64 <= dim; i += 64) {
        float d = __fsub_rn(q[i + j], v[i + j]); a0 = __fmaf_rn(d, d, a0);
        d = __fsub_rn(q[i + 16 + j], v[i + 16 + j]); a1 = __fmaf_rn(d, d, a1);
        d = __fsub_rn(q[i + 32 + j], v[i + 32 + j]); a2 = __fmaf_rn(d, d, a2);
        d = __fsub_rn(q[i + 48 + j], v[i + 48 + j]); a3 = __fmaf_rn(d, d, a3);
    }
    for (; i + 16 <= dim; i += 16) {
        const float d = __fsub_rn(q[i + j], v[i + j]); a0 = __fmaf_rn(d, d, a0);
    }
    float s = __fadd_rn(__fadd_rn(a0, a1), __fadd_rn(a2, a3));
    s = __fadd_rn(s, __shfl_xor_sync(hmask, s, 8));
    s = __fadd_rn(s, __shfl_xor_sync(hmask, s, 4));
    s = __fadd_rn(s, __shfl_xor_sync(hmask, s, 2));
    s = __fadd_rn(s, __shfl_xor_sync(hmask, s, 1));
    for (; i < dim; ++i) { const float d = __fsub_rn(q[i], v[i]); s = __fmaf_rn(d, d, s); }
    return s;
}

__device__ __forceinline__ float l2_u8_halfwarp(const unsigned char* __restrict__ q, const unsigned char* __restrict__ v,
                                                int dim, int j, unsigned hmask) {
    int s = 0;
    if (((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(v) | (uintptr_t)dim) & 3) == 0) {   // whole numbers: any order
        unsigned acc = 0;
        for (int i = j; i < dim / 4; i += 16) {
            const unsigned d = __vabsdiffu4(reinterpret_cast<const unsigned*>(q)[i], reinterpret_cast<const unsigned*>(v)[i]);
            acc = __dp4a(d, d, acc);
        }
        s = (int)acc;
    } else {
        for (int i = j; i < dim; i += 16) { const int d = (int)q[i] - (int)v[i]; s += d * d; }
    }
    s += __shfl_xor_sync(hmask, s, 8);
    s += __shfl_xor_sync(hmask, s, 4);
    s += __shfl_xor_sync(hmask, s, 2);
    s += __shfl_xor_sync(hmask, s, 1);
    return (float)s;
}

constexpr int kScoreThreads = 256;
constexpr int kScoreRows = 4;                                       // rows a warp has in flight
constexpr int kScoreBlock = kScoreThreads / 32 * kScoreRows;        // candidates per CTA
__host__ __device__ __forceinline__ int score_pitch(int row_bytes) { return (row_bytes + 15) / 16 * 16 + 16; }
// grid (nq, candidate_count / kScoreBlock): dist[q][i] = exact distance of candidate i, +inf when the row is invalid, beyond the
// query's count, or not held by this session.  slot_of null: the rows lie at src by their number (device memory, or host memory
// mapped here); else at src by their slot.  Rows are fetched whole, 16 bytes per lane, into shared memory (through = 0: too long
// for it, read in place).
__global__ void __launch_bounds__(kScoreThreads)
k_rerank_score(const unsigned char* __restrict__ src, const int* __restrict__ slot_of, RowMap mp, int dim, int elem_bytes, int through,
               const unsigned char* __restrict__ queries, const int* __restrict__ cand, int candidate_count,
               int candidate_stride, const int* __restrict__ counts, float* __restrict__ out_dist, unsigned long long* mark) {
    behind();
    mark_start(mark);
    extern __shared__ __align__(16) unsigned char s_score[];
    const int q = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row_bytes = dim * elem_bytes, pitch = score_pitch(row_bytes);
    unsigned char* s_q = s_score;
    unsigned char* s_row = s_score + pitch + (size_t)warp * kScoreRows * pitch;
    if ((row_bytes & 3) == 0)
        for (int i = threadIdx.x; i < row_bytes / 4; i += kScoreThreads) reinterpret_cast<uint32_t*>(s_q)[i] = reinterpret_cast<const uint32_t*>(queries + (size_t)q * row_bytes)[i];
    else
        for (int i = threadIdx.x; i < row_bytes; i += kScoreThreads) s_q[i] = queries[(size_t)q * row_bytes + i];
    const int n = cand_count(counts, q, candidate_count);
    const int i0 = blockIdx.y * kScoreBlock + warp * kScoreRows;
    int at = -1;
    if (lane < kScoreRows && i0 + lane < n) {
        const long long row = local_row(mp, cand[(size_t)q * candidate_stride + i0 + lane]);
        if (row >= 0) at = slot_of ? slot_of[row] : (int)row;
    }
    if (through) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(src) | (uintptr_t)row_bytes;
        const int unit = (a & 15) == 0 ? 16 : ((a & 3) == 0 ? 4 : 1);
        const int units = row_bytes / unit;
        for (int j0 = 0; j0 < units; j0 += 32) {
            const int j = j0 + lane;
            uint4 v[kScoreRows];
#pragma unroll
            for (int u = 0; u < kScoreRows; ++u) {
                const int r = __shfl_sync(0xffffffffu, at, u);
                if (r < 0 || j >= units) continue;
                const unsigned char* p = src + (size_t)r * row_bytes + (size_t)j * unit;
                if (unit == 16) v[u] = __ldg(reinterpret_cast<const uint4*>(p));
                else if (unit == 4) v[u].x = __ldg(reinterpret_cast<const uint32_t*>(p));
                else v[u].x = __ldg(p);
            }
#pragma unroll
            for (int u = 0; u < kScoreRows; ++u) {
                if (__shfl_sync(0xffffffffu, at, u) < 0 || j >= units) continue;
                unsigned char* d = s_row + u * pitch + j * unit;
                if (unit == 16) *reinterpret_cast<uint4*>(d) = v[u];
                else if (unit == 4) *reinterpret_cast<uint32_t*>(d) = v[u].x;
                else *d = (unsigned char)v[u].x;
            }
        }
    }
    __syncthreads();
    const int half = lane >> 4, j = lane & 15;
    const unsigned hmask = 0xffffu << (lane & 16);
#pragma unroll
    for (int u0 = 0; u0 < kScoreRows; u0 += 2) {
        const int u = u0 + half;
        const int r = __shfl_sync(0xffffffffu, at, u);
        float d = __int_as_float(0x7f800000);
        if (r >= 0) {
            const unsigned char* v = through ? s_row + u * pitch : src + (size_t)r * row_bytes;
            d = elem_bytes == 4 ? l2_halfwarp(reinterpret_cast<const float*>(s_q), reinterpret_cast<const float*>(v), dim, j, hmask)
                                : l2_u8_halfwarp(s_q, v, dim, j, hmask);
        }
        if (j == 0 && i0 + u < candidate_count) out_dist[(size_t)q * candidate_count + i0 + u] = d;
    }
}

// The same scores for rows of whole 16-byte units.  Eight lanes a row: lane l stands for lanes 4 (l % 4) .. + 3 of the CPU kernel's 16 and
// for its accumulators l / 4 and l / 4 + 2, so the row comes in as 128-byte lines straight into registers, the additions are
// the CPU kernel's own, and a row takes 73 warp instructions where a half-warp and a trip through shared memory took 160, which is
// what bound it: 2,000 queries x 500 rows of 384 bytes 165 -> 122 us.
// Two rows per lane group at a time cost the occupancy more than they brought (72 registers: 136 us).
template <bool U8>
__global__ void __launch_bounds__(kScoreThreads, 6)
k_rerank_score_wide(const unsigned char* __restrict__ src, const int* __restrict__ slot_of, RowMap mp, int dim,
                    const unsigned char* __restrict__ queries, const int* __restrict__ cand, int candidate_count,
                    int candidate_stride, const int* __restrict__ counts, float* __restrict__ out_dist, unsigned long long* mark) {
    behind();
    mark_start(mark);
    extern __shared__ __align__(16) unsigned char s_score[];
    const int q = blockIdx.x, lane = threadIdx.x & 31, l = lane & 7;
    const int units = (U8 ? dim : dim * 4) >> 4;
    const int i = (blockIdx.y * (kScoreThreads / 32) + (threadIdx.x >> 5)) * 4 + (lane >> 3);
    long long at = i < cand_count(counts, q, candidate_count) ? local_row(mp, cand[(size_t)q * candidate_stride + i]) : -1;
    if (at >= 0 && slot_of) at = slot_of[at];
    const uint4* own = reinterpret_cast<const uint4*>(queries) + (size_t)q * units;
    const uint4* row = at >= 0 ? reinterpret_cast<const uint4*>(src) + (size_t)at * units : own;   // no row: any will do
    uint4* query = reinterpret_cast<uint4*>(s_score);
    for (int u = threadIdx.x; u < units; u += kScoreThreads) query[u] = own[u];
    __syncthreads();
    float result;
    if constexpr (U8) {
        unsigned acc = 0;
#pragma unroll 4
        for (int u = l; u < units; u += 8) {
            const uint4 v = __ldg(row + u), y = query[u];
            unsigned d = __vabsdiffu4(v.x, y.x); acc = __dp4a(d, d, acc);
            d = __vabsdiffu4(v.y, y.y); acc = __dp4a(d, d, acc);
            d = __vabsdiffu4(v.z, y.z); acc = __dp4a(d, d, acc);
            d = __vabsdiffu4(v.w, y.w); acc = __dp4a(d, d, acc);
        }
        acc += __shfl_xor_sync(0xffffffffu, acc, 4);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        result = (float)(int)acc;
    } else {
        float a0[4] = {0.f, 0.f, 0.f, 0.f}, a1[4] = {0.f, 0.f, 0.f, 0.f};   // accumulators l / 4 and l / 4 + 2
        auto fold = [](float (&acc)[4], const uint4& x, const uint4& y) {   // y: the query
            float d = __fsub_rn(__uint_as_float(y.x), __uint_as_float(x.x)); acc[0] = __fmaf_rn(d, d, acc[0]);
            d = __fsub_rn(__uint_as_float(y.y), __uint_as_float(x.y)); acc[1] = __fmaf_rn(d, d, acc[1]);
            d = __fsub_rn(__uint_as_float(y.z), __uint_as_float(x.z)); acc[2] = __fmaf_rn(d, d, acc[2]);
            d = __fsub_rn(__uint_as_float(y.w), __uint_as_float(x.w)); acc[3] = __fmaf_rn(d, d, acc[3]);
        };
        const int full = units & ~15;   // 16-byte units in whole blocks of 64 elements
#pragma unroll 2
        for (int u = l; u < full; u += 16) {
            const uint4 v0 = __ldg(row + u), v1 = __ldg(row + u + 8);
            fold(a0, v0, query[u]);
            fold(a1, v1, query[u + 8]);
        }
        if (l < 4) {   // what is left goes to accumulator 0, 16 elements at a time
#pragma unroll
            for (int c = 0; c < 3; ++c)
                if (full + 4 * c + 4 <= units) fold(a0, __ldg(row + full + 4 * c + l), query[full + 4 * c + l]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)   // (a0 + a1) + (a2 + a3)
            a0[e] = __fadd_rn(__fadd_rn(a0[e], __shfl_xor_sync(0xffffffffu, a0[e], 4)), __fadd_rn(a1[e], __shfl_xor_sync(0xffffffffu, a1[e], 4)));
#pragma unroll
        for (int e = 0; e < 4; ++e) a0[e] = __fadd_rn(a0[e], __shfl_xor_sync(0xffffffffu, a0[e], 2));   // halving tree: 8 apart,
#pragma unroll
        for (int e = 0; e < 4; ++e) a0[e] = __fadd_rn(a0[e], __shfl_xor_sync(0xffffffffu, a0[e], 1));   // 4,
        result = __fadd_rn(__fadd_rn(a0[0], a0[2]), __fadd_rn(a0[1], a0[3]));                           // 2 and 1
        if (l == 0) {
#pragma unroll 1
            for (int d = dim & ~15; d < dim; ++d) {
                const float diff = __fsub_rn(reinterpret_cast<const float*>(s_score)[d], __ldg(reinterpret_cast<const float*>(row) + d));
                result = __fmaf_rn(diff, diff, result);
            }
        }
    }
    if (l == 0 && i < candidate_count) out_dist[(size_t)q * candidate_count + i] = at >= 0 ? result : __int_as_float(0x7f800000);
}

constexpr int kSelectThreads = 256;
// dist [nq][candidate_count] (dense), cand [nq][candidate_stride] global rows.  ids: original ids by row (out_ids is written
// instead of out_rows).  The smallest come from select.cuh; when a row turns up twice among them - the ADC stage names a row once, a
// caller's own candidates need not - everything is sorted and duplicates, equal keys next to each other, are dropped.
__global__ void __launch_bounds__(kSelectThreads)
k_topk_select(const float* __restrict__ dist, const int* __restrict__ cand, int candidate_count, int candidate_stride,
              const int* __restrict__ counts, int topk, int np, int buffer, int* __restrict__ out_rows, float* __restrict__ out_dist,
              const long long* __restrict__ ids, long long* __restrict__ out_ids) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    uint64_t* s_keys = reinterpret_cast<uint64_t*>(s_raw);            // [max(np, buffer)]
    int* s_rank = reinterpret_cast<int*>(s_raw + (size_t)max(np, buffer) * 8);  // [max(np, kMaxGroups)]: ranks, or the selection's runs
    __shared__ sel::Words w;
    __shared__ int s_warp[32];
    __shared__ int s_total, s_twice;
    behind();
    const int q = blockIdx.x;
    const int n = cand_count(counts, q, candidate_count);
    const int* rows = cand + (size_t)q * candidate_stride;
    const float inf = __int_as_float(0x7f800000);
    auto put = [&](int r, uint64_t key) {
        if (out_ids) out_ids[(size_t)q * topk + r] = key == KEY_MAX ? -1 : ids[key_idx(key)];
        else out_rows[(size_t)q * topk + r] = key == KEY_MAX ? -1 : (int)key_idx(key);
        out_dist[(size_t)q * topk + r] = key == KEY_MAX ? FLT_MAX : key_dist(key);
    };
    const int keep = sel::smallest<kSelectThreads>(dist + (size_t)q * candidate_count, n, topk, [&](int i) { return (uint32_t)rows[i]; }, s_keys, buffer,
                                                   s_rank, &w);
    if (threadIdx.x == 0) s_twice = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < keep; i += kSelectThreads)   // a row twice, or a distance without a row
        if (key_dist(s_keys[i]) != inf && ((i && s_keys[i] == s_keys[i - 1]) || (int)key_idx(s_keys[i]) < 0)) s_twice = 1;
    __syncthreads();
    if (!s_twice) {
        for (int r = threadIdx.x; r < topk; r += kSelectThreads) put(r, r < keep && key_dist(s_keys[r]) != inf ? s_keys[r] : KEY_MAX);
        return;
    }
    for (int i = threadIdx.x; i < np; i += kSelectThreads) {
        uint64_t key = KEY_MAX;
        if (i < n) {
            const float d = dist[(size_t)q * candidate_count + i];
            if (rows[i] >= 0 && d != inf) key = make_key(d, (uint32_t)rows[i]);
        }
        s_keys[i] = key;
    }
    __syncthreads();
    block_bitonic_sort(s_keys, np);
    int base = 0;
    for (int c0 = 0; c0 < np; c0 += kSelectThreads) {
        const int i = c0 + threadIdx.x;
        int fresh = 0;
        if (i < np) {
            const uint64_t key = s_keys[i];
            fresh = key != KEY_MAX && (i == 0 || s_keys[i - 1] != key);
        }
        const int ex = block_exclusive_scan(fresh, s_warp, &s_total);
        if (i < np) s_rank[i] = fresh ? base + ex : -1;
        base += s_total;
        __syncthreads();
    }
    for (int i = threadIdx.x; i < np; i += kSelectThreads) {
        const int r = s_rank[i];
        if (r >= 0 && r < topk) put(r, s_keys[i]);
    }
    for (int r = base + threadIdx.x; r < topk; r += kSelectThreads) put(r, KEY_MAX);
}

// out[i] = original id of global row rows[i] when this session holds the row, else -1.
__global__ void k_map_ids(const int* __restrict__ rows, long long n, const long long* __restrict__ reordered, RowMap mp,
                          long long* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long l = local_row(mp, rows[i]);
    out[i] = l >= 0 ? reordered[l] : -1ll;
}

__global__ void k_widen_ids(const int* __restrict__ in, long long n, long long* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[i];
}

__global__ void k_offset_rows(int* __restrict__ rows, long long n, int delta) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && rows[i] >= 0) rows[i] += delta;
}

// Per query: the k smallest (distance,row) of parts*k shard candidates.
__global__ void __launch_bounds__(1024)
k_merge(const int* __restrict__ rows, const float* __restrict__ dist, int parts, int nq, int k, int np,
        int* __restrict__ out_rows, float* __restrict__ out_dist) {
    extern __shared__ __align__(16) uint64_t s_mkeys[];
    const int q = blockIdx.x;
    const int total = parts * k;
    for (int i = threadIdx.x; i < np; i += blockDim.x) {
        uint64_t key = KEY_MAX;
        if (i < total) {
            const int p = i / k, e = i % k;
            const size_t at = ((size_t)p * nq + q) * k + e;
            const int r = rows[at];
            if (r >= 0) key = make_key(dist[at], (uint32_t)r);
        }
        s_mkeys[i] = key;
    }
    __syncthreads();
    block_bitonic_sort(s_mkeys, np);
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        const uint64_t key = s_mkeys[i];
        const bool ok = key != KEY_MAX;
        out_rows[(size_t)q * k + i] = ok ? (int)key_idx(key) : -1;
        out_dist[(size_t)q * k + i] = ok ? key_dist(key) : FLT_MAX;
    }
}

}  // namespace

size_t claim_words(long long count) { return (size_t)((std::max<long long>(1, count) + 31) / 32); }
size_t claim_sums(long long count) { return (claim_words(count) + kPlaceThreads - 1) / kPlaceThreads; }

psb_status launch_claim_rows(const RowMap& mp, const int* d_candidates, int nq, int candidate_count, int candidate_stride, const int* d_counts,
                             const ClaimBuffers& b, const int* d_begin, int* d_end, int* d_n_unique, cudaStream_t s) {
    if (nq <= 0) return PSB_OK;
    const long long total = (long long)nq * candidate_count, words = (long long)claim_words(b.count);
    const unsigned ctas = (unsigned)claim_sums(b.count);
    PSB_TRY(prefer_max_shared(k_mark_rows));
    k_mark_rows<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(mp, d_candidates, nq, candidate_count, candidate_stride, d_counts, b.slot_of, b.bits);
    const bool counted = words > kSelfCountWords;
    if (counted) {
        PSB_TRY(prefer_max_shared(k_count_rows));
        k_count_rows<<<ctas, kPlaceThreads, 0, s>>>(b.bits, words, b.sums);
    }
    PSB_TRY(prefer_max_shared(k_place_rows));
    k_place_rows<<<ctas, kPlaceThreads, 0, s>>>(b.bits, b.old_bits, words, counted ? b.sums : nullptr, d_begin, d_end, d_n_unique, b.slot_of, b.unique);
    count_launch(counted ? 3 : 2);
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_release_rows(const int* d_unique, const int* d_n_unique, int* d_slot_of, unsigned long long* d_fetched, int sm_count, cudaStream_t s) {
    PSB_TRY(prefer_max_shared(k_release_rows));
    k_release_rows<<<sm_count * 2, 256, 0, s>>>(d_unique, d_n_unique, d_slot_of, d_fetched);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_gather_unique(const void* src, int row_bytes, const int* d_unique, const int* d_begin, const int* d_end, int host_pct,
                                void* d_stage, cudaStream_t s, int sm_count, int compact_ctas, int owned_sms) {
    const unsigned char* from = static_cast<const unsigned char*>(src);
    unsigned char* to = static_cast<unsigned char*>(d_stage);
    if (owned_sms > 0) {
        constexpr int kOwnedSmem = 200 * 1024;   // claimed, not used: keeps every kernel that needs shared memory off the SM
        PSB_TRY(prefer_max_shared(k_gather_unique_owned));
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_gather_unique_owned), kOwnedSmem));
        k_gather_unique_owned<<<owned_sms, 1024, kOwnedSmem, s>>>(from, row_bytes, d_unique, d_begin, d_end, host_pct, to);
    } else if (compact_ctas > 0) {
        PSB_TRY(prefer_max_shared(k_gather_unique_beside));
        k_gather_unique_beside<<<compact_ctas, 128, 0, s>>>(from, row_bytes, d_unique, d_begin, d_end, host_pct, to);
    } else {
        PSB_TRY(prefer_max_shared(k_gather_unique));
        k_gather_unique<<<sm_count * 2, 256, 0, s>>>(from, row_bytes, d_unique, d_begin, d_end, host_pct, to);
    }
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_rerank_score(const void* d_src, const int* d_slot_of, const RowMap& mp, int dim, int elem_bytes, const void* d_queries,
                               const int* d_candidates, int nq, int candidate_count, int candidate_stride,
                               const int* d_counts, float* d_out_dist, cudaStream_t s, unsigned long long* mark, bool chained) {
    if (nq <= 0) return PSB_OK;
    const int row_bytes = dim * elem_bytes;
    const dim3 grid(nq, (candidate_count + kScoreBlock - 1) / kScoreBlock);
    if (((reinterpret_cast<uintptr_t>(d_src) | reinterpret_cast<uintptr_t>(d_queries) | row_bytes) & 15) == 0 && row_bytes <= 48 * 1024) {
        auto kernel = elem_bytes == 4 ? k_rerank_score_wide<false> : k_rerank_score_wide<true>;
        PSB_TRY(prefer_max_shared(kernel));
        PSB_TRY(launch_behind(chained, kernel, grid, kScoreThreads, row_bytes, s, static_cast<const unsigned char*>(d_src), d_slot_of, mp, dim, static_cast<const unsigned char*>(d_queries), d_candidates, candidate_count, candidate_stride, d_counts, d_out_dist, mark));
        count_launch();
        PSB_LAUNCH_CHECK();
        return PSB_OK;
    }
    const size_t pitch = (size_t)score_pitch(dim * elem_bytes);
    size_t smem = pitch * (1 + kScoreBlock);
    const int through = smem <= (size_t)200 * 1024 ? 1 : 0;
    if (!through) smem = pitch;
    if (smem > (size_t)220 * 1024) return fail(PSB_UNSUPPORTED_SHAPE, "rows too long for the exact rerank");
    if (smem > 48 * 1024) PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_rerank_score), smem));
    PSB_TRY(prefer_max_shared(k_rerank_score));
    PSB_TRY(launch_behind(chained, k_rerank_score, grid, kScoreThreads, smem, s, static_cast<const unsigned char*>(d_src), d_slot_of, mp, dim, elem_bytes, through, static_cast<const unsigned char*>(d_queries), d_candidates, candidate_count, candidate_stride, d_counts, d_out_dist, mark));
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_call_tail(const unsigned long long* d_words, const int* d_coarse, CallTail* h_tail, cudaStream_t s, bool chained) {
    PSB_TRY(prefer_max_shared(k_call_tail));
    PSB_TRY(launch_behind(chained, k_call_tail, dim3(1), 32, 0, s, d_words, d_coarse, h_tail));
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_topk_select(const float* d_dist, const int* d_candidates, int nq, int candidate_count,
                              int candidate_stride, const int* d_counts, int topk, int* d_out_rows,
                              float* d_out_dist, cudaStream_t s, const long long* d_ids, long long* d_out_ids, bool chained) {
    if (nq <= 0) return PSB_OK;
    if (candidate_count > kMaxRerankWidth) return fail(PSB_UNSUPPORTED_SHAPE, "rerank accepts at most 4096 candidates per query");
    int np = 32;
    while (np < candidate_count) np <<= 1;
    const int buffer = sel::buffer_entries(topk);
    const size_t smem = (size_t)std::max(np, buffer) * 8 + (size_t)std::max(np, sel::kMaxGroups) * 4;
    if (smem > 32 * 1024)
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_topk_select), smem));
    PSB_TRY(prefer_max_shared(k_topk_select));
    PSB_TRY(launch_behind(chained, k_topk_select, dim3((unsigned)nq), kSelectThreads, smem, s, d_dist, d_candidates, candidate_count, candidate_stride, d_counts, topk, np, buffer, d_out_rows, d_out_dist, d_ids, d_out_ids));
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_map_ids(const int* d_rows, long long n, const long long* d_reordered, const RowMap& mp,
                          long long* d_out, cudaStream_t s) {
    if (n <= 0) return PSB_OK;
    PSB_TRY(prefer_max_shared(k_map_ids));
    k_map_ids<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_rows, n, d_reordered, mp, d_out);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_widen_ids(const int* d_in, long long n, long long* d_out, cudaStream_t s) {
    if (n <= 0) return PSB_OK;
    k_widen_ids<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_in, n, d_out);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_offset_rows(int* d_rows, long long n, int delta, cudaStream_t s) {
    if (n <= 0 || delta == 0) return PSB_OK;
    k_offset_rows<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_rows, n, delta);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_merge(const int* d_rows, const float* d_dist, int parts, int nq, int k, int* d_out_rows,
                        float* d_out_dist, cudaStream_t s) {
    if (nq <= 0) return PSB_OK;
    const long long total = (long long)parts * k;
    if (total > 16384) return fail(PSB_UNSUPPORTED_SHAPE, "merge accepts at most 16384 candidates per query");
    int np = 2;
    while (np < total) np <<= 1;
    const size_t smem = (size_t)np * 8;
    if (smem > 32 * 1024) PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_merge), smem));
    k_merge<<<nq, 1024, smem, s>>>(d_rows, d_dist, parts, nq, k, np, d_out_rows, d_out_dist);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

}  // namespace psb
