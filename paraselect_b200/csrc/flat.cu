// IVF-Flat fine scan over device-resident rows: for every query the exact fp32 squared L2 distance to every row of its
// probed lists, and the topk nearest by (distance, row), as original ids.
//
// Two halves with a distance row per query between them.  The distances: every (query, probe) pair owns a stretch of the query's
// row; when lists have enough visitors they are computed list by list in tiles of 32 visiting queries x 64 rows (dist_tile.cuh), so
// that a list's rows are read once per 32 visitors and the arithmetic - sequential, sub / mul / add without FMA, the reference's
// l2_distance_squared (src/cpu/utils/cpu_distance.h:74-81) - runs at its issue limit; with few visitors a thread takes one row of
// one query and the rows of a query are spread over the whole chip.  The selection reads each query's distances twice (select.cuh).
// One CTA per query that did both took 872 us for 1,000 queries x 16 lists of 390 rows x 128 (L2 traffic of every visit) and
// 573 us for 4 queries (four CTAs).  Results equal the reference's cpu_ivf_search (src/cpu/search/cpu_search.h:226-332) with ties
// by row.
//
// Reference counterpart: the GPU-resident fine kernels of src/search/kernels/fine/gpu_fine/resident/resident_full_l2_topk.cu:19-178
// behind ivfflat_search (src/search/ivfflat/ivfflat_search.cuh:41-51).
#include <cuda_bf16.h>
#include <algorithm>

#include "common.cuh"
#include "dist_tile.cuh"
#include "kernels.h"
#include "scan_common.cuh"
#include "select.cuh"

namespace psb {

using namespace tile;

namespace {

// One warp per query: where each probe's distances start in the query's row, the rows it scans, and (list form) the pair's place
// among its list's visitors.
__global__ void __launch_bounds__(128) k_row_segments(const int* __restrict__ probes, int nq, int nprobe, const long long* __restrict__ offsets, int lb, int le,
                                                    int* __restrict__ seg, int* __restrict__ vis_count, int* __restrict__ slot,
                                                    unsigned long long* __restrict__ counters, unsigned long long* mark) {
    behind();
    mark_start(mark);
    const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (q >= nq) return;
    int* s = seg + (size_t)q * (nprobe + 1);
    int carry = 0;
    for (int p0 = 0; p0 < nprobe; p0 += 32) {
        const int p = p0 + lane;
        int len = 0, l = -1;
        if (p < nprobe) {
            l = probes[(size_t)q * nprobe + p];
            if (l >= lb && l < le) len = (int)(offsets[l + 1] - offsets[l]); else l = -1;
        }
        int in = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int up = __shfl_up_sync(0xffffffffu, in, o); if (lane >= o) in += up; }
        if (p < nprobe) {
            s[p] = carry + in - len;
            if (slot) slot[(size_t)q * nprobe + p] = l >= 0 ? atomicAdd(&vis_count[l], 1) : -1;
        }
        carry += __shfl_sync(0xffffffffu, in, 31);
    }
    if (lane == 0) {
        s[nprobe] = carry;
        if (counters) atomicAdd(&counters[0], (unsigned long long)carry);
    }
}

// Single CTA: exclusive scans over the lists (visitor offsets, tiles).
__global__ void __launch_bounds__(1024) k_flat_lists(const int* __restrict__ vis_count, const long long* __restrict__ offsets, int nlist,
                                                     int* __restrict__ vis_off, long long* __restrict__ item_off) {
    __shared__ int s_warp[32];
    __shared__ int s_total;
    __shared__ long long s_items[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;
    long long items = 0;
    for (int base = 0; base < nlist; base += blockDim.x) {
        const int l = base + threadIdx.x;
        const int v = l < nlist ? vis_count[l] : 0;
        const long long len = l < nlist ? offsets[l + 1] - offsets[l] : 0;
        const long long it = (long long)((v + SQ - 1) / SQ) * ((len + SC - 1) / SC);
        const int ex = block_exclusive_scan(v, s_warp, &s_total);
        long long in = it;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const long long up = __shfl_up_sync(0xffffffffu, in, o); if (lane >= o) in += up; }
        if (lane == 31) s_items[warp] = in;
        __syncthreads();
        long long before = 0, all = 0;
        for (int w = 0; w < 32; ++w) { const long long x = s_items[w]; if (w < warp) before += x; all += x; }
        if (l < nlist) { vis_off[l] = carry + ex; item_off[l] = items + before + in - it; }
        carry += s_total;
        items += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) { vis_off[nlist] = carry; item_off[nlist] = items; }
}

__global__ void k_flat_visitors(const int* __restrict__ probes, long long pairs, const int* __restrict__ slot, const int* __restrict__ vis_off,
                                int* __restrict__ visitors) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pairs || slot[i] < 0) return;
    visitors[vis_off[probes[i]] + slot[i]] = (int)i;
}

// Persistent CTAs over the tiles: (list, 32 of its visitors, 64 of its rows).  again: only the visitors of the queries it names, of which there are
// *n_again (null: all); a tile without one costs its look-ups.
__global__ void __launch_bounds__(kSmallThreads)
k_flat_tiles(const float* __restrict__ queries, int dim, int nprobe, const long long* __restrict__ offsets, int nlist, const float* __restrict__ rows,
             const int* __restrict__ vis_off, const long long* __restrict__ item_off, const int* __restrict__ visitors, const int* __restrict__ seg,
             long long stride, float* __restrict__ dist, const int* __restrict__ again, const int* __restrict__ n_again) {
    behind();
    if (again && *n_again == 0) return;
    extern __shared__ __align__(16) float s_flat[];
    __shared__ int s_list, s_pair[SQ];
    __shared__ long long s_dst[SQ];
    const int pitch = small_pitch(dim);
    float* qs = s_flat;
    float* cs = s_flat + SQ * pitch;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long total = item_off[nlist];
    const bool vec = rows_vec(queries, dim);
    for (long long item = blockIdx.x; item < total; item += gridDim.x) {
        __syncthreads();   // the previous tile is done with shared memory
        if (warp == 0) { const int l = scan::find_list(item_off, nlist, item); if (lane == 0) s_list = l; }
        __syncthreads();
        const int l = s_list;
        const int v0 = vis_off[l], nvis = vis_off[l + 1] - v0;
        const int groups = (nvis + SQ - 1) / SQ;
        const long long local = item - item_off[l];
        const int g = (int)(local % groups);
        const long long r0 = local / groups * SC, len = offsets[l + 1] - offsets[l];
        const int nv = min(SQ, nvis - g * SQ), nr = (int)min((long long)SC, len - r0);
        bool live = false;
        if (threadIdx.x < SQ) {
            int pair = threadIdx.x < nv ? visitors[v0 + g * SQ + threadIdx.x] : -1;
            const int q = pair >= 0 ? pair / nprobe : 0;
            if (again && pair >= 0 && !again[q]) pair = -1;
            live = pair >= 0;
            s_pair[threadIdx.x] = pair;
            if (live) s_dst[threadIdx.x] = (long long)q * stride + seg[(size_t)q * (nprobe + 1) + (pair - q * nprobe)] + r0;
        }
        if (again && !__syncthreads_or(live)) continue;
        stage_rows<kSmallThreads>(cs, pitch, rows + (size_t)(offsets[l] + r0) * dim, nr, dim);
        __syncthreads();
        for (int i = warp; i < nv; i += kSmallThreads / 32) if (s_pair[i] >= 0) stage_row(qs + i * pitch, queries + (size_t)(s_pair[i] / nprobe) * dim, dim, vec, lane);
        stage_wait();
        if ((s_pair[ty * 4] & s_pair[ty * 4 + 1] & s_pair[ty * 4 + 2] & s_pair[ty * 4 + 3]) >= 0) {   // one of the four visitors is wanted
            float acc[4][4];
            tile_distances(qs + ty * 4 * pitch, cs + tx * pitch, pitch, dim, acc);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (s_pair[ty * 4 + i] < 0) continue;
                float* out = dist + s_dst[ty * 4 + i];
#pragma unroll
                for (int j = 0; j < 4; ++j) if (tx + 16 * j < nr) out[tx + 16 * j] = acc[i][j];
            }
        }
    }
}

// Few visitors per list: a thread per (query, row).  grid (row blocks, queries).
__global__ void __launch_bounds__(128)
k_flat_rows(const float* __restrict__ queries, int dim, const int* __restrict__ probes, int nprobe, const long long* __restrict__ offsets,
            const float* __restrict__ rows, const int* __restrict__ seg, long long stride, float* __restrict__ dist, float* __restrict__ runs,
            long long run_stride) {
    extern __shared__ __align__(16) float s_q[];
    behind();
    const int q = blockIdx.y;
    const int* s = seg + (size_t)q * (nprobe + 1);
    const int n = s[nprobe];
    if ((int)(blockIdx.x * 128) >= n) return;
    for (int d = threadIdx.x; d < dim; d += 128) s_q[d] = queries[(size_t)q * dim + d];
    __syncthreads();
    const bool vec = rows_vec(rows, dim);
    float* out = dist + (size_t)q * stride;
    for (int i = blockIdx.x * 128 + threadIdx.x; i - (int)(threadIdx.x & 31) < n; i += gridDim.x * 128) {   // whole runs
        float sum = __int_as_float(0x7f800000);
        if (i < n) {
            int lo = 0, hi = nprobe;   // largest p with s[p] <= i
            while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s[mid] <= i) lo = mid; else hi = mid; }
            const float* x = rows + (size_t)(offsets[probes[(size_t)q * nprobe + lo]] + (i - s[lo])) * dim;
            out[i] = sum = row_distance(s_q, x, dim, vec);
        }
        if (runs) sel::store_run(runs + (size_t)q * run_stride, i / sel::kRun, sum);
    }
}

// One CTA per query: the topk nearest of its distances, ties by row; original ids out.  again: of the queries it names (null: of all).
template <int T>
__global__ void __launch_bounds__(T)
k_flat_select(const float* __restrict__ dist, long long stride, const int* __restrict__ probes, int nprobe, const long long* __restrict__ offsets,
              const int* __restrict__ seg, int topk, int buffer, const long long* __restrict__ ids, long long* __restrict__ out_ids,
              float* __restrict__ out_dist, const float* __restrict__ runs, long long run_stride, const int* __restrict__ again) {
    extern __shared__ __align__(16) uint64_t s_key[];   // [buffer] keys, the selection's runs, the segments (where they fit)
    __shared__ sel::Words w;
    behind();
    const int q = blockIdx.x;
    if (again && !again[q]) return;
    const int* s = seg + (size_t)q * (nprobe + 1);
    if (nprobe <= sel::kSegShared) {   // a search for every key: not in global memory
        int* s_seg = reinterpret_cast<int*>(s_key + buffer) + sel::kMaxGroups;
        for (int p = threadIdx.x; p <= nprobe; p += T) s_seg[p] = s[p];
        __syncthreads();
        s = s_seg;
    }
    auto row_of = [&](int i) -> uint32_t {
        int lo = 0, hi = nprobe;
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s[mid] <= i) lo = mid; else hi = mid; }
        return (uint32_t)(offsets[probes[(size_t)q * nprobe + lo]] + (i - s[lo]));
    };
    const int keep = sel::smallest<T>(dist + (size_t)q * stride, s[nprobe], topk, row_of, s_key, buffer, reinterpret_cast<int*>(s_key + buffer), &w,
                                      runs ? runs + (size_t)q * run_stride : nullptr);
    for (int i = threadIdx.x; i < topk; i += T) {
        const bool ok = i < keep;
        out_ids[(size_t)q * topk + i] = ok ? ids[key_idx(s_key[i])] : -1;
        out_dist[(size_t)q * topk + i] = ok ? key_dist(s_key[i]) : FLT_MAX;
    }
}

// ---- list form behind a filter --------------------------------------------------------------------------------------------------
// The distances of a list's visitors to its rows are a matrix product; in the reference's arithmetic they are three instructions per
// dimension and pair.  Where a selection follows anyway, the tiles are taken from mma.sync with both operands split into two bf16 terms
// (|q|^2 + |x|^2 - 2 q.x in fp32), the selection keeps every row that the approximate distance cannot rule out, and those - a few more
// than topk - are evaluated exactly.  (A list has sixty visitors in the benchmark's configuration, and
// often ten: too few for the M of a tcgen05 product.  With its rows as M and the visitors as N they would do; that form is not built.)
// Bound: latency, a tile being a chain of look-ups, two stagings and a short product; four CTAs an SM.  1,000 queries x 16 lists of 390 rows x 128,
// topk 10: tiles 163 -> 71 us, selection 14 -> 23, the whole call 244 -> 140.  Eight warps a tile 91, four rows' loads at a time 78.
//   Error of an approximate distance against the exact arithmetic's, S = (|q| + |x|)^2 <= 2 (|q|^2 + |x|^2):  products, splits 3.1 * 2^-18 and 3 K
//   additions of 2^-22 each, of |q||x| <= S / 4, twice; norms (K + 4) 2^-24 S; their sum 2^-22 S; the exact arithmetic's own (K + 2) 2^-23 S; and
//   2^-126 for each of 3 K products and 3 K partial sums that are subnormal and may vanish, twice: 12 K 2^-126 <= 3.7e-35 for the 256 dimensions the operands hold.
//   Together e = slack (|q|^2 + |x|^2) + 3.7e-35, and the tiles leave the lower bound, approximation - e.
//   The topk rows of the smallest lower bounds, t at most, lie within t + 2 e: of all rows in the visited lists |x|^2 is at most `most`, and of rows
//   with |x| >= 3 |q| the lower bound is at least ((2/3)^2 - 2 * 10/9 slack) |x|^2 >= 0.4 |x|^2, so that |x|^2 <= max(9 |q|^2, 2.5 t) for the topk: one row far
//   out does not loosen the bound for the others.  Only rows whose lower bound is below that can be among the topk.
//   A row whose norm is too large for a bound, or not a number, is evaluated for every query that visits its list.
// Where more than 1,024 rows are left - all rows far from the origin, or equally near by the thousand - the bound is no help: such queries are noted, and
// two more launches, which leave at once where there are none, take them through the exact tiles.  1,000 queries x 16 lists of 390 rows x 128, us: exact tiles
// for all
// 227, behind the filter 131; one row of 1,000 times the norm, or not a number, 131; an offset of 100 with a spread of 0.3 301; all rows the same 488 (exact
// tiles 376).  With one norm for the whole index and the way back in the selection's own block these were 926, 917 and 1,237.
constexpr int kFilterThreads = 128;   // four warps: 16 visitors x 32 rows each
constexpr float kFilterTiny = 3.7e-35f;
__host__ __device__ __forceinline__ int filter_dims(int dim) { return (dim + 15) / 16 * 16; }
__host__ __device__ __forceinline__ int filter_pitch(int dim) { return filter_dims(dim) + 8; }   // bf16 between rows: eight rows' 16 bytes in different banks
inline size_t filter_bytes(int dim) { return (size_t)(SQ + SC) * filter_pitch(dim) * 4; }
__device__ __forceinline__ float filter_slack(int dim) {   // <= 3.2e-4: operands of 256 dimensions at most
    const float k = (float)filter_dims(dim);
    return 2.0002f * (5.913e-6f + k * (3.577e-7f + 5.97e-8f + 1.193e-7f) + 1.0e-6f);
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Squared norms of the rows, and the largest of each list as the bits of a float (not a number: the largest of all).  A warp takes `per` rows, one
// after the other.
__global__ void __launch_bounds__(256) k_flat_norms(const float* __restrict__ rows, long long n, int dim, const long long* __restrict__ offsets, int nlist,
                                                    int per, float* __restrict__ norms, unsigned* __restrict__ most) {
    const int lane = threadIdx.x & 31;
    const long long r0 = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * per, r1 = min(n, r0 + per);
    if (r0 >= r1) return;
    int l = scan::find_list(offsets, nlist, r0);
    long long end = offsets[l + 1];
    unsigned top = 0;
    for (long long r = r0; r < r1; ++r) {
        if (r >= end) {
            if (lane == 0 && top) atomicMax(&most[l], top);
            top = 0;
            while (r >= end) end = offsets[++l + 1];
        }
        float s = 0.0f;
        for (int d = lane; d < dim; d += 32) { const float v = rows[(size_t)r * dim + d]; s = fmaf(v, v, s); }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) norms[r] = s;
        top = max(top, __float_as_uint(s) & 0x7fffffffu);
    }
    if (lane == 0 && top) atomicMax(&most[l], top);
}

__global__ void __launch_bounds__(kFilterThreads)
k_flat_tiles_filter(const float* __restrict__ queries, int dim, int nprobe, const long long* __restrict__ offsets, int nlist, const float* __restrict__ rows,
                    const float* __restrict__ norms, const int* __restrict__ vis_off, const long long* __restrict__ item_off,
                    const int* __restrict__ visitors, const int* __restrict__ seg, long long stride, float* __restrict__ dist) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ int s_list, s_pair[SQ];
    __shared__ long long s_dst[SQ];
    __shared__ float s_qn[SQ];
    const int pitch = filter_pitch(dim), dims = filter_dims(dim);
    __nv_bfloat16* qh = reinterpret_cast<__nv_bfloat16*>(s_raw);   // [SQ][pitch] visitors, high terms
    __nv_bfloat16* ql = qh + SQ * pitch;
    __nv_bfloat16* xh = ql + SQ * pitch;                           // [SC][pitch] rows
    __nv_bfloat16* xl = xh + SC * pitch;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long total = item_off[nlist];
    const float less = 1.0f - filter_slack(dim), none = __int_as_float(0x7fffffff);
    auto lower = [&](float dot, float norms2) { return norms2 < 1.0e36f ? fmaf(-2.0f, dot, fmaf(norms2, less, -kFilterTiny)) : none; };
    // One row by a warp, four elements a lane, several rows' loads before the first is used: two bf16 terms of each, and the squares' sum.
    auto stage = [&](auto src_of, int count, __nv_bfloat16* high, __nv_bfloat16* low, bool vec, auto sum_of) {
        constexpr int U = 8;
        for (int r0 = warp; r0 < count; r0 += U * (kFilterThreads / 32)) {
            float sums[U];
#pragma unroll
            for (int u = 0; u < U; ++u) sums[u] = 0.0f;
            for (int d = lane * 4; d < dims; d += 128) {
                float4 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int r = r0 + u * (kFilterThreads / 32);
                    v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (r >= count) continue;
                    const float* x = src_of(r) + d;
                    if (vec) { if (d < dim) v[u] = __ldg(reinterpret_cast<const float4*>(x)); }
                    else {
                        if (d < dim) v[u].x = __ldg(x);
                        if (d + 1 < dim) v[u].y = __ldg(x + 1);
                        if (d + 2 < dim) v[u].z = __ldg(x + 2);
                        if (d + 3 < dim) v[u].w = __ldg(x + 3);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int r = r0 + u * (kFilterThreads / 32);
                    if (r >= count) continue;
                    const __nv_bfloat162 h0 = __floats2bfloat162_rn(v[u].x, v[u].y), h1 = __floats2bfloat162_rn(v[u].z, v[u].w);
                    const __nv_bfloat162 l0 = __floats2bfloat162_rn(v[u].x - __low2float(h0), v[u].y - __high2float(h0)),
                                         l1 = __floats2bfloat162_rn(v[u].z - __low2float(h1), v[u].w - __high2float(h1));
                    uint2 w;
                    w.x = *reinterpret_cast<const uint32_t*>(&h0); w.y = *reinterpret_cast<const uint32_t*>(&h1);
                    *reinterpret_cast<uint2*>(high + (size_t)r * pitch + d) = w;
                    w.x = *reinterpret_cast<const uint32_t*>(&l0); w.y = *reinterpret_cast<const uint32_t*>(&l1);
                    *reinterpret_cast<uint2*>(low + (size_t)r * pitch + d) = w;
                    sums[u] = fmaf(v[u].x, v[u].x, fmaf(v[u].y, v[u].y, fmaf(v[u].z, v[u].z, fmaf(v[u].w, v[u].w, sums[u]))));
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) sum_of(r0 + u * (kFilterThreads / 32), sums[u]);
        }
    };
    for (long long item = blockIdx.x; item < total; item += gridDim.x) {
        __syncthreads();   // the previous tile is done with shared memory
        if (warp == 0) { const int l = scan::find_list(item_off, nlist, item); if (lane == 0) s_list = l; }
        __syncthreads();
        const int l = s_list;
        const int v0 = vis_off[l], nvis = vis_off[l + 1] - v0;
        const int groups = (nvis + SQ - 1) / SQ;
        const long long local = item - item_off[l];
        const int g = (int)(local % groups);
        const long long r0 = local / groups * SC, len = offsets[l + 1] - offsets[l], first = offsets[l] + r0;
        const int nv = min(SQ, nvis - g * SQ), nr = (int)min((long long)SC, len - r0);
        if (threadIdx.x < SQ) {
            const int pair = threadIdx.x < nv ? visitors[v0 + g * SQ + threadIdx.x] : -1;
            s_pair[threadIdx.x] = pair;
            if (pair >= 0) { const int q = pair / nprobe; s_dst[threadIdx.x] = (long long)q * stride + seg[(size_t)q * (nprobe + 1) + (pair - q * nprobe)] + r0; }
        }
        stage([&](int r) { return rows + (size_t)(first + r) * dim; }, nr, xh, xl, rows_vec(rows, dim), [](int, float) {});
        __syncthreads();
        stage([&](int r) { return queries + (size_t)(s_pair[r] / nprobe) * dim; }, nv, qh, ql, rows_vec(queries, dim), [&](int r, float sum) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane == 0 && r < nv) s_qn[r] = sum;
        });
        __syncthreads();
        const int m0 = (warp & 1) * 16, n0 = (warp >> 1) * 32;   // the warp's visitors and rows
        if (m0 >= nv || n0 >= nr) continue;
        float acc[4][4];
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[t][j] = 0.0f;
        const int arow = (m0 + (lane & 15)) * pitch + (lane >> 4) * 8, brow = (n0 + (lane & 7) + (lane >> 4) * 8) * pitch + ((lane >> 3) & 1) * 8;
#pragma unroll 2
        for (int k0 = 0; k0 < dims; k0 += 16) {   // (rows past nv and nr hold what an earlier tile left: their sums are not written)
            uint32_t ah[4], al[4], bh[2][4], bl[2][4];
            ldmatrix4(ah, qh + arow + k0);
            ldmatrix4(al, ql + arow + k0);
#pragma unroll
            for (int h = 0; h < 2; ++h) { ldmatrix4(bh[h], xh + brow + h * 16 * pitch + k0); ldmatrix4(bl[h], xl + brow + h * 16 * pitch + k0); }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                mma_bf16(acc[t], ah, bl[t >> 1][(t & 1) * 2], bl[t >> 1][(t & 1) * 2 + 1]);
                mma_bf16(acc[t], al, bh[t >> 1][(t & 1) * 2], bh[t >> 1][(t & 1) * 2 + 1]);
                mma_bf16(acc[t], ah, bh[t >> 1][(t & 1) * 2], bh[t >> 1][(t & 1) * 2 + 1]);
            }
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int c = n0 + t * 8 + (lane & 3) * 2;
            const float x0 = c < nr ? __ldg(norms + first + c) : 0.0f, x1 = c + 1 < nr ? __ldg(norms + first + c + 1) : 0.0f;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int v = m0 + (lane >> 2) + h * 8;
                if (v >= nv) continue;
                float* out = dist + s_dst[v] + c;
                const float qn = s_qn[v];
                if (c < nr) out[0] = lower(acc[t][h * 2], qn + x0);
                if (c + 1 < nr) out[1] = lower(acc[t][h * 2 + 1], qn + x1);
            }
        }
    }
}

// One CTA per query: the topk nearest of the rows that their lower bounds do not rule out, evaluated exactly; ties by row; original ids out.  A query
// with too many of them is noted in `again` and counted, and left.
template <int T>
__global__ void __launch_bounds__(T)
k_flat_select_filter(const float* __restrict__ dist, long long stride, const float* __restrict__ queries, int dim, const float* __restrict__ rows,
                     const unsigned* __restrict__ most, const int* __restrict__ probes, int nprobe, const long long* __restrict__ offsets, int nlist,
                     const int* __restrict__ seg, int topk, int buffer, const long long* __restrict__ ids, long long* __restrict__ out_ids,
                     float* __restrict__ out_dist, int* __restrict__ again, int* __restrict__ n_again) {
    extern __shared__ __align__(16) uint64_t s_key[];   // [buffer] keys, the query, the segments (where they fit)
    __shared__ sel::Words w;
    behind();
    float* s_q = reinterpret_cast<float*>(s_key + buffer);
    const int q = blockIdx.x, lane = threadIdx.x & 31;
    unsigned top = 0;   // the largest norm in the lists the query visits; the same in every warp
    for (int p = lane; p < nprobe; p += 32) {
        const int l = probes[(size_t)q * nprobe + p];
        if (l >= 0 && l < nlist) top = max(top, most[l]);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    const int* s = seg + (size_t)q * (nprobe + 1);
    for (int d = threadIdx.x; d < dim; d += T) s_q[d] = queries[(size_t)q * dim + d];
    if (nprobe <= sel::kSegShared) {
        int* s_seg = reinterpret_cast<int*>(s_q + ((dim + 3) & ~3));
        for (int p = threadIdx.x; p <= nprobe; p += T) s_seg[p] = s[p];
        s = s_seg;
    }
    if (threadIdx.x == 0) w.cnt = 0;
    __syncthreads();
    auto row_of = [&](int i) -> uint32_t {
        int lo = 0, hi = nprobe;
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s[mid] <= i) lo = mid; else hi = mid; }
        return (uint32_t)(offsets[probes[(size_t)q * nprobe + lo]] + (i - s[lo]));
    };
    const bool vec = rows_vec(rows, dim);
    const float* vals = dist + (size_t)q * stride;
    const int n = s[nprobe];
    const int keep = min(topk, n);
    float qn = 0.0f;
    for (int d = lane; d < dim; d += 32) qn = fmaf(s_q[d], s_q[d], qn);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) qn += __shfl_xor_sync(0xffffffffu, qn, o);   // the same in every warp
    const float inf = __int_as_float(0x7f800000);
    float cut = inf;
    if (n > 4 * topk && n >= 96) {   // as sel::smallest does
        float* s_min = reinterpret_cast<float*>(s_key);
        const int per = (2 * topk + T - 1) / T;
        for (int g = 0; g < per; ++g) {
            float m = inf;
#pragma unroll 8
            for (int i = threadIdx.x + g * T; i < n; i += per * T) m = fminf(m, vals[i]);
            s_min[g * T + threadIdx.x] = m;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            const float at = per == 1 ? sel::bound_of<T / 32>(s_min, T, topk) : sel::bound_of<0>(s_min, per * T, topk);
            if (lane == 0) w.cut = at;
        }
        __syncthreads();
        const float t = w.cut;
        cut = fmaf(2.0002f * filter_slack(dim), qn + fminf(__uint_as_float(top), fmaxf(9.0f * qn, 2.5f * t)), fmaf(fabsf(t), 1.0e-6f, t)) + 2.0f * 1.01f * kFilterTiny;
    }
#pragma unroll 8
    for (int i = threadIdx.x; i < n; i += T)
        if (!(vals[i] > cut)) {   // not a number: no bound
            const int pos = atomicAdd(&w.cnt, 1);
            if (pos < buffer) s_key[pos] = (uint64_t)i;
        }
    __syncthreads();
    const int c = w.cnt;
    const bool sure = c >= keep && c <= buffer;
    if (threadIdx.x == 0) {
        again[q] = sure ? 0 : 1;
        if (!sure) atomicAdd(n_again, 1);
    }
    if (!sure) return;
    for (int e = threadIdx.x; e < c; e += T) {
        const uint32_t r = row_of((int)s_key[e]);
        s_key[e] = make_key(row_distance(s_q, rows + (size_t)r * dim, dim, vec), r);
    }
    __syncthreads();
    sel::put_in_order<T>(s_key, c, topk);
    for (int i = threadIdx.x; i < topk; i += T) {
        const bool ok = i < keep;
        out_ids[(size_t)q * topk + i] = ok ? ids[key_idx(s_key[i])] : -1;
        out_dist[(size_t)q * topk + i] = ok ? key_dist(s_key[i]) : FLT_MAX;
    }
}

}  // namespace

psb_status launch_row_segments(const int* d_probes, int nq, int nprobe, const long long* d_offsets, int list_begin, int list_end, int* d_seg,
                               int* d_vis_count, int* d_slot, unsigned long long* d_counters, cudaStream_t s, bool chained, unsigned long long* mark) {
    PSB_TRY(launch_behind(chained, k_row_segments, dim3((unsigned)((nq + 3) / 4)), 128, 0, s, d_probes, nq, nprobe, d_offsets, list_begin, list_end, d_seg, d_vis_count, d_slot,
                          d_counters, mark));
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

bool flat_list_form(int nq, int nprobe, int nlist, long long rows, int dim) {
    // The list form's tiles read a list's rows once for 32 visitors: 2.4e-7 us for each dimension of a visited row against 1.0e-6 in the row
    // form, for 16 to 30 us more of launches.  Both forms of 225 drawn batches (dim 32 to 128, 20,000 to 300,000 rows in 64 to 512 lists, 4 to 32
    // probes, 4 to 1,000 queries): with the line at 4e7 visited dimensions the form taken is on average 0.1 % and at most 7 % slower than the
    // other, at 2e7 30 %, at 6e7 29, at eight visitors a list 42.  586-row lists of dim 96: 3 visitors 120 us in lists, 131 in rows, 12
    // visitors 194 and 386.  With one visitor a tile has no one to share with, whatever the batch visits.  The tile's rows have to fit.
    return (double)nq * nprobe * rows / nlist * dim >= 4e7 && (long long)nq * nprobe >= 2ll * nlist && small_tile_bytes(dim) <= (size_t)200 * 1024;
}

// The list form's tiles from the filter: its operands fit, the selection's buffer holds topk and what the slack lets through, and it pays.  For each
// query it saves 9.5e-8 us per dimension of a row visited (less 13 of them: what a row costs either way) and costs 5e-3 us and 7e-7 for each dimension of topk rows, which are evaluated again; up to four
// rows visited for each wanted there is no bound and all are.  Of 375 batches (dim 32 to 240, 1 to 16 probes, topk 1 to 256, 600 to 4,000 queries) the form taken is
// on average 0.9 % and at most 15 % slower than the other, and at most 4 % slower than the exact tiles; behind the filter always it was 12 % and 116 %.
// 1,000 queries x 4 lists of 195 rows x 96, topk 200: 179 -> 119 us; 16 lists, topk 100, which stay: 106 against 152.
bool flat_filter_form(int form, int dim, int topk, double visits) {
    if (form == 1 || form == 2 || topk > 256 || filter_bytes(dim) > (size_t)100 * 1024) return false;
    return form == 3 || (visits > 4.0 * topk && visits * (dim - 13) > 60000.0 + 9.0 * topk * dim);
}

psb_status launch_flat_norms(const float* d_rows, long long n, int dim, const long long* d_offsets, int nlist, float* d_norms, unsigned* d_most, cudaStream_t s) {
    PSB_CUDA(cudaMemsetAsync(d_most, 0, sizeof(unsigned) * (size_t)nlist, s));
    if (n <= 0) return PSB_OK;
    const int per = (int)((n + 32767) / 32768);
    k_flat_norms<<<(unsigned)((n + 8ll * per - 1) / (8ll * per)), 256, 0, s>>>(d_rows, n, dim, d_offsets, nlist, per, d_norms, d_most);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_flat_scan(const FlatScan& f, int nq, cudaStream_t s) {
    if (nq <= 0) return PSB_OK;
    if (f.topk <= 0 || f.topk > kMaxTopk) return fail(PSB_UNSUPPORTED_SHAPE, "flat scan supports topk in 1..2048");
    const bool lists = flat_list_form(nq, f.nprobe, f.nlist, f.n_rows, f.dim);
    bool filtered = false;   // the exact tiles and the selection take the queries for which the filter's bound did not hold
    const long long pairs = (long long)nq * f.nprobe;
    int* n_again = lists ? f.vis_count + f.nlist : nullptr;
    if (lists) PSB_CUDA(cudaMemsetAsync(f.vis_count, 0, sizeof(int) * ((size_t)f.nlist + 1), s));
    PSB_TRY(launch_row_segments(f.probes, nq, f.nprobe, f.offsets, 0, f.nlist, f.seg, f.vis_count, lists ? f.slot : nullptr, f.counters, s, true));
    if (lists) {
        k_flat_lists<<<1, 1024, 0, s>>>(f.vis_count, f.offsets, f.nlist, f.vis_off, f.item_off);
        count_launch();
        PSB_LAUNCH_CHECK();
        k_flat_visitors<<<(unsigned)((pairs + 255) / 256), 256, 0, s>>>(f.probes, pairs, f.slot, f.vis_off, f.visitors);
        count_launch();
        PSB_LAUNCH_CHECK();
        filtered = flat_filter_form(f.form, f.dim, f.topk, (double)f.nprobe * f.n_rows / f.nlist);
        if (filtered) {
            const size_t smem = filter_bytes(f.dim);
            PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_flat_tiles_filter), smem));
            const int per_sm = (int)std::max<size_t>(1, std::min<size_t>(8, (size_t)220 * 1024 / (smem + 2048)));
            k_flat_tiles_filter<<<(unsigned)(f.sm_count * per_sm), kFilterThreads, smem, s>>>(f.queries, f.dim, f.nprobe, f.offsets, f.nlist, f.rows, f.norms,
                                                                                              f.vis_off, f.item_off, f.visitors, f.seg, f.stride, f.dist);
            count_launch();
            PSB_LAUNCH_CHECK();
            const size_t keys = (size_t)sel::buffer_entries(f.topk) * 8 + (size_t)((f.dim + 3) & ~3) * 4 + (f.nprobe <= sel::kSegShared ? ((size_t)f.nprobe + 1) * sizeof(int) : 0);
            auto select = [&](auto kernel, int threads) -> psb_status {
                PSB_TRY(kernel_shared(reinterpret_cast<const void*>(kernel), keys));
                return launch_behind(select_behind(nq, f.sm_count, f.topk, 128), kernel, dim3((unsigned)nq), (unsigned)threads, keys, s, f.dist, f.stride, f.queries, f.dim, f.rows, f.most, f.probes, f.nprobe, f.offsets,
                                     f.nlist, f.seg, f.topk, sel::buffer_entries(f.topk), f.ids, f.out_ids, f.out_dist, f.again, n_again);
            };
            if (nq <= f.sm_count) PSB_TRY(select(k_flat_select_filter<1024>, 1024));
            else PSB_TRY(select(k_flat_select_filter<256>, 256));
            count_launch();
            PSB_LAUNCH_CHECK();
        }
        const size_t smem = small_tile_bytes(f.dim);
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_flat_tiles), smem));
        const int per_sm = (int)std::max<size_t>(1, std::min<size_t>(8, (size_t)220 * 1024 / (smem + 1024)));
        PSB_TRY(launch_behind(true, k_flat_tiles, dim3((unsigned)(f.sm_count * per_sm)), kSmallThreads, smem, s, f.queries, f.dim, f.nprobe, f.offsets, f.nlist, f.rows, f.vis_off,
                              f.item_off, f.visitors, f.seg, f.stride, f.dist, filtered ? f.again : nullptr, n_again));
    } else {
        const long long blocks = std::min<long long>((f.stride + 127) / 128, 8192);
        const size_t smem = (size_t)((f.dim + 3) & ~3) * sizeof(float);
        if (smem > 48 * 1024) PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_flat_rows), smem));
        // (behind: 8 queries x 8 lists of 428 rows of 64 25.4 us against 26.7, 32 29.4 and 31.3, 64 45.0 and 41.0, 128 62.9 and 55.4)
        PSB_TRY(launch_behind(nq <= 32, k_flat_rows, dim3((unsigned)std::max<long long>(1, blocks), (unsigned)nq), 128, smem, s, f.queries, f.dim, f.probes, f.nprobe, f.offsets, f.rows, f.seg, f.stride, f.dist, f.runs, f.run_stride));
    }
    count_launch();
    PSB_LAUNCH_CHECK();
    const size_t smem = sel::shared_bytes(f.topk) + (f.nprobe <= sel::kSegShared ? ((size_t)f.nprobe + 1) * sizeof(int) : 0);
    auto select = [&](auto kernel, int threads) -> psb_status {   // fewer queries than SMs: large blocks
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(kernel), smem));
        return launch_behind(select_behind(nq, f.sm_count, f.topk, 128), kernel, dim3((unsigned)nq), (unsigned)threads, smem, s, f.dist, f.stride, f.probes, f.nprobe, f.offsets, f.seg, f.topk, sel::buffer_entries(f.topk), f.ids, f.out_ids, f.out_dist, lists ? nullptr : f.runs, f.run_stride,
                             filtered ? f.again : nullptr);
    };
    if (nq <= f.sm_count) PSB_TRY(select(k_flat_select<1024>, 1024));
    else PSB_TRY(select(k_flat_select<256>, 256));
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

}  // namespace psb
