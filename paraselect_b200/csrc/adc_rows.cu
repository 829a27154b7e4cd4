// ADC scan, row form: every distance of every query, then the stage1_k smallest of each query's row of distances.
//
// The list-centric scans (pq_scan.cu, scan_tc.cu) sample a cutoff, schedule the visitors of every list, filter, re-score and sort pools:
// about 180 us of kernels that a small batch pays in full, most of them one CTA per query.  Here a CTA builds the query's table in shared
// memory (residual mode: the table of a (query, probe) pair; a caller's own tables are read instead), scores its share of the query's rows
// with it and writes the distances out; nothing is sampled, scheduled or re-scored, and a query's rows spread over the chip.  Bound:
// shared-memory gathers, m per row visit, about 3.5 cycles per warp-wide gather of random banks.  The selection is select.cuh's, reading
// each distance twice, or (plain mode) the minima of 32 and the distances of the runs that matter.
// Same arithmetic and order as the other scans (reference: src/search/ivfpq/stage/ivfpq_fine_cpu_lut.cpp:51-63,76-80;
// src/search/ivfrespq/stage/ivfrespq_cpu_rerank.cpp:87-130,226-259,440-451), so the same candidates.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "scan_common.cuh"
#include "select.cuh"

namespace psb {

using namespace scan;

namespace {

constexpr int kRowsThreads = 256;

// The table of the (residual) query in s_q: entry = sequential non-fused sum of (q - c)^2 over the sub-vector.
__device__ __forceinline__ void build_table(float* __restrict__ s_tab, const float* __restrict__ s_q, const float* __restrict__ codebook, int m, int k, int dsub) {
    auto add = [](float e, float q, float c) { const float t = __fsub_rn(q, c); return __fadd_rn(e, __fmul_rn(t, t)); };
    const bool wide = (reinterpret_cast<uintptr_t>(codebook) & 15) == 0;
#pragma unroll 8
    for (int e = threadIdx.x; e < m * k; e += kRowsThreads) {
        const int sub = k == 256 ? e >> 8 : e / k;
        const float* q = s_q + sub * dsub;
        float d = 0.0f;
        if (dsub == 2 && wide) {
            const float2 c = __ldg(reinterpret_cast<const float2*>(codebook) + e);
            d = add(add(d, q[0], c.x), q[1], c.y);
        } else if (dsub == 4 && wide) {
            const float4 c = __ldg(reinterpret_cast<const float4*>(codebook) + e);
            d = add(add(add(add(d, q[0], c.x), q[1], c.y), q[2], c.z), q[3], c.w);
        } else if (dsub == 8 && wide) {
            const float4 c = __ldg(reinterpret_cast<const float4*>(codebook) + 2 * (size_t)e), b = __ldg(reinterpret_cast<const float4*>(codebook) + 2 * (size_t)e + 1);
            d = add(add(add(add(d, q[0], c.x), q[1], c.y), q[2], c.z), q[3], c.w);
            d = add(add(add(add(d, q[4], b.x), q[5], b.y), q[6], b.z), q[7], b.w);
        } else {
            for (int i = 0; i < dsub; ++i) d = add(d, q[i], __ldg(codebook + (size_t)e * dsub + i));
        }
        s_tab[e] = d;
    }
}

// The table of a block: the caller's where there is one, else built on the (residual) query in s_q.
__device__ __forceinline__ void block_table(float* __restrict__ s_tab, const float* __restrict__ s_q, const AdcRows& g, long long table) {
    if (g.lut) {
        const float* from = g.lut + (size_t)table * g.m * g.k;
#pragma unroll 8
        for (int e = threadIdx.x; e < g.m * g.k; e += kRowsThreads) s_tab[e] = __ldg(from + e);
    } else {
        build_table(s_tab, s_q, g.codebook, g.m, g.k, g.dim / g.m);
    }
}

// Plain mode: grid (row blocks, queries); a block takes `block_rows` consecutive rows of the query's probed lists laid end to end.
template <int M>
__global__ void __launch_bounds__(kRowsThreads)
k_adc_rows(const AdcRows g, int block_rows) {
    behind();
    extern __shared__ __align__(16) float s_rows[];
    float* s_tab = s_rows;                                      // [m * k]
    float* s_q = s_rows + g.m * g.k;                            // [dim]
    int* s_seg = reinterpret_cast<int*>(s_q + g.dim);           // [nprobe + 1]
    const int q = blockIdx.y;
    const int* seg = g.seg + (size_t)q * (g.nprobe + 1);
    const int n = seg[g.nprobe];
    const int i0 = blockIdx.x * block_rows, i1 = min(n, i0 + block_rows);
    if (i0 >= n) return;
    for (int d = threadIdx.x; d < g.dim; d += kRowsThreads) s_q[d] = g.queries[(size_t)q * g.dim + d];
    for (int p = threadIdx.x; p <= g.nprobe; p += kRowsThreads) s_seg[p] = seg[p];
    __syncthreads();
    block_table(s_tab, s_q, g, q);
    __syncthreads();
    float* out = g.dist + (size_t)q * g.stride;
    const int lane = threadIdx.x & 31;
    for (int i = i0 + threadIdx.x; i - lane < i1; i += kRowsThreads) {   // whole runs: i0 and the warps' strides are multiples of 32
        float d = __int_as_float(0x7f800000);
        if (i < i1) {
            int lo = 0, hi = g.nprobe;   // largest p with seg[p] <= i
            while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s_seg[mid] <= i) lo = mid; else hi = mid; }
            const long long row = g.offsets[g.probes[(size_t)q * g.nprobe + lo]] + (i - s_seg[lo]);
            out[i] = d = adc_row<M>(g.codes + (size_t)(row - g.row_base) * g.m, s_tab, g.m, g.k, false);
        }
        if (g.runs) sel::store_run(g.runs + (size_t)q * g.run_stride, i / sel::kRun, d);
    }
}

// Residual mode: block = (pair, chunk of block_rows rows of its list).
template <int M>
__global__ void __launch_bounds__(kRowsThreads)
k_adc_pair_rows(const AdcRows g, int block_rows, int chunks) {
    behind();
    extern __shared__ __align__(16) float s_rows[];
    float* s_tab = s_rows;
    float* s_q = s_rows + g.m * g.k;
    const long long pair = blockIdx.x / chunks;
    const int chunk = (int)(blockIdx.x - pair * chunks), q = (int)(pair / g.nprobe), p = (int)(pair - (long long)q * g.nprobe);
    const int l = g.probes[pair];
    if (l < g.list_begin || l >= g.list_end) return;
    const long long b = g.offsets[l], len = g.offsets[l + 1] - b;
    const long long r0 = (long long)chunk * block_rows, r1 = min(len, r0 + block_rows);
    if (r0 >= len) return;
    for (int d = threadIdx.x; d < g.dim; d += kRowsThreads)
        s_q[d] = __fsub_rn(g.queries[(size_t)q * g.dim + d], __ldg(g.centroids + (size_t)l * g.dim + d));
    __syncthreads();
    block_table(s_tab, s_q, g, pair);
    __syncthreads();
    float* out = g.dist + (size_t)q * g.stride + g.seg[(size_t)q * (g.nprobe + 1) + p];
    for (long long r = r0 + threadIdx.x; r < r1; r += kRowsThreads)
        out[r] = adc_row<M>(g.codes + (size_t)(b + r - g.row_base) * g.m, s_tab, g.m, g.k, g.tree != 0);
}

template <int T>
__global__ void __launch_bounds__(T)
k_adc_select(const AdcRows g, int buffer) {
    behind();
    extern __shared__ __align__(16) uint64_t s_key[];   // [buffer] keys, the selection's runs, the segments (where they fit)
    __shared__ sel::Words w;
    const int q = blockIdx.x;
    const int* s = g.seg + (size_t)q * (g.nprobe + 1);
    if (g.nprobe <= sel::kSegShared) {   // a search for every key: not in global memory
        int* s_seg = reinterpret_cast<int*>(s_key + buffer) + sel::kMaxGroups;
        for (int p = threadIdx.x; p <= g.nprobe; p += T) s_seg[p] = s[p];
        __syncthreads();
        s = s_seg;
    }
    auto row_of = [&](int i) -> uint32_t {
        int lo = 0, hi = g.nprobe;
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s[mid] <= i) lo = mid; else hi = mid; }
        const int l = g.probes[(size_t)q * g.nprobe + lo];
        return (uint32_t)(g.offsets[l] + (i - s[lo]) + (g.row_delta ? g.row_delta[l] : 0));
    };
    const int keep = sel::smallest<T>(g.dist + (size_t)q * g.stride, s[g.nprobe], g.stage1_k, row_of, s_key, buffer, reinterpret_cast<int*>(s_key + buffer), &w,
                                      g.runs ? g.runs + (size_t)q * g.run_stride : nullptr);
    for (int i = threadIdx.x; i < g.stage1_k; i += T) {
        const bool ok = i < keep;
        g.out_rows[(size_t)q * g.stage1_k + i] = ok ? (int)key_idx(s_key[i]) : -1;
        if (g.out_dist) g.out_dist[(size_t)q * g.stage1_k + i] = ok ? key_dist(s_key[i]) : FLT_MAX;
    }
    if (threadIdx.x == 0) {
        if (g.out_count) g.out_count[q] = keep;
        atomicAdd(&g.counters[1], (unsigned long long)keep);
    }
}

template <int M>
psb_status run_rows(const AdcRows& g, int nq, cudaStream_t s) {
    const int block = adc_rows_block((double)nq * g.expected_rows, g.sm_count);
    const size_t tab = ((size_t)g.m * g.k + g.dim) * sizeof(float);
    if (g.residual) {
        const int chunks = (int)std::max<long long>(1, (g.longest_list + block - 1) / block);
        const long long blocks = (long long)nq * g.nprobe * chunks;
        if (blocks > 0x7fffffffLL) return fail(PSB_UNSUPPORTED_SHAPE, "too many (query, probe) pairs in one batch");
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_adc_pair_rows<M>), tab));
        // (behind: 128 queries x 8 of 700 lists of 428 rows, m 16, the call 75.8 us against 84.1, 333 115 and 108, 1,000 x 32 579 and 522)
        PSB_TRY(launch_behind(nq <= g.sm_count, k_adc_pair_rows<M>, dim3((unsigned)blocks), kRowsThreads, tab, s, g, block, chunks));
    } else {
        const size_t smem = tab + ((size_t)g.nprobe + 1) * sizeof(int);
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_adc_rows<M>), smem));
        PSB_TRY(launch_behind(true, k_adc_rows<M>, dim3((unsigned)((g.stride + block - 1) / block), (unsigned)nq), kRowsThreads, smem, s, g, block));
    }
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

}  // namespace

psb_status launch_adc_rows(const AdcRows& g, int nq, cudaStream_t s) {
    if (nq <= 0) return PSB_OK;
    PSB_TRY(launch_row_segments(g.probes, nq, g.nprobe, g.offsets, g.list_begin, g.list_end, g.seg, nullptr, nullptr, g.counters, s, g.chained, g.mark));
    switch (g.m) {
        case 8: PSB_TRY(run_rows<8>(g, nq, s)); break;
        case 16: PSB_TRY(run_rows<16>(g, nq, s)); break;
        case 20: PSB_TRY(run_rows<20>(g, nq, s)); break;
        case 24: PSB_TRY(run_rows<24>(g, nq, s)); break;
        case 32: PSB_TRY(run_rows<32>(g, nq, s)); break;
        case 48: PSB_TRY(run_rows<48>(g, nq, s)); break;
        case 64: PSB_TRY(run_rows<64>(g, nq, s)); break;
        default: PSB_TRY(run_rows<0>(g, nq, s)); break;
    }
    const int buffer = sel::buffer_entries(g.stage1_k);
    const size_t smem = sel::shared_bytes(g.stage1_k) + (g.nprobe <= sel::kSegShared ? ((size_t)g.nprobe + 1) * sizeof(int) : 0);
    // Fewer queries than SMs: one selecting block per SM at most, so a large one.
    auto select = [&](auto kernel, int threads) -> psb_status {
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(kernel), smem));
        return launch_behind(select_behind(nq, g.sm_count, g.stage1_k, 128), kernel, dim3((unsigned)nq), (unsigned)threads, smem, s, g, buffer);
    };
    if (nq <= g.sm_count) PSB_TRY(select(k_adc_select<1024>, 1024));
    else PSB_TRY(select(k_adc_select<256>, 256));
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

}  // namespace psb
