// The re-scoring selection behind the tensor-core scan (scan_tc.cu): exact distances of the filter's survivors and the stage1_k
// smallest of each query.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "scan_common.cuh"

namespace psb {

using namespace scan;

namespace {

// A pool entry is either an exact key (distance bits with the top bit set: written by the SIMT
// scans) or an unscored survivor of the tensor-core filter: (list id, or in residual mode the (query, probe) pair) << 32 |
// scanned row.  Unscored entries get their exact fp32 ADC distance here - plain mode from the query's fp32 table staged in
// shared memory, residual mode from the pair's residual and the codebook, both in the CPU path's summation order - and are
// dropped when it exceeds the cutoff.  The keys stay in registers; a bisection over them finds a bound with stage1_k to
// next_pow2(stage1_k) keys below it, and only these are sorted.  A pool that overflowed, or holds fewer than min(stage1_k, rows
// scanned) entries within the cutoff, sends the query to the exact fallback.
//
// What it replaces sorted the whole pool in shared memory (8,192 keys: 50 of a block's 110 us at stage1_k = 1000) and, in residual
// mode, gathered codewords and centroids dimension by dimension through L1 (130 us per query of 1,500 survivors; 880 us for
// 2,000 queries).  Residual mode now keeps the codebook in shared memory, one persistent block per SM, and the query's residual
// against each probe beside it.
struct RescoreArgs {
    const uint64_t* pool; const int* pool_cnt; int pool_cap;
    const long long* q_rows; const float* thr; int stage1_k, nq;
    const float* lut;          // plain mode: [nq][m * k]
    const float* queries; const float* centroids; const float* codebook; const int* probes; int nprobe, dim, nlist;  // residual mode
    const uint8_t* codes; long long row_base; const long long* row_delta;
    int m, k, residual, tree;
    int* out_rows; float* out_dist; int* out_count;
    int* fail_list; int* n_fail; unsigned long long* counters;
    int shared_cut;   // the cutoff covers the rows of all shards: this shard need not reach stage1_k rows
    int sort_n;       // next_pow2(stage1_k)
    int staged;       // residual mode: codebook and residuals fit shared memory (else they are read through L1)
    int above, upto;  // the launch takes the queries with more pooled rows than this, and at most that many
};

__host__ __device__ __forceinline__ int residual_pitch(int dim, int dsub) { return dim + dsub; }   // residuals of different probes in different banks

// Exact residual-mode distance of one code row: res the residual of its pair, book the codebook, both in shared memory.
template <int DSUB>
__device__ __forceinline__ float residual_entry(const float* __restrict__ r, const float* __restrict__ c) {
    float v[DSUB], w[DSUB];
    if constexpr (DSUB == 2) {
        const float2 a = *reinterpret_cast<const float2*>(r), b = *reinterpret_cast<const float2*>(c);
        v[0] = a.x; v[1] = a.y; w[0] = b.x; w[1] = b.y;
    } else {
#pragma unroll
        for (int d = 0; d < DSUB; d += 4) {
            const float4 a = *reinterpret_cast<const float4*>(r + d), b = *reinterpret_cast<const float4*>(c + d);
            v[d] = a.x; v[d + 1] = a.y; v[d + 2] = a.z; v[d + 3] = a.w; w[d] = b.x; w[d + 1] = b.y; w[d + 2] = b.z; w[d + 3] = b.w;
        }
    }
    float e = 0.0f;
#pragma unroll
    for (int d = 0; d < DSUB; ++d) { const float t = __fsub_rn(v[d], w[d]); e = __fadd_rn(e, __fmul_rn(t, t)); }
    return e;
}
// (Not inlined: a thread's keys sit in registers, so the loop over them is unrolled sixteen times around the call.)
template <int DSUB, int TREE>   // TREE: 8 or 16 sub-quantisers summed as a pairwise tree, 0: any number, in sequence
__device__ __noinline__ float residual_row(const uint8_t* __restrict__ row, const float* __restrict__ res, const float* __restrict__ book, int m, int k) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(row);
    if constexpr (TREE > 0) {
        float t[TREE];
#pragma unroll
        for (int w = 0; w < TREE / 4; ++w) {
            const uint32_t c = __ldg(p + w);
#pragma unroll
            for (int j = 0; j < 4; ++j) t[w * 4 + j] = residual_entry<DSUB>(res + (w * 4 + j) * DSUB, book + ((size_t)(w * 4 + j) * k + ((c >> (8 * j)) & 255u)) * DSUB);
        }
        return tree_sum<TREE>(t);
    } else {
        float acc = 0.0f;
#pragma unroll 4
        for (int w = 0; w < (m >> 2); ++w) {
            const uint32_t c = __ldg(p + w);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                acc = __fadd_rn(acc, residual_entry<DSUB>(res + (w * 4 + j) * DSUB, book + ((size_t)(w * 4 + j) * k + ((c >> (8 * j)) & 255u)) * DSUB));
        }
        return acc;
    }
}

template <int M>
__device__ __noinline__ float plain_row(const uint8_t* __restrict__ row, const float* __restrict__ tab, int m, int k) { return adc_row<M>(row, tab, m, k, false); }
template <int M>
__device__ __noinline__ float direct_row(const uint8_t* __restrict__ row, const float* __restrict__ q, const float* __restrict__ book, int m, int k, int dsub,
                                         const float* __restrict__ cen) { return adc_row_direct<M>(row, q, book, m, k, dsub, M > 0, cen); }

// Sum of one int per thread over the block; s [2][32] alternates between calls, one barrier each.
template <int T>
__device__ __forceinline__ int block_count(int v, int* s) {
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = (threadIdx.x & 31) < T / 32 ? s[threadIdx.x & 31] : 0;
    return __reduce_add_sync(0xffffffffu, t);
}

// The query's keys are in registers (KEY_MAX: none): writes its stage1_k smallest, or puts it on the fail list.
template <int T, int KPT>
__device__ __forceinline__ void select_keys(const RescoreArgs& g, int q, long long need, const uint64_t (&key)[KPT], uint64_t* s_keys, int* s_cnt, int* s_pos) {
    int flip = 0, mine = 0;
#pragma unroll
    for (int j = 0; j < KPT; ++j) mine += key[j] != KEY_MAX ? 1 : 0;
    const int nv = block_count<T>(mine, s_cnt + 32 * (flip ^= 1));
    if (nv < need) {
        if (threadIdx.x == 0) g.fail_list[atomicAdd(g.n_fail, 1)] = q;
        return;
    }
    const int want = nv < g.stage1_k ? nv : g.stage1_k;
    uint64_t cut = KEY_MAX - 1;
    int below = nv;
    if (nv > g.sort_n) {
        uint64_t lo = KEY_MAX, hi = 0;
#pragma unroll
        for (int j = 0; j < KPT; ++j) if (key[j] != KEY_MAX) { lo = key[j] < lo ? key[j] : lo; hi = key[j] > hi ? key[j] : hi; }
        // the block's extremes by the high words (distances); the low word takes any row
        const unsigned l32 = __reduce_min_sync(0xffffffffu, (unsigned)(lo >> 32)), h32 = __reduce_max_sync(0xffffffffu, (unsigned)(hi >> 32));
        if (threadIdx.x == 0) { s_pos[1] = -1; s_pos[2] = 0; }
        __syncthreads();
        if ((threadIdx.x & 31) == 0) { atomicMin(reinterpret_cast<unsigned*>(s_pos + 1), l32); atomicMax(reinterpret_cast<unsigned*>(s_pos + 2), h32); }
        __syncthreads();
        lo = (uint64_t)(unsigned)s_pos[1] << 32; hi = ((uint64_t)(unsigned)s_pos[2] << 32) | 0xffffffffu;
        for (int it = 0; it < 70 && lo < hi; ++it) {
            const uint64_t mid = lo + ((hi - lo) >> 1);
            int c = 0;
#pragma unroll
            for (int j = 0; j < KPT; ++j) c += key[j] <= mid ? 1 : 0;
            c = block_count<T>(c, s_cnt + 32 * (flip ^= 1));
            if (c < want) { lo = mid + 1; continue; }
            hi = mid; cut = mid; below = c;
            if (c <= g.sort_n) break;
        }
        if (below > g.sort_n) {   // one key many times over (a list probed twice): the fallback sorts it out
            if (threadIdx.x == 0) g.fail_list[atomicAdd(g.n_fail, 1)] = q;
            return;
        }
    }
    if (threadIdx.x == 0) { *s_pos = 0; atomicAdd(&g.counters[1], (unsigned long long)nv); }
    const int n = next_pow2(max(below, 2));
    for (int i = below + threadIdx.x; i < n; i += T) s_keys[i] = KEY_MAX;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < KPT; ++j) if (key[j] <= cut) s_keys[atomicAdd(s_pos, 1)] = key[j];
    __syncthreads();
    block_bitonic_sort(s_keys, n);
    for (int i = threadIdx.x; i < g.stage1_k; i += T) {
        const bool ok = i < want;
        g.out_rows[(size_t)q * g.stage1_k + i] = ok ? (int)key_idx(s_keys[i]) : -1;
        if (g.out_dist) g.out_dist[(size_t)q * g.stage1_k + i] = ok ? key_dist(s_keys[i]) : FLT_MAX;
    }
    if (g.out_count && threadIdx.x == 0) g.out_count[q] = want;
}

// Rows the query owes, or -1 when its pool cannot answer (it goes on the fail list).
__device__ __forceinline__ long long rescore_need(const RescoreArgs& g, int q, int c) {
    const long long N = g.q_rows[q];
    long long need = N < g.stage1_k ? N : g.stage1_k;
    if (g.shared_cut && g.thr[q] < __int_as_float(0x7f800000)) need = 0;   // sharded search: the shards owe stage1_k rows together
    if (c > g.pool_cap || c < need) {
        if (threadIdx.x == 0) g.fail_list[atomicAdd(g.n_fail, 1)] = q;
        return -1;
    }
    return need;
}

template <int M, int T, int KPT>
__global__ void __launch_bounds__(T, T == 512 && KPT <= 8 ? 2 : 1) k_select_rescore(const RescoreArgs g) {
    extern __shared__ __align__(16) unsigned char s_sel[];
    uint64_t* s_keys = reinterpret_cast<uint64_t*>(s_sel);                      // [sort_n]
    float* s_tab = reinterpret_cast<float*>(s_sel + (size_t)g.sort_n * 8);      // [m * k]
    __shared__ int s_cnt[64], s_pos[3];
    const int q = blockIdx.x;
    const int c = g.pool_cnt[q];
    if (c <= g.above || c > g.upto) return;
    const long long need = rescore_need(g, q, c);
    if (need < 0) return;
    const int mk = g.m * g.k;
    const float* lut = g.lut + (size_t)q * mk;
    if ((mk & 3) == 0 && (reinterpret_cast<uintptr_t>(g.lut) & 15) == 0) {   // a caller's tables may start at any float
#pragma unroll 4
        for (int e = threadIdx.x; e < mk / 4; e += T) reinterpret_cast<float4*>(s_tab)[e] = __ldg(reinterpret_cast<const float4*>(lut) + e);
    } else {
        for (int e = threadIdx.x; e < mk; e += T) s_tab[e] = lut[e];
    }
    const float cut = g.thr[q];
    uint64_t key[KPT];
#pragma unroll
    for (int j = 0; j < KPT; ++j) { const int i = threadIdx.x + j * T; key[j] = i < c ? g.pool[(size_t)q * g.pool_cap + i] : KEY_MAX; }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
        if (key[j] >> 63) continue;   // exact already (and within the cutoff), or none
        const long long r = (long long)(uint32_t)key[j];
        const int l = (int)(key[j] >> 32);
        const float d = plain_row<M>(g.codes + (size_t)(r - g.row_base) * g.m, s_tab, g.m, g.k);
        key[j] = d <= cut ? make_key(d, (uint32_t)(r + (g.row_delta ? g.row_delta[l] : 0))) : KEY_MAX;
    }
    select_keys<T, KPT>(g, q, need, key, s_keys, s_cnt, s_pos);
}

// Takes the queries with more than g.above and at most g.upto pooled rows.
template <int DSUB, int TREE, int T, int KPT>
__global__ void __launch_bounds__(T, T == 512 && KPT <= 8 ? 2 : 1) k_select_rescore_residual(const RescoreArgs g) {
    extern __shared__ __align__(16) unsigned char s_sel[];
    const int pitch = residual_pitch(g.dim, DSUB);
    float* s_book = reinterpret_cast<float*>(s_sel);                            // [m][k][DSUB] when staged
    uint64_t* s_keys = reinterpret_cast<uint64_t*>(s_book + (g.staged ? (size_t)g.m * g.k * DSUB : 0));   // [sort_n]
    float* s_res = reinterpret_cast<float*>(s_keys + g.sort_n);                 // staged: [nprobe][pitch] residuals, else the query [dim]
    __shared__ int s_cnt[64], s_pos[3];
    bool there = !g.staged;   // the codebook
    for (int q = blockIdx.x; q < g.nq; q += gridDim.x) {
        const int c = g.pool_cnt[q];
        if (c <= g.above || c > g.upto) continue;   // uniform
        if (!there) {
            const int n4 = g.m * g.k * DSUB / 4;
#pragma unroll 4
            for (int i = threadIdx.x; i < n4; i += T) reinterpret_cast<float4*>(s_book)[i] = __ldg(reinterpret_cast<const float4*>(g.codebook) + i);
            there = true;
        }
        __syncthreads();   // the previous query is done with shared memory
        const long long need = rescore_need(g, q, c);
        if (need < 0) continue;   // uniform
        const float* qv = g.queries + (size_t)q * g.dim;
        uint64_t key[KPT];
#pragma unroll
        for (int j = 0; j < KPT; ++j) { const int i = threadIdx.x + j * T; key[j] = i < c ? g.pool[(size_t)q * g.pool_cap + i] : KEY_MAX; }
        if (g.staged) {
            for (int p = threadIdx.x >> 5; p < g.nprobe; p += T / 32) {
                const int l = g.probes[(size_t)q * g.nprobe + p];
                if (l < 0 || l >= g.nlist) continue;
                for (int d = threadIdx.x & 31; d < g.dim; d += 32) s_res[p * pitch + d] = __fsub_rn(__ldg(qv + d), __ldg(g.centroids + (size_t)l * g.dim + d));
            }
        } else {
            for (int d = threadIdx.x; d < g.dim; d += T) s_res[d] = __ldg(qv + d);
        }
        const float cut = g.thr[q];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            if (key[j] >> 63) continue;
            const long long r = (long long)(uint32_t)key[j];
            const int pair = (int)(key[j] >> 32);
            const uint8_t* row = g.codes + (size_t)(r - g.row_base) * g.m;
            float d;
            if (g.staged) {
                d = residual_row<DSUB, TREE>(row, s_res + (pair - q * g.nprobe) * pitch, s_book, g.m, g.k);
            } else {
                d = direct_row<TREE>(row, s_res, g.codebook, g.m, g.k, DSUB, g.centroids + (size_t)g.probes[pair] * g.dim);
            }
            key[j] = d <= cut ? make_key(d, (uint32_t)(r + (g.row_delta ? g.row_delta[g.probes[pair]] : 0))) : KEY_MAX;
        }
        select_keys<T, KPT>(g, q, need, key, s_keys, s_cnt, s_pos);
    }
}

// Threads and keys per thread by the pool's capacity (pool_capacity: a power of two from 1,024 to 16,384).
template <typename F>
psb_status by_capacity(int cap, F run) {
    if (cap <= 1024) return run(std::integral_constant<int, 256>(), std::integral_constant<int, 4>());
    if (cap <= 2048) return run(std::integral_constant<int, 256>(), std::integral_constant<int, 8>());
    if (cap <= 4096) return run(std::integral_constant<int, 256>(), std::integral_constant<int, 16>());
    if (cap <= 8192) return run(std::integral_constant<int, 512>(), std::integral_constant<int, 16>());
    return run(std::integral_constant<int, 1024>(), std::integral_constant<int, 16>());
}
// A pool is sized for sixteen times the rows wanted, and rarely holds twice as many: with room for 2,048 (4,096) keys a thread needs half the
// registers, and two blocks of 512 share an SM, one's latencies behind the other's work.  The few queries with more go to a launch of their own.
template <typename F>
psb_status by_pool(RescoreArgs& g, F run) {
    const int usual = g.stage1_k <= 512 ? 2048 : 4096;
    g.above = -1; g.upto = INT_MAX;
    if (g.pool_cap > usual) {
        g.upto = usual;
        if (usual == 2048) PSB_TRY(run(std::integral_constant<int, 512>(), std::integral_constant<int, 4>()));
        else PSB_TRY(run(std::integral_constant<int, 512>(), std::integral_constant<int, 8>()));
        count_launch();
        PSB_LAUNCH_CHECK();
        g.above = usual; g.upto = INT_MAX;
    }
    return by_capacity(g.pool_cap, run);
}
template <int M>
psb_status run_select_rescore(RescoreArgs g, cudaStream_t s) {
    const size_t smem = (size_t)g.sort_n * 8 + (size_t)g.m * g.k * 4;
    if (smem > (size_t)220 * 1024) return fail(PSB_UNSUPPORTED_SHAPE, "re-scoring selection does not fit shared memory");
    return by_pool(g, [&](auto t, auto kpt) -> psb_status {
        constexpr int T = decltype(t)::value, KPT = decltype(kpt)::value;
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_select_rescore<M, T, KPT>), smem));
        PSB_TRY(prefer_max_shared(k_select_rescore<M, T, KPT>));
        k_select_rescore<M, T, KPT><<<g.nq, T, smem, s>>>(g);
        return PSB_OK;
    });
}
template <int DSUB, int TREE>
psb_status run_select_rescore_residual(RescoreArgs g, int sm_count, cudaStream_t s) {
    const size_t keys = (size_t)g.sort_n * 8, book = (size_t)g.m * g.k * DSUB * 4, res = (size_t)g.nprobe * residual_pitch(g.dim, DSUB) * 4;
    g.staged = keys + book + res <= (size_t)220 * 1024 && ((size_t)g.m * g.k * DSUB) % 4 == 0 ? 1 : 0;
    const size_t smem = keys + (g.staged ? book + res : (size_t)g.dim * 4);
    auto run = [&](auto t, auto kpt) -> psb_status {
        constexpr int T = decltype(t)::value, KPT = decltype(kpt)::value;
        auto kernel = k_select_rescore_residual<DSUB, TREE, T, KPT>;
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(kernel), smem));
        PSB_TRY(prefer_max_shared(kernel));
        // An SM's 228 KB, of which a block takes one for itself, and the static words.
        const int per_sm = (int)std::max<size_t>(1, std::min<size_t>((size_t)228 * 1024 / (smem + 1024 + 272), 1024 / T));
        kernel<<<(unsigned)std::min(g.nq, sm_count * per_sm), T, smem, s>>>(g);
        return PSB_OK;
    };
    return by_pool(g, run);
}
template <int DSUB>
psb_status run_select_rescore_tree(const RescoreArgs& g, int sm_count, cudaStream_t s) {
    if (g.tree && g.m == 8) return run_select_rescore_residual<DSUB, 8>(g, sm_count, s);
    if (g.tree && g.m == 16) return run_select_rescore_residual<DSUB, 16>(g, sm_count, s);
    return run_select_rescore_residual<DSUB, 0>(g, sm_count, s);
}
}  // namespace

psb_status launch_select_rescore(const SelectRescoreLaunch& L, int nq, cudaStream_t s) {
    if (nq <= 0) return PSB_OK;
    RescoreArgs g;
    g.pool = L.pool; g.pool_cnt = L.pool_cnt; g.pool_cap = L.pool_cap; g.q_rows = L.q_rows; g.thr = L.thr; g.stage1_k = L.stage1_k; g.nq = nq;
    g.lut = L.lut; g.queries = L.queries; g.centroids = L.centroids; g.codebook = L.codebook; g.probes = L.probes;
    g.nprobe = L.nprobe; g.dim = L.dim; g.nlist = L.nlist; g.codes = L.codes; g.row_base = L.row_base; g.row_delta = L.row_delta;
    g.m = L.m; g.k = L.k; g.residual = L.residual ? 1 : 0; g.tree = L.tree ? 1 : 0;
    g.out_rows = L.out_rows; g.out_dist = L.out_dist; g.out_count = L.out_count; g.fail_list = L.fail_list; g.n_fail = L.n_fail;
    g.counters = L.counters; g.shared_cut = L.shared_cut ? 1 : 0; g.staged = 0;
    g.sort_n = 2;
    while (g.sort_n < L.stage1_k) g.sort_n <<= 1;
    if (g.residual) {
        switch (L.dim / L.m) {   // the sub-vector lengths the tensor-core scan takes
            case 2: PSB_TRY(run_select_rescore_tree<2>(g, L.sm_count, s)); break;
            case 4: PSB_TRY(run_select_rescore_tree<4>(g, L.sm_count, s)); break;
            case 8: PSB_TRY(run_select_rescore_tree<8>(g, L.sm_count, s)); break;
            default: return fail(PSB_UNSUPPORTED_SHAPE, "re-scoring selection does not support this shape");
        }
    } else {
        switch (L.m) {
            case 8: PSB_TRY(run_select_rescore<8>(g, s)); break;
            case 16: PSB_TRY(run_select_rescore<16>(g, s)); break;
            case 24: PSB_TRY(run_select_rescore<24>(g, s)); break;
            case 32: PSB_TRY(run_select_rescore<32>(g, s)); break;
            case 48: PSB_TRY(run_select_rescore<48>(g, s)); break;
            case 64: PSB_TRY(run_select_rescore<64>(g, s)); break;
            default: PSB_TRY(run_select_rescore<0>(g, s)); break;
        }
    }
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

}  // namespace psb
