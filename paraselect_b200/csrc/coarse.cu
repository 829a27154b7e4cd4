// Coarse stage, exact part: fp32 squared-L2 distances in the CPU path's arithmetic (sequential, non-fused:
// sum += (q-c)*(q-c), reference src/cpu/utils/cpu_distance.h:74-81) and per-row selection of the k smallest
// (distance, id) pairs.  The tensor-core filter in coarse_tc.cu narrows the centroid set first; what it keeps
// is scored by the kernels here, so results are bit-identical with or without it.
#include "common.cuh"
#include "dist_tile.cuh"
#include "kernels.h"
#include "select.cuh"

namespace psb {

using namespace tile;

namespace {

constexpr int BQ = 64, BC = 128, KC = 16, kDistThreads = 256;

// dist[q][c] for a BQ x BC tile; each thread owns 4 queries x 8 centroids.
__global__ void __launch_bounds__(kDistThreads)
k_coarse_dist_exact(const float* __restrict__ queries, int nq, const float* __restrict__ centroids, int nlist,
                    int dim, float* __restrict__ dist, unsigned long long* mark) {
    mark_start(mark);
    __shared__ __align__(16) float qs[KC][BQ];
    __shared__ __align__(16) float cs[KC][BC];
    const int q0 = blockIdx.y * BQ, c0 = blockIdx.x * BC;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    for (int d0 = 0; d0 < dim; d0 += KC) {
        for (int i = threadIdx.x; i < BQ * KC; i += kDistThreads) {
            const int row = i % BQ, d = i / BQ;
            qs[d][row] = (q0 + row < nq && d0 + d < dim) ? queries[(size_t)(q0 + row) * dim + d0 + d] : 0.0f;
        }
        for (int i = threadIdx.x; i < BC * KC; i += kDistThreads) {
            const int row = i % BC, d = i / BC;
            cs[d][row] = (c0 + row < nlist && d0 + d < dim) ? centroids[(size_t)(c0 + row) * dim + d0 + d] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int d = 0; d < KC; ++d) {
            const float4 qv = *reinterpret_cast<const float4*>(&qs[d][ty * 4]);
            const float4 ca = *reinterpret_cast<const float4*>(&cs[d][tx * 8]);
            const float4 cb = *reinterpret_cast<const float4*>(&cs[d][tx * 8 + 4]);
            const float qa[4] = {qv.x, qv.y, qv.z, qv.w};
            const float cc[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float diff = __fsub_rn(qa[i], cc[j]);
                    acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(diff, diff));
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int q = q0 + ty * 4 + i;
        if (q >= nq) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = c0 + tx * 8 + j;
            if (c < nlist) dist[(size_t)q * nlist + c] = acc[i][j];
        }
    }
}

// The same for batches whose BQ x BC tiles do not fill the chip: 32 queries x 64 centroids per CTA of 128 threads (4 x 4 each), all
// dimensions staged at once by 16-byte loads, one barrier.  A batch of 333 queries x 700 centroids x 100 dimensions is 36 of the large
// tiles, each a chain of load, barrier and compute steps (38 us); a single query against 1,024 centroids took 24 us the same way.
__global__ void __launch_bounds__(kSmallThreads)
k_coarse_dist_small(const float* __restrict__ queries, int nq, const float* __restrict__ centroids, int nlist, int dim, float* __restrict__ dist,
                    unsigned long long* mark) {
    behind();
    mark_start(mark);
    extern __shared__ __align__(16) float s_small[];
    const int pitch = small_pitch(dim);
    float* qs = s_small;                  // [SQ][pitch]
    float* cs = s_small + SQ * pitch;     // [SC][pitch]
    const int q0 = blockIdx.y * SQ, c0 = blockIdx.x * SC;
    stage_rows<kSmallThreads>(qs, pitch, queries + (size_t)q0 * dim, min(SQ, nq - q0), dim);
    stage_rows<kSmallThreads>(cs, pitch, centroids + (size_t)c0 * dim, min(SC, nlist - c0), dim);
    stage_wait();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    if (q0 + ty * 4 >= nq) return;
    float acc[4][4];
    tile_distances(qs + ty * 4 * pitch, cs + tx * pitch, pitch, dim, acc);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int q = q0 + ty * 4 + i;
        if (q >= nq) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = c0 + tx + 16 * j;
            if (c < nlist) dist[(size_t)q * nlist + c] = acc[i][j];
        }
    }
}

// The same for few pairs: a thread per centroid and query, the query in shared memory.  Of a tile most threads have no query, and the others
// have four centroids each, one after the other.  With the selection behind it, tiles against this, us: 1,024 centroids x 96, 1 query 15.2 / 11.3,
// 32 queries 17.2 / 14.3, 64 19.3 / 19.2, 128 19.1 / 25.3; 4,096, 8 queries 15.3 / 14.1, 16 16.3 / 17.2; 512 x 126, 64 queries 23.5 / 19.4; 256 x 96,
// 128 queries 19.2 / 15.3: the line lies at 32,768 pairs.
constexpr int kFewThreads = kCoarseFewBlock;
constexpr long long kFewPairs = 32768;
__global__ void __launch_bounds__(kFewThreads)
k_coarse_dist_few(const float* __restrict__ queries, const float* __restrict__ centroids, int nlist, int dim, float* __restrict__ dist,
                  unsigned long long* mark, float* __restrict__ copy) {
    extern __shared__ __align__(16) float s_q[];
    const int q = blockIdx.y, c = blockIdx.x * kFewThreads + threadIdx.x;
    behind();
    mark_start(mark);
    for (int d = threadIdx.x; d < dim; d += kFewThreads) {
        const float v = queries[(size_t)q * dim + d];
        s_q[d] = v;
        if (copy && blockIdx.x == 0) copy[(size_t)q * dim + d] = v;
    }
    __syncthreads();
    if (c < nlist) dist[(size_t)q * nlist + c] = row_distance(s_q, centroids + (size_t)c * dim, dim, rows_vec(centroids, dim));
}

// Nearest centroid of every row, without a matrix of distances: 64 rows a CTA, the centroids pass by in tiles of 64 (4 x 4 pairs a thread), the next
// tile on its way while one is compared; every thread keeps the nearest of its own centroids for its four rows.  The same distances; ties go to
// the lower id.  Bound: fp32 issue, three instructions per dimension and pair.  (Distances to memory and a selecting block per row: 70,338 x 96, 237
// centroids, two iterations of a training 5,688 us, now 1,071; 400,000 x 128, 64 centroids, five 14,450 and 6,030.)
// So few rows that CTAs of them leave SMs idle: the centroids are cut into ranges, a CTA each, and the smallest key of a row is taken in `keys` (a chain of
// all tiles took 272 us for 700 x 64, 3,000 centroids, where the distances to memory took 91; in ranges 34).
constexpr int kNearThreads = 256, kNearRows = 64;
inline size_t near_bytes(int dim) { return (size_t)(kNearRows + 2 * SC) * small_pitch(dim) * 4; }
__global__ void __launch_bounds__(kNearThreads)
k_nearest_rows(const float* __restrict__ rows, int n, const float* __restrict__ centroids, int k_all, int dim, int range, unsigned long long* __restrict__ keys,
               int* __restrict__ out_ids, float* __restrict__ out_dist) {
    extern __shared__ __align__(16) float s_near[];
    const int pitch = small_pitch(dim), tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float* rs = s_near;
    float* cs = s_near + kNearRows * pitch;   // [2][SC][pitch]
    const int r0 = blockIdx.x * kNearRows, first = blockIdx.y * range, k = min(range, k_all - first);   // of this CTA's centroids
    centroids += (size_t)first * dim;
    stage_rows<kNearThreads>(rs, pitch, rows + (size_t)r0 * dim, min(kNearRows, n - r0), dim);
    stage_rows<kNearThreads>(cs, pitch, centroids, min(SC, k), dim);
    asm volatile("cp.async.commit_group;" ::: "memory");
    float best[4];
    int id[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { best[i] = __int_as_float(0x7f800000); id[i] = -1; }
    for (int c0 = 0, t = 0; c0 < k; c0 += SC, t ^= 1) {
        if (c0 + SC < k) stage_rows<kNearThreads>(cs + (t ^ 1) * SC * pitch, pitch, centroids + (size_t)(c0 + SC) * dim, min(SC, k - c0 - SC), dim);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        float acc[4][4];
        tile_distances(rs + ty * 4 * pitch, cs + (t * SC + tx) * pitch, pitch, dim, acc);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = c0 + tx + 16 * j;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (acc[i][j] < best[i] && c < k) { best[i] = acc[i][j]; id[i] = c; }
        }
        __syncthreads();   // the tile may be written over
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint64_t key = id[i] >= 0 ? make_key(best[i], (uint32_t)(first + id[i])) : KEY_MAX;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) { const uint64_t other = __shfl_xor_sync(0xffffffffu, key, o); key = other < key ? other : key; }
        const int r = r0 + ty * 4 + i;
        if (r >= n) continue;   // (the same for the sixteen lanes of a row, which alone exchange)
        if (key == KEY_MAX && tx == 0) {   // no distance is a finite number: the smallest all the same, infinity before what is not a number
            for (int c = 0; c < k; ++c) {
                const uint64_t other = make_key(row_distance(rs + (ty * 4 + i) * pitch, centroids + (size_t)c * dim, dim, rows_vec(centroids, dim)), (uint32_t)(first + c));
                key = other < key ? other : key;
            }
        }
        if (tx != 0) continue;
        if (keys) atomicMin(keys + r, (unsigned long long)key);
        else { out_ids[r] = (int)key_idx(key); out_dist[r] = key_dist(key); }
    }
}

__global__ void __launch_bounds__(256) k_nearest_out(const unsigned long long* __restrict__ keys, int n, int* __restrict__ out_ids, float* __restrict__ out_dist) {
    const int r = blockIdx.x * 256 + threadIdx.x;
    if (r < n) { out_ids[r] = (int)key_idx(keys[r]); out_dist[r] = key_dist(keys[r]); }
}

// Per row: the k smallest (value, index) pairs, ascending.
constexpr int kSelThreads = 256;
__global__ void __launch_bounds__(kSelThreads)
k_select_rows(const float* __restrict__ dist, int n, int k, int buffer, int* __restrict__ out_ids, float* __restrict__ out_dist) {
    extern __shared__ __align__(16) uint64_t s_sel[];  // [buffer] keys, then the selection's runs
    __shared__ sel::Words w;
    behind();
    const int keep = sel::smallest<kSelThreads>(dist + (size_t)blockIdx.x * n, n, k, [](int i) { return (uint32_t)i; }, s_sel, buffer,
                                   reinterpret_cast<int*>(s_sel + buffer), &w);
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        const bool ok = i < keep;
        out_ids[(size_t)blockIdx.x * k + i] = ok ? (int)key_idx(s_sel[i]) : -1;
        if (out_dist) out_dist[(size_t)blockIdx.x * k + i] = ok ? key_dist(s_sel[i]) : FLT_MAX;
    }
}

}  // namespace

bool coarse_few(int nq, int nlist, int dim) { return (long long)nq * nlist <= kFewPairs && nq <= 65535 && (size_t)dim * sizeof(float) <= (size_t)200 * 1024; }

psb_status launch_coarse_dist_exact(const float* d_queries, int nq, const float* d_centroids, int nlist,
                                    int dim, float* d_dist, int sm_count, cudaStream_t s, unsigned long long* mark, float* d_copy) {
    if (nq <= 0) return PSB_OK;
    if (d_copy && !coarse_few(nq, nlist, dim)) return fail(PSB_INTERNAL, "host queries are for few pairs");
    const size_t smem = (size_t)((dim + 3) & ~3) * sizeof(float);
    if (coarse_few(nq, nlist, dim)) {
        if (smem > 48 * 1024) PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_coarse_dist_few), smem));
        k_coarse_dist_few<<<dim3((unsigned)((nlist + kFewThreads - 1) / kFewThreads), (unsigned)nq), kFewThreads, smem, s>>>(d_queries, d_centroids, nlist, dim, d_dist, mark,
                                                                                                                                  d_copy);
        count_launch();
        PSB_LAUNCH_CHECK();
        return PSB_OK;
    }
    dim3 grid((nlist + BC - 1) / BC, (nq + BQ - 1) / BQ);
    // Small tiles while the large ones would leave SMs without one (two waves of small tiles still beat one of large ones), if
    // their rows fit.
    const size_t small = small_tile_bytes(dim);
    if ((long long)grid.x * grid.y < sm_count && small <= (size_t)200 * 1024) {
        const dim3 g2((nlist + SC - 1) / SC, (nq + SQ - 1) / SQ);
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_coarse_dist_small), small));
        k_coarse_dist_small<<<g2, kSmallThreads, small, s>>>(d_queries, nq, d_centroids, nlist, dim, d_dist, mark);
        count_launch();
        PSB_LAUNCH_CHECK();
        return PSB_OK;
    }
    k_coarse_dist_exact<<<grid, kDistThreads, 0, s>>>(d_queries, nq, d_centroids, nlist, dim, d_dist, mark);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

bool nearest_rows_fit(int dim) { return near_bytes(dim) <= (size_t)200 * 1024; }
// Whether it beats distances to memory and a selection.  Not for few rows and pairs (700 x 128 to 100 centroids, three iterations, 223 us, distances to memory 196), nor for long
// rows, which leave an SM one CTA, and many centroids (20,000 x 200, trainings of three iterations, ms: 600 centroids 2.06, distances to memory 1.96, 3,000 8.3 and 7.0).
bool nearest_rows_pays(int n, int k, int dim) { return nearest_rows_fit(dim) && (n >= 1024 || (long long)n * k >= 98304) && (dim <= 128 || k < 512 || n < 2048); }

// Cut until there are two CTAs an SM; two tiles of short rows are not worth the keys' passes.
int nearest_rows_range(int n, int k, int dim, int sm_count) {
    const int tiles = (k + SC - 1) / SC, blocks = (n + kNearRows - 1) / kNearRows;
    if (tiles < (dim >= 96 ? 2 : 3) || blocks >= 2 * sm_count) return k;
    const int parts = std::min(tiles, (2 * sm_count + blocks - 1) / blocks), each = (tiles + parts - 1) / parts;
    return each < tiles ? each * SC : k;
}

psb_status launch_nearest_rows(const float* d_rows, int n, const float* d_centroids, int k, int dim, int range, unsigned long long* d_keys, int* d_ids, float* d_dist,
                               cudaStream_t s) {
    if (n <= 0) return PSB_OK;
    if (range < k) PSB_CUDA(cudaMemsetAsync(d_keys, 0xff, sizeof(unsigned long long) * (size_t)n, s));   // KEY_MAX
    const size_t smem = near_bytes(dim);
    PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_nearest_rows), smem));
    k_nearest_rows<<<dim3((unsigned)((n + kNearRows - 1) / kNearRows), (unsigned)((k + range - 1) / range)), kNearThreads, smem, s>>>(
        d_rows, n, d_centroids, k, dim, range, range < k ? d_keys : nullptr, d_ids, d_dist);
    count_launch();
    PSB_LAUNCH_CHECK();
    if (range < k) {
        k_nearest_out<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_keys, n, d_ids, d_dist);
        count_launch();
        PSB_LAUNCH_CHECK();
    }
    return PSB_OK;
}

psb_status launch_select_rows(const float* d_dist, int nq, int n, int k, int* d_ids, float* d_out, cudaStream_t s) {
    if (nq <= 0) return PSB_OK;
    if (k <= 0 || k > kMaxProbe) return fail(PSB_UNSUPPORTED_SHAPE, "row selection supports 1..4096 results");
    const size_t smem = sel::shared_bytes(k);
    PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_select_rows), smem));
    PSB_TRY(launch_behind(select_behind(nq, (long long)nq * n <= 8192 ? nq : 2, k, 32), k_select_rows, dim3((unsigned)nq), kSelThreads, smem, s, d_dist, n, k, sel::buffer_entries(k), d_ids, d_out));
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

}  // namespace psb

// ---- coarse search without any allocation ---------------------------------------------------------------
// Some callers may not allocate device memory at the moment they need a coarse search: a serving thread that
// holds a fixed memory budget granted at start-up, code that runs under a memory pool it must not touch, or a
// plugin host that forbids cudaMalloc after initialisation because an allocation synchronises the device and
// can fail late.  For them the distance tile [nq][nlist] lives in the array below, which every GPU that loads
// this library holds until the process exits.
namespace psb {
namespace {
constexpr size_t kStaticCoarseFloats = (size_t)4 << 20;  // 4 Mi distances = 16 MiB: nq * nlist must not exceed it
static __device__ __align__(256) float g_coarse_scratch[kStaticCoarseFloats];
constexpr int kMaxDevices = 64;
float* g_scratch_ptr[kMaxDevices] = {};  // per device: the array's DEVICE address (the symbol itself is a host stand-in)
}  // namespace
}  // namespace psb

extern "C" psb_status psb_coarse_search_static(const float* d_queries, int nq, const float* d_centroids, int nlist,
                                               int dim, int nprobe, int* d_ids, float* d_dist, void* stream) {
    using namespace psb;
    if (!d_queries || !d_centroids || !d_ids || nq < 0 || nlist <= 0 || dim <= 0)
        return fail(PSB_INVALID_ARGUMENT, "invalid coarse request");
    if (nprobe <= 0 || nprobe > nlist) return fail(PSB_INVALID_ARGUMENT, "nprobe must be in 1..nlist");
    if (nprobe > kMaxProbe) return fail(PSB_UNSUPPORTED_SHAPE, "nprobe above 4096 is not supported");
    if ((size_t)nq * (size_t)nlist > kStaticCoarseFloats)
        return fail(PSB_UNSUPPORTED_SHAPE,
                    "psb_coarse_search_static: nq * nlist exceeds the 4,194,304 distances of the built-in scratch; "
                    "split the query batch or use psb_stage_coarse");
    if (nq == 0) return PSB_OK;
    int device = -1;
    PSB_CUDA(cudaGetDevice(&device));
    if (device < 0 || device >= kMaxDevices) return fail(PSB_UNSUPPORTED_SHAPE, "device ordinal above 63");
    if (!g_scratch_ptr[device]) {
        // First call on this device: resolve the array's device address (this device is current).
        float* p = nullptr;
        PSB_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_coarse_scratch));
        g_scratch_ptr[device] = p;
    }
    float* tile = g_scratch_ptr[device];
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int sms = 0;
    PSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    PSB_TRY(launch_coarse_dist_exact(d_queries, nq, d_centroids, nlist, dim, tile, sms, st));
    return launch_select_rows(tile, nq, nlist, nprobe, d_ids, d_dist, st);
}
