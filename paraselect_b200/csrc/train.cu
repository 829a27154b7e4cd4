// Training and encoding kernels: PQ encode (the shapes pq_nearest.cu does not take), PQ codebook seeding and Lloyd updates,
// k-means accumulation / update, and the counter-based synthetic data generators used by the bench.
//
// Semantics follow the reference trainers: assignment = argmin of squared L2 with strict '<' so the lowest
// index wins ties (src/clustering/kmeans/kmeans_utils.cu:359-413, src/quantization/pq/pq_encode.cuh:24-40),
// update = mean of members, empty cluster keeps its centroid (src/clustering/kmeans/kmeans_utils.cu:267-284).
// Member sums are accumulated in fp64 so the result does not depend on the summation order.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace psb {
namespace {

constexpr int kEncThreads = 256;

// One CTA encodes kEncThreads rows for every sub-quantiser; codes are staged in shared memory and written
// out as whole rows.
__global__ void __launch_bounds__(kEncThreads)
k_pq_encode(const float* __restrict__ data, long long n, int dim, const float* __restrict__ codebook, int m, int k,
            uint8_t* __restrict__ codes) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int dsub = dim / m;
    float* s_cb = reinterpret_cast<float*>(s_raw);                            // [k * dsub]
    uint8_t* s_codes = s_raw + (size_t)k * dsub * sizeof(float);              // [kEncThreads * m]
    const long long row = (long long)blockIdx.x * kEncThreads + threadIdx.x;
    for (int sub = 0; sub < m; ++sub) {
        __syncthreads();
        for (int i = threadIdx.x; i < k * dsub; i += kEncThreads) s_cb[i] = codebook[(size_t)sub * k * dsub + i];
        __syncthreads();
        if (row < n) {
            const float* x = data + (size_t)row * dim + (size_t)sub * dsub;
            float best = FLT_MAX; int bc = 0;
            for (int c = 0; c < k; ++c) {
                float dist = 0.0f;
                for (int d = 0; d < dsub; ++d) {
                    const float diff = __fsub_rn(__ldg(x + d), s_cb[c * dsub + d]);
                    dist = __fadd_rn(dist, __fmul_rn(diff, diff));
                }
                if (dist < best) { best = dist; bc = c; }
            }
            s_codes[threadIdx.x * m + sub] = (uint8_t)bc;
        }
    }
    __syncthreads();
    const long long row0 = (long long)blockIdx.x * kEncThreads;
    const long long rows_here = min((long long)kEncThreads, n - row0);
    for (long long i = threadIdx.x; i < rows_here * m; i += kEncThreads) codes[(size_t)row0 * m + i] = s_codes[i];
}

// Same result, rows staged in shared memory: the CTA's rows are read once with coalesced loads into a tile padded to
// dim + 1 floats per row (conflict-free when every thread reads its own row), and every thread walks the codewords with its
// own sub-vectors (broadcast reads of the codewords).
__global__ void __launch_bounds__(kEncThreads)
k_pq_encode_tile(const float* __restrict__ data, long long n, int dim, const float* __restrict__ codebook, int m, int k,
                 uint8_t* __restrict__ codes) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int dsub = dim / m;
    const int pitch = dim + 1;
    float* s_x = reinterpret_cast<float*>(s_raw);                                            // [kEncThreads][pitch]
    float* s_cb = s_x + (size_t)kEncThreads * pitch;                                         // [k * dsub]
    uint8_t* s_codes = reinterpret_cast<uint8_t*>(s_cb + (size_t)k * dsub);                  // [kEncThreads * m]
    const long long row0 = (long long)blockIdx.x * kEncThreads;
    const long long rows_here = min((long long)kEncThreads, n - row0);
    for (long long i = threadIdx.x; i < rows_here * dim; i += kEncThreads) {
        const int r = (int)(i / dim), d = (int)(i % dim);
        s_x[(size_t)r * pitch + d] = data[(size_t)row0 * dim + i];
    }
    const bool live = threadIdx.x < rows_here;
    const float* xs = s_x + (size_t)threadIdx.x * pitch;
    for (int sub = 0; sub < m; ++sub) {
        __syncthreads();
        for (int i = threadIdx.x; i < k * dsub; i += kEncThreads) s_cb[i] = codebook[(size_t)sub * k * dsub + i];
        __syncthreads();
        if (live) {
            float best = FLT_MAX; int bc = 0;
            for (int c = 0; c < k; ++c) {
                float dist = 0.0f;
                for (int d = 0; d < dsub; ++d) {
                    const float diff = __fsub_rn(xs[sub * dsub + d], s_cb[c * dsub + d]);
                    dist = __fadd_rn(dist, __fmul_rn(diff, diff));
                }
                if (dist < best) { best = dist; bc = c; }
            }
            s_codes[threadIdx.x * m + sub] = (uint8_t)bc;
        }
    }
    __syncthreads();
    for (long long i = threadIdx.x; i < rows_here * m; i += kEncThreads) codes[(size_t)row0 * m + i] = s_codes[i];
}

// ---- k-means++ seeding of the PQ codebooks, all sub-quantisers at once ------------------------------------------------------
// The reference's initialisation picks codeword after codeword: the running fp64 sum of the rows' squared distances to the nearest
// codeword so far, a draw r in [0, sum), and the first row at which the running sum reaches r.  On one host thread this took 0.5 s
// for 32,768 rows x 24 sub-quantisers, 98 % of a codebook training.  Here a cluster of eight CTAs holds a sub-quantiser's rows and
// their distances in shared memory (rows that do not fit are read through L2); a pick is one update of the distances, two cluster
// barriers and a search in one warp's stretch of rows, of which a lane takes eight at a time (kSeedShort: one); the warp that finds the row
// hands it round with its values: 4.3 us (32,768 rows, 24 sub-quantisers; 5.6 with values from global memory, rows read word by word and a
// stretch walked 32 rows a step), 255 picks, every sub-quantiser on SMs of its own.
// The draws are made by the host (they do not depend on the data).  The rows picked are the reference's: its sequential sum and the
// tree sum used here each stay within (n + 64) 2^-53 of the exact one, so when r is further than three times that from the
// borders of the row found, the sequential search finds the same row; when it is not (about one draw in a million), one thread
// repeats the search sequentially.  A sum that is not a positive finite number is left to the host's own initialisation (status).
constexpr int kSeedCluster = 8, kSeedCtaThreads = 512, kSeedCtaWarps = kSeedCtaThreads / 32;
// Rows of a warp's stretch up to which the search takes a row a lane, in a kernel of its own: a lane's eight rows are two chains of sums, and the warps of a
// round share an instruction cache that it finds cold.  Eight / one, us, four sub-quantisers of 4: 2,000 rows 710 / 626, 4,096 747 / 657, 8,192
// (stretches of 64) 785 / 733, 16,384 (128) 832 / 843.  Both searches in one kernel: 646, 673, 745.
constexpr int kSeedShort = 64;

__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t a, double v) { asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }
__device__ __forceinline__ void cluster_store(uint32_t a, int v) { asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void cluster_store(uint32_t a, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ float cluster_load(uint32_t a) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double warp_inclusive(double v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += up;
    }
    return v;
}

// draws [m][k - 1] uniform in [0, 1); first [m]; rows_out [m][k]; status [m] = 1: left to the host.  per = rows per CTA.
template <int D, bool SHORT>
__global__ void __launch_bounds__(kSeedCtaThreads) __cluster_dims__(kSeedCluster, 1, 1)
k_pq_seed(const float* __restrict__ data, int n, int dim, int dsub_rt, int k, int per, int staged, const double* __restrict__ draws,
          const int* __restrict__ first, long long* __restrict__ rows_out, int* __restrict__ status) {
    extern __shared__ __align__(16) float s_seed[];
    const int dsub = D > 0 ? D : dsub_rt;
    float* s_min = s_seed;                                  // [per] distance of each row to its nearest codeword so far
    float* s_rows = s_seed + (per + 511) / 256 * 256;       // [per][dsub] when staged; the search reads up to 255 places past a stretch's end
    __shared__ double s_sum[kSeedCluster * kSeedCtaWarps];  // every warp's sum, of all eight CTAs
    __shared__ int s_pick;
    __shared__ float s_cen[D > 0 ? D : 1];
    const int sub = blockIdx.y, rank = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = min(n, rank * per), cnt = min(n, b + per) - b;
    const int wper = ((per + kSeedCtaWarps - 1) / kSeedCtaWarps + 31) / 32 * 32;   // a warp's stretch of rows: begins on a vector
    const int w0 = min(cnt, warp * wper), w1 = min(cnt, w0 + wper);
    const float* src = data + (size_t)sub * dsub;
    if (staged)
        for (int i = tid; i < cnt * dsub; i += kSeedCtaThreads) { const int r = i / dsub; s_rows[i] = src[(size_t)(b + r) * dim + (i - r * dsub)]; }
    long long* out = rows_out + (size_t)sub * k;
    const int keff = min(k, n);
    int pick = first[sub];
    if (rank == 0 && tid == 0) out[0] = pick;
    __syncthreads();
    // A row's values: whole vectors where rows lie on their boundaries (staged ones of 2, 4, 6, 8 dimensions).
    auto row_of = [&](int r, float (&x)[D > 0 ? D : 1]) {
        if constexpr (D > 0) {
            if (!staged) {
#pragma unroll
                for (int d = 0; d < D; ++d) x[d] = __ldg(src + (size_t)(b + r) * dim + d);
            } else if constexpr (D % 4 == 0) {
#pragma unroll
                for (int d = 0; d < D; d += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(s_rows + (size_t)r * D + d);
                    x[d] = v.x; x[d + 1] = v.y; x[d + 2] = v.z; x[d + 3] = v.w;
                }
            } else if constexpr (D % 2 == 0) {
#pragma unroll
                for (int d = 0; d < D; d += 2) { const float2 v = *reinterpret_cast<const float2*>(s_rows + (size_t)r * D + d); x[d] = v.x; x[d + 1] = v.y; }
            } else {
#pragma unroll
                for (int d = 0; d < D; ++d) x[d] = s_rows[(size_t)r * D + d];
            }
        }
    };
    float cv[D > 0 ? D : 1];
    if constexpr (D > 0) {
#pragma unroll
        for (int d = 0; d < D; ++d) cv[d] = __ldg(src + (size_t)pick * dim + d);
    }
    for (int c = 1; c < keff; ++c) {
        const float* cen = src + (size_t)pick * dim;
        double sum = 0.0;
        for (int r = w0 + lane; r < w1; r += 32) {
            float acc = 0.0f;
            if constexpr (D > 0) {
                float x[D];
                row_of(r, x);
#pragma unroll
                for (int d = 0; d < D; ++d) { const float diff = __fsub_rn(x[d], cv[d]); acc = __fadd_rn(acc, __fmul_rn(diff, diff)); }
            } else {
                const float* x = staged ? s_rows + (size_t)r * dsub : src + (size_t)(b + r) * dim;
                for (int d = 0; d < dsub; ++d) { const float diff = __fsub_rn(x[d], __ldg(cen + d)); acc = __fadd_rn(acc, __fmul_rn(diff, diff)); }
            }
            float m = c == 1 ? acc : s_min[r];
            if (acc < m) m = acc;
            s_min[r] = m;
            sum += (double)m;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane < kSeedCluster) cluster_store(cluster_addr(&s_sum[rank * kSeedCtaWarps + warp], lane), sum);
        cluster_sync();
        // the stretch the draw falls into, found by every warp on its own: four consecutive sums per lane
        const double v0 = s_sum[4 * lane], v1 = s_sum[4 * lane + 1], v2 = s_sum[4 * lane + 2], v3 = s_sum[4 * lane + 3];
        const double incl = warp_inclusive(v0 + v1 + v2 + v3, lane);
        const double total = __shfl_sync(0xffffffffu, incl, 31);
        if (!(total > 0.0) || isinf(total)) {   // uniform over the cluster; also when not a number
            if (rank == 0 && tid == 0) status[sub] = 1;
            return;
        }
        const double r = __dmul_rn(draws[(size_t)sub * (k - 1) + (c - 1)], total);
        const double slack = 3.0 * (double)(n + 64) * 1.1102230246251565e-16 * total;
        const unsigned bal = __ballot_sync(0xffffffffu, incl >= r);
        const int gl = bal ? __ffs((int)bal) - 1 : 31;
        double before = __shfl_sync(0xffffffffu, incl - (v0 + v1 + v2 + v3), gl);
        int chunk = 4 * gl;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double next = before + s_sum[chunk];
            if (next < r && chunk < 4 * gl + 3) { before = next; ++chunk; }
        }
        if (chunk / kSeedCtaWarps == rank && chunk % kSeedCtaWarps == warp) {
            int found = -1;
            bool sure = false;
            double run = before;
            if constexpr (SHORT) {   // a row a lane
                for (int r0 = w0; r0 < w1; r0 += 32) {
                    const int row = r0 + lane;
                    const double in = warp_inclusive(row < w1 ? (double)s_min[row] : 0.0, lane) + run;
                    const unsigned hit = __ballot_sync(0xffffffffu, row < w1 && in >= r);
                    if (hit) {
                        const int l = __ffs((int)hit) - 1;
                        const double hi = __shfl_sync(0xffffffffu, in, l), lo = __shfl_sync(0xffffffffu, in, l ? l - 1 : 0), below = l ? lo : run;
                        found = b + r0 + l;
                        sure = hi - r > slack && (r - below > slack || found == 0);
                        break;
                    }
                    run = __shfl_sync(0xffffffffu, in, 31);
                }
            } else for (int r0 = w0; r0 < w1; r0 += 256) {   // eight rows a lane
                const int row = r0 + lane * 8;
                double x[8], mine = 0.0;
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(s_min + row + i);   // (the last stretch may reach past the rows: into what lies behind them)
                    x[i] = v.x; x[i + 1] = v.y; x[i + 2] = v.z; x[i + 3] = v.w;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) { if (row + i >= w1) x[i] = 0.0; mine += x[i]; }
                const double in = warp_inclusive(mine, lane) + run;
                const unsigned hit = __ballot_sync(0xffffffffu, row < w1 && in >= r);
                if (hit) {
                    const int l = __ffs((int)hit) - 1;
                    const double upto = __shfl_up_sync(0xffffffffu, in, 1);
                    if (lane == l) {   // one of this lane's rows
                        double below = lane ? upto : run, hi = below;
                        int i = 0;
                        bool there = false;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            if (there) continue;
                            const double next = below + x[j];
                            if (next < r && j < 7 && row + j + 1 < w1) { below = next; i = j + 1; }
                            else { hi = next; there = true; }
                        }
                        found = b + row + i;
                        sure = hi - r > slack && (r - below > slack || found == 0);
                    }
                    found = __shfl_sync(0xffffffffu, found, l);
                    sure = __shfl_sync(0xffffffffu, sure ? 1 : 0, l) != 0;
                    break;
                }
                run = __shfl_sync(0xffffffffu, in, 31);
            }
            if (!sure) {   // too close to a border, or beyond the stretch: the sequential sums decide
                if (lane == 0) {
                    double t = 0.0;
#pragma unroll 1
                    for (int i = 0; i < n; ++i) t += (double)cluster_load(cluster_addr(&s_min[i % per], i / per));
                    const double rs = __dmul_rn(draws[(size_t)sub * (k - 1) + (c - 1)], t);
                    double cum = 0.0;
                    found = n - 1;
#pragma unroll 1
                    for (int i = 0; i < n; ++i) {
                        cum += (double)cluster_load(cluster_addr(&s_min[i % per], i / per));
                        if (cum >= rs) { found = i; break; }
                    }
                }
                found = __shfl_sync(0xffffffffu, found, 0);
            }
            if (lane < kSeedCluster) {
                cluster_store(cluster_addr(&s_pick, lane), found);
                if constexpr (D > 0) {
                    float x[D];   // (the sequential search may have found a row of another CTA)
                    if (found >= b && found < b + cnt) row_of(found - b, x);
                    else {
#pragma unroll
                        for (int d = 0; d < D; ++d) x[d] = __ldg(src + (size_t)found * dim + d);
                    }
#pragma unroll
                    for (int d = 0; d < D; ++d) cluster_store(cluster_addr(&s_cen[d], lane), x[d]);
                }
            }
            if (lane == 0) out[c] = found;
        }
        cluster_sync();
        pick = s_pick;
        if constexpr (D > 0) {
#pragma unroll
            for (int d = 0; d < D; ++d) cv[d] = s_cen[d];
        }
    }
    for (int c = keff + tid; rank == 0 && c < k; c += kSeedCtaThreads) out[c] = first[sub];
}

// Codeword sums: a CTA takes one sub-quantiser's codes of a range of rows, orders the rows by codeword in shared memory (counts,
// prefix, slots) and lets a warp sum each codeword's rows in fp64, so that only one fp64 atomic per non-empty codeword and
// dimension leaves it.  A lane keeps one dimension: P lanes read a row's sub-vector side by side, 32 / P rows at a time, and two to four
// exchanges end it.  (A row per lane took five exchanges for each dimension: 44 us for 32,768 x 96, m = 24, 19 now; fp64 atomics in shared
// memory per element 459.)
constexpr int kPqAccRows = 4096, kPqAccThreads = 1024;   // threads: each warp's codewords follow one another, a list and a row's latency each
__global__ void __launch_bounds__(kPqAccThreads) k_pq_accumulate(const float* __restrict__ data, long long n, int dim, const uint8_t* __restrict__ codes,
                                                       int m, int k, double* __restrict__ sums, int* __restrict__ counts) {
    __shared__ int s_off[257], s_cur[256], s_warp[32], s_total;
    __shared__ uint16_t s_row[kPqAccRows];
    const int dsub = dim / m, sub = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long r0 = (long long)blockIdx.x * kPqAccRows;
    const int rows = (int)min((long long)kPqAccRows, n - r0);
    __shared__ uint8_t s_code[kPqAccRows];
    if (threadIdx.x < 256) s_cur[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int i = threadIdx.x; i < rows; i += kPqAccThreads) {
        const uint8_t c = __ldg(codes + (size_t)(r0 + i) * m + sub);
        s_code[i] = c;
        atomicAdd(&s_cur[c], 1);
    }
    __syncthreads();
    const int mine = threadIdx.x < 256 ? s_cur[threadIdx.x] : 0;
    const int ex = block_exclusive_scan(mine, s_warp, &s_total);
    if (threadIdx.x < 256) { s_off[threadIdx.x] = ex; s_cur[threadIdx.x] = ex; }
    if (threadIdx.x == 0) s_off[256] = rows;
    if (mine) atomicAdd(&counts[(size_t)sub * k + threadIdx.x], mine);
    __syncthreads();
    for (int i = threadIdx.x; i < rows; i += kPqAccThreads) s_row[atomicAdd(&s_cur[s_code[i]], 1)] = (uint16_t)i;   // (its own codes: no barrier needed)
    __syncthreads();
    const float* src = data + (size_t)r0 * dim + (size_t)sub * dsub;
    int p = 1;   // lanes of a row
    while (p < dsub && p < 32) p <<= 1;
    const int at = lane & (p - 1), first = lane / p, step = 32 / p;
    for (int c = warp; c < k; c += kPqAccThreads / 32) {
        const int b = s_off[c], e = s_off[c + 1];
        if (b == e) continue;
        for (int d0 = 0; d0 < dsub; d0 += p) {
            const int d = d0 + at;
            double acc = 0.0;
            if (d < dsub) {
#pragma unroll 4
                for (int i = b + first; i < e; i += step) acc += (double)__ldg(src + (size_t)s_row[i] * dim + d);
            }
            for (int o = p; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane < p && d < dsub) atomicAdd(&sums[((size_t)sub * k + c) * dsub + d], acc);
        }
    }
}

// Codewords from their sums; the sums and counts are left zeroed for the next iteration.
__global__ void k_pq_update(double* __restrict__ sums, int* __restrict__ counts, int codewords, int dsub, float* __restrict__ codebook) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= codewords) return;
    const int c = counts[i];
    counts[i] = 0;
    for (int d = 0; d < dsub; ++d) {
        const double s = sums[(size_t)i * dsub + d];
        sums[(size_t)i * dsub + d] = 0.0;
        if (c > 0) codebook[(size_t)i * dsub + d] = (float)(s / (double)c);
    }
}

__global__ void k_mean_update(const double* __restrict__ sums, const int* __restrict__ counts, long long n_centres,
                              int width, float* __restrict__ centres) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_centres * width) return;
    const int c = counts[i / width];
    if (c > 0) centres[i] = (float)(sums[i] / (double)c);
}

// out[row] = data[row] - centroids[assign[row]] (fp32 subtraction): what residual-mode PQ is trained on and encodes.
__global__ void k_residual_rows(const float* __restrict__ data, long long n, int dim, const float* __restrict__ centroids,
                                const int* __restrict__ assign, float* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * dim) return;
    const long long row = i / dim;
    const int d = (int)(i - row * dim);
    out[i] = __fsub_rn(data[i], __ldg(centroids + (size_t)assign[row] * dim + d));
}

__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// ---- k-means accumulation: rows grouped by centroid, then one CTA sums each group --------------------------------------
// (the reference sorts by assignment and accumulates segment by segment for the same reason: src/clustering/kmeans/
// kmeans.cu:519-575, kmeans_utils.cu:541-574; per-element atomics onto k * dim fp64 words serialise on popular centroids).
// 1. k_km_count:   counts[c] (one int atomic per row) and the objective (one fp64 atomic per CTA)
// 2. k_km_offsets: exclusive prefix of the counts, one CTA in coalesced rounds
// 3. k_km_fill:    order[offset[c] + slot] = row (one int atomic per row)
// 4. k_km_sums:    CTA c sums its rows in fp64, two threads per dimension (eight where groups are large), and writes sums[c][:]; a group of more than 1,024 rows (the
//                  nearest of a crowd without a centroid of its own) is cut over kKmSplit CTAs that add atomically, or it alone
//                  takes most of the pass.  The rows of a group of at most 1,024 are put in order first (each finds its rank among the others: one barrier where a bitonic sort of
//                  64 rows has 21), so that the sum does not depend on the order the slots were taken
constexpr int kKmSplit = 8;
// Of the four kernels below each passes over a row whose assignment is no centroid (a row that is not a number has no nearest one).
__global__ void k_km_count(const int* __restrict__ assign, const float* __restrict__ best, long long n, int k, int* __restrict__ counts,
                           double* __restrict__ obj) {
    __shared__ double s_part[8];
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double b = 0.0;
    if (i < n) {
        const int c = assign[i];
        if ((unsigned)c < (unsigned)k) atomicAdd(&counts[c], 1);
        if (best) b = (double)best[i];
    }
    if (!obj) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_part[w];
        atomicAdd(obj, t);
    }
}
__global__ void __launch_bounds__(1024) k_km_offsets(const int* __restrict__ counts, int k, int* __restrict__ offsets, int* __restrict__ cursor) {
    __shared__ int s_warp[32];
    __shared__ int s_total;
    int carry = 0;
    for (int base = 0; base < k; base += blockDim.x) {
        const int c = base + threadIdx.x;
        const int v = c < k ? counts[c] : 0;
        const int ex = block_exclusive_scan(v, s_warp, &s_total);
        if (c < k) { offsets[c] = carry + ex; cursor[c] = 0; }
        carry += s_total;
        __syncthreads();
    }
    if (threadIdx.x == 0) offsets[k] = carry;
}
__global__ void k_km_fill(const int* __restrict__ assign, long long n, int k, const int* __restrict__ offsets, int* __restrict__ cursor,
                          int* __restrict__ order) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = assign[i];
    if ((unsigned)c >= (unsigned)k) return;
    order[offsets[c] + atomicAdd(&cursor[c], 1)] = (int)i;
}
// The same two for few centroids, whose counters all rows would queue at: a block counts its kFewRows rows in shared memory first, and takes the
// places of each centroid's with one atomic (400,000 rows, 64
// centroids, five iterations: 4.7 -> 3.3 ms).  A block's own part, which it does whatever the rows, costs 2 to 3 us more in all, so that there have to be rows enough
// and rows enough a centroid.  Whole accumulation of 64 dimensions, us, rows by themselves / by blocks: 512 centroids, 20 rows each 33.0 / 36.2, 32 37.4 / 37.0, 96
// 49.0 / 40.6; 1,024, 16 35.9 / 39.3, 32 40.4 / 39.7; 2,048, 16 46.2 / 46.9, 32 50.1 / 50.1, 48 54.8 / 51.9; 256, 32 32.6 / 36.1, 64 37.8 / 38.3, 160 53.3 / 44.7; 64, 96
// 35.8 / 38.1, 400 50.6 / 41.8.
constexpr int kFewCentroids = 2048, kFewRows = 4096;
constexpr long long kFewPerCentroid = 32, kFewLeast = 16384;
__global__ void __launch_bounds__(1024) k_km_count_few(const int* __restrict__ assign, const float* __restrict__ best, long long n, int k, int* __restrict__ counts,
                                                       double* __restrict__ obj) {
    __shared__ int s_count[kFewCentroids];
    __shared__ double s_part[32];
    for (int c = threadIdx.x; c < k; c += 1024) s_count[c] = 0;
    __syncthreads();
    double b = 0.0;
#pragma unroll
    for (int t = 0; t < kFewRows / 1024; ++t) {
        const long long i = (long long)blockIdx.x * kFewRows + t * 1024 + threadIdx.x;
        if (i < n) {
            const int c = assign[i];
            if ((unsigned)c < (unsigned)k) atomicAdd(&s_count[c], 1);
            if (best) b += (double)best[i];
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < k; c += 1024) if (s_count[c]) atomicAdd(&counts[c], s_count[c]);
    if (!obj) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 32; ++w) t += s_part[w];
        atomicAdd(obj, t);
    }
}
__global__ void __launch_bounds__(1024) k_km_fill_few(const int* __restrict__ assign, long long n, int k, const int* __restrict__ offsets, int* __restrict__ cursor,
                                                      int* __restrict__ order) {
    __shared__ int s_count[kFewCentroids], s_first[kFewCentroids];
    for (int c = threadIdx.x; c < k; c += 1024) s_count[c] = 0;
    __syncthreads();
    int own[kFewRows / 1024], slot[kFewRows / 1024];
#pragma unroll
    for (int t = 0; t < kFewRows / 1024; ++t) {
        const long long i = (long long)blockIdx.x * kFewRows + t * 1024 + threadIdx.x;
        own[t] = i < n ? assign[i] : -1;
        if (own[t] >= k) own[t] = -1;
        slot[t] = own[t] >= 0 ? atomicAdd(&s_count[own[t]], 1) : 0;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < k; c += 1024) if (s_count[c]) s_first[c] = offsets[c] + atomicAdd(&cursor[c], s_count[c]);
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kFewRows / 1024; ++t)
        if (own[t] >= 0) order[s_first[own[t]] + slot[t]] = (int)((long long)blockIdx.x * kFewRows + t * 1024 + threadIdx.x);
}
template <int T>
__global__ void __launch_bounds__(T) k_km_sums(const float* __restrict__ data, int dim, const int* __restrict__ offsets,
                                                           const int* __restrict__ order, double* __restrict__ sums) {
    __shared__ int s_in[1024], s_rows[1024];
    constexpr int kDims = 128, PARTS = T / kDims;   // threads of a dimension
    __shared__ double s_part[PARTS - 1][kDims];
    const int c = blockIdx.x;
    int b0 = offsets[c], cnt = offsets[c + 1] - b0;
    const bool split = cnt > 1024;
    if (split) {
        const int b = (int)((long long)cnt * blockIdx.y / kKmSplit), e = (int)((long long)cnt * (blockIdx.y + 1) / kKmSplit);
        b0 += b; cnt = e - b;
    } else if (blockIdx.y) {
        return;
    }
    const int* rows = order + b0;
    if (!split && cnt > 1) {   // canonical order for the usual, small group
        for (int i = threadIdx.x; i < cnt; i += T) s_in[i] = rows[i];
        __syncthreads();
        for (int i = threadIdx.x; i < cnt; i += T) {
            const int mine = s_in[i];
            int rank = 0;
            for (int j = 0; j < cnt; ++j) rank += s_in[j] < mine ? 1 : 0;
            s_rows[rank] = mine;
        }
        __syncthreads();
        rows = s_rows;
    }
    const int part = threadIdx.x / kDims, at = threadIdx.x % kDims;   // rows part, part + PARTS, ...
    for (int d0 = 0; d0 < dim; d0 += kDims) {
        const int d = d0 + at;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        if (d < dim) {
            const float* x = data + d;
            int j = part;
            for (; j + 15 * PARTS < cnt; j += 16 * PARTS) {   // sixteen loads in flight
                float v[16];
#pragma unroll
                for (int t = 0; t < 16; ++t) v[t] = __ldg(x + (size_t)rows[j + PARTS * t] * dim);
#pragma unroll
                for (int t = 0; t < 16; ++t) acc[t & 3] += (double)v[t];
            }
            for (; j + 3 * PARTS < cnt; j += 4 * PARTS) {
                float v[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) v[t] = __ldg(x + (size_t)rows[j + PARTS * t] * dim);
#pragma unroll
                for (int t = 0; t < 4; ++t) acc[t] += (double)v[t];
            }
            for (; j < cnt; j += PARTS) acc[0] += (double)__ldg(x + (size_t)rows[j] * dim);
        }
        const double sum = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        if (part) s_part[part - 1][at] = sum;
        __syncthreads();
        if (!part && d < dim) {
            double total = sum;
#pragma unroll
            for (int p = 0; p < PARTS - 1; ++p) total += s_part[p][at];
            if (split) atomicAdd(&sums[(size_t)c * dim + d], total);
            else sums[(size_t)c * dim + d] = total;
        }
        __syncthreads();
    }
}

// Standard normal from a counter: Box-Muller on two 24-bit uniforms of one hashed 64-bit word.
__device__ __forceinline__ float normal_from(uint64_t seed, uint64_t counter) {
    const uint64_t h = splitmix64(splitmix64(seed) ^ (counter * 0xD1342543DE82EF95ull + 0x2545F4914F6CDD1Dull));
    const float u1 = ((float)((h >> 40) & 0xFFFFFF) + 1.0f) * (1.0f / 16777216.0f);  // (0,1]
    const float u2 = (float)((h >> 8) & 0xFFFFFF) * (1.0f / 16777216.0f);            // [0,1)
    return sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
}

__global__ void k_gen_mixture(const float* __restrict__ centres, const long long* __restrict__ offsets, int ncomp,
                              int dim, float sigma, uint64_t seed, long long row_begin, long long n,
                              float* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * dim) return;
    const long long row = row_begin + i / dim;
    const int d = (int)(i % dim);
    int lo = 0, hi = ncomp;  // largest c with offsets[c] <= row
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (offsets[mid] <= row) lo = mid; else hi = mid;
    }
    out[i] = centres[(size_t)lo * dim + d] + sigma * normal_from(seed, (uint64_t)row * (uint64_t)dim + (uint64_t)d);
}

__global__ void k_gen_normal(uint64_t seed, long long first, long long n, float scale, float* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = scale * normal_from(seed, (uint64_t)(first + i));
}

}  // namespace

psb_status launch_pq_encode(const float* d_data, long long n, int dim, const float* d_codebook, int m, int k,
                            uint8_t* d_codes, int sm_count, cudaStream_t s) {
    if (n <= 0) return PSB_OK;
    const int dsub = dim / m;
    if (pq_nearest_supported(dsub, k, false)) return launch_pq_nearest(d_data, n, dim, d_codebook, m, k, false, d_codes, sm_count, s);
    // Few codewords or long sub-vectors: one by one.
    const unsigned grid = (unsigned)((n + kEncThreads - 1) / kEncThreads);
    const size_t tile = (size_t)kEncThreads * (dim + 1) * sizeof(float) + (size_t)k * dsub * sizeof(float) + (size_t)kEncThreads * m;
    if (tile <= 200 * 1024) {  // rows staged in shared memory
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_pq_encode_tile), tile));
        k_pq_encode_tile<<<grid, kEncThreads, tile, s>>>(d_data, n, dim, d_codebook, m, k, d_codes);
    } else {
        const size_t smem = (size_t)k * dsub * sizeof(float) + (size_t)kEncThreads * m;
        if (smem > 32 * 1024) PSB_TRY(kernel_shared(reinterpret_cast<const void*>(k_pq_encode), smem));
        k_pq_encode<<<grid, kEncThreads, smem, s>>>(d_data, n, dim, d_codebook, m, k, d_codes);
    }
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_pq_assign_train(const float* d_data, long long n, int dim, const float* d_codebook, int m, int k,
                                  uint8_t* d_codes, int sm_count, cudaStream_t s) {
    if (n <= 0) return PSB_OK;
    if (pq_nearest_supported(dim / m, k, true)) return launch_pq_nearest(d_data, n, dim, d_codebook, m, k, true, d_codes, sm_count, s);
    return launch_pq_encode(d_data, n, dim, d_codebook, m, k, d_codes, sm_count, s);
}

psb_status launch_pq_accumulate(const float* d_data, long long n, int dim, const uint8_t* d_codes, int m, int k,
                                double* d_sums, int* d_counts, cudaStream_t s) {
    if (n <= 0) return PSB_OK;
    k_pq_accumulate<<<dim3((unsigned)((n + kPqAccRows - 1) / kPqAccRows), (unsigned)m), kPqAccThreads, 0, s>>>(d_data, n, dim, d_codes, m, k, d_sums, d_counts);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_pq_update(double* d_sums, int* d_counts, int m, int k, int dsub, float* d_codebook, cudaStream_t s) {
    k_pq_update<<<(unsigned)((m * k + 127) / 128), 128, 0, s>>>(d_sums, d_counts, m * k, dsub, d_codebook);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

// A CTA of the seeding keeps four bytes per row at least.
bool pq_seed_fits(long long n) { return (n + kSeedCluster - 1) / kSeedCluster * 4 <= (long long)200 * 1024; }

psb_status launch_pq_seed(const float* d_data, int n, int dim, int m, int k, const double* d_draws, const int* d_first, long long* d_rows,
                          int* d_status, cudaStream_t s) {
    const int dsub = dim / m;
    const int per = (n + kSeedCluster - 1) / kSeedCluster;
    const size_t mins = (size_t)(per + 511) / 256 * 1024, rows = (size_t)per * dsub * 4;
    const int staged = mins + rows <= (size_t)202 * 1024 ? 1 : 0;   // 2 KB for the places past a stretch's end
    const size_t smem = mins + (staged ? rows : 0);
    auto run = [&](auto few, auto many) -> psb_status {
        auto kernel = per <= kSeedShort * kSeedCtaWarps ? few : many;
        PSB_TRY(kernel_shared(reinterpret_cast<const void*>(kernel), smem));
        kernel<<<dim3(kSeedCluster, (unsigned)m), kSeedCtaThreads, smem, s>>>(d_data, n, dim, dsub, k, per, staged, d_draws, d_first, d_rows, d_status);
        return PSB_OK;
    };
    switch (dsub) {
        case 2: PSB_TRY(run(k_pq_seed<2, true>, k_pq_seed<2, false>)); break;
        case 3: PSB_TRY(run(k_pq_seed<3, true>, k_pq_seed<3, false>)); break;
        case 4: PSB_TRY(run(k_pq_seed<4, true>, k_pq_seed<4, false>)); break;
        case 5: PSB_TRY(run(k_pq_seed<5, true>, k_pq_seed<5, false>)); break;
        case 6: PSB_TRY(run(k_pq_seed<6, true>, k_pq_seed<6, false>)); break;
        case 8: PSB_TRY(run(k_pq_seed<8, true>, k_pq_seed<8, false>)); break;
        default: PSB_TRY(run(k_pq_seed<0, true>, k_pq_seed<0, false>)); break;
    }
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

// codebook[sub][c] = the sub-vector `sub` of data row rows[sub * k + c]
__global__ void k_pq_init_rows(const float* __restrict__ data, int dim, int m, int k, const long long* __restrict__ rows,
                               float* __restrict__ codebook) {
    const int dsub = dim / m;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)m * k * dsub) return;
    const int d = (int)(i % dsub);
    const long long e = i / dsub;   // sub * k + c
    const int sub = (int)(e / k);
    codebook[i] = data[(size_t)rows[e] * dim + (size_t)sub * dsub + d];
}

psb_status launch_pq_init_rows(const float* d_data, int dim, int m, int k, const long long* d_rows, float* d_codebook, cudaStream_t s) {
    const long long total = (long long)m * k * (dim / m);
    k_pq_init_rows<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(d_data, dim, m, k, d_rows, d_codebook);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_kmeans_accumulate(const float* d_data, long long n, int dim, const int* d_assign, const float* d_best, int k,
                                    double* d_sums, int* d_counts, double* d_obj, const KmeansAccumWs& ws, cudaStream_t s) {
    if (n > 0x7fffffffLL) return fail(PSB_UNSUPPORTED_SHAPE, "more than 2^31-1 rows in one accumulation");
    if (!ws.order || !ws.offsets || !ws.cursor) return fail(PSB_INTERNAL, "k-means accumulation workspace missing");
    // d_counts and *d_obj were zeroed by the caller; d_sums is written whole
    const bool few = k <= kFewCentroids && n >= kFewLeast && n >= kFewPerCentroid * k;
    if (n > 0) {
        if (few) k_km_count_few<<<(unsigned)((n + kFewRows - 1) / kFewRows), 1024, 0, s>>>(d_assign, d_best, n, k, d_counts, d_obj);
        else k_km_count<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_assign, d_best, n, k, d_counts, d_obj);
        count_launch();
        PSB_LAUNCH_CHECK();
    }
    k_km_offsets<<<1, 1024, 0, s>>>(d_counts, k, ws.offsets, ws.cursor);
    count_launch();
    PSB_LAUNCH_CHECK();
    if (n > 0) {
        if (few) k_km_fill_few<<<(unsigned)((n + kFewRows - 1) / kFewRows), 1024, 0, s>>>(d_assign, n, k, ws.offsets, ws.cursor, ws.order);
        else k_km_fill<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_assign, n, k, ws.offsets, ws.cursor, ws.order);
        count_launch();
        PSB_LAUNCH_CHECK();
    }
    PSB_CUDA(cudaMemsetAsync(d_sums, 0, sizeof(double) * (size_t)k * dim, s));   // what the split groups add to
    // Average groups of 128 rows and more: eight threads a dimension (400,000 x 128 to 64
    // centroids, five iterations: with 256 threads 6.0 ms, with 1,024 4.7).
    if (n / k >= 128) k_km_sums<1024><<<dim3((unsigned)k, kKmSplit), 1024, 0, s>>>(d_data, dim, ws.offsets, ws.order, d_sums);
    else k_km_sums<256><<<dim3((unsigned)k, kKmSplit), 256, 0, s>>>(d_data, dim, ws.offsets, ws.order, d_sums);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_kmeans_update(const double* d_sums, const int* d_counts, int k, int dim, float* d_centroids,
                                cudaStream_t s) {
    const long long total = (long long)k * dim;
    k_mean_update<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(d_sums, d_counts, k, dim, d_centroids);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_residual_rows(const float* d_data, long long n, int dim, const float* d_centroids, const int* d_assign,
                                float* d_out, cudaStream_t s) {
    if (n <= 0) return PSB_OK;
    k_residual_rows<<<(unsigned)((n * dim + 255) / 256), 256, 0, s>>>(d_data, n, dim, d_centroids, d_assign, d_out);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_gen_mixture(const float* d_centres, const long long* d_offsets, int ncomp, int dim, float sigma,
                              uint64_t seed, long long row_begin, long long n, float* d_out, cudaStream_t s) {
    if (n <= 0) return PSB_OK;
    const long long total = n * dim;
    k_gen_mixture<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(d_centres, d_offsets, ncomp, dim, sigma, seed, row_begin, n, d_out);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

psb_status launch_gen_normal(uint64_t seed, long long first, long long n, float scale, float* d_out, cudaStream_t s) {
    if (n <= 0) return PSB_OK;
    k_gen_normal<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(seed, first, n, scale, d_out);
    count_launch();
    PSB_LAUNCH_CHECK();
    return PSB_OK;
}

}  // namespace psb
