// TurboQuant 1-bit residual codec: random sign flips and a Walsh-Hadamard rotation, one sign bit per rotated dimension and one
// scale per row, and the candidate search over sign-coded lists.
//
//   k_sign_encode   one warp per row.  The reference runs one CTA of padded_dim threads per row with the values in shared
//                   memory and a __syncthreads() per butterfly width (src/quantization/turboquant/turboquant_1bit_encode.cu:
//                   33-110); here lane l holds elements l, l+32, l+64, ... in registers, widths below 32 are lane exchanges and
//                   widths from 32 up are register pairs.  Every butterfly still computes (lhs + rhs, lhs - rhs) on the same
//                   pairs, the per-row statistic goes through the same two shuffle-down trees, so the bits are the same; a row
//                   costs no barrier and the loads of 8 rows per CTA are in flight together.
//   k_sign_scan_*   one CTA per (query, slice of its probes): rows of the probed lists are scored against the state of their
//                   (query, probe) - one chain over d = 0..dim-1 of +-state[d] for float states, a popcount for sign-coded
//                   ones (src/quantization/turboquant/turboquant_1bit_score.cuh:17-72) - and the candidate_count smallest
//                   (score, row) keys are kept in shared memory: a row enters the buffer only below the current cutoff, a full
//                   buffer is cut back to candidate_count by a radix selection, and the survivors are sorted once at the end.
//                   For float states the tensor cores give every row a score with a known error bound first; only rows that
//                   could be among the candidate_count get the exact chain (see the kernel).  The reference sorts every
//                   group of 8 chunks of 2,048 rows and merges the groups' lists per query
//                   (turboquant_1bit_grouped_scan.cu:92-190, 45-90); the result, the exact candidate_count smallest keys in
//                   ascending order, is the same.
//   k_sign_merge    joins the slices of one query when its probes were split over several CTAs (few queries).
#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "kernels.h"

namespace psb {

namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ uint32_t sign_mix(uint32_t v) {   // turboquant_1bit_encode.cu:13-19
    v ^= v >> 16; v *= 0x7feb352du; v ^= v >> 15; v *= 0x846ca68bu;
    return v ^ (v >> 16);
}

// Lane 0 gets what lane 0 of a warp holds after `for delta = 16..1: v += shfl_down(v, delta)`.
__device__ __forceinline__ float tree32(float v) {
#pragma unroll
    for (int delta = 16; delta > 0; delta >>= 1) v = __fadd_rn(v, __shfl_down_sync(kFull, v, delta));
    return v;
}

// Sum of one value per element in the order of the reference's block reduction: a tree per 32 elements, then the same tree
// over the group sums (zero beyond the last group).  Valid on lane 0.
template <int J>
__device__ __forceinline__ float block_order_sum(const float (&x)[J], int lane) {
    float g = 0.f;
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const float t = __shfl_sync(kFull, tree32(x[j]), 0);
        if (lane == j) g = t;
    }
    return tree32(g);
}

// v[j] = element lane + 32 j of the (zero padded) row on entry, of the rotated row on return.
template <int J>
__device__ __forceinline__ void rotate_in_warp(float (&v)[J], int lane, uint32_t seed, float scale) {
#pragma unroll
    for (int j = 0; j < J; ++j)
        if (sign_mix(seed ^ (uint32_t)(lane + 32 * j)) & 1u) v[j] = -v[j];
#pragma unroll
    for (int w = 1; w < 32; w <<= 1) {
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const float o = __shfl_xor_sync(kFull, v[j], w);
            v[j] = (lane & w) ? __fsub_rn(o, v[j]) : __fadd_rn(v[j], o);   // right: lhs - rhs, left: lhs + rhs
        }
    }
#pragma unroll
    for (int wj = 1; wj < J; wj <<= 1) {
#pragma unroll
        for (int j = 0; j < J; ++j)
            if ((j & wj) == 0) {
                const float lhs = v[j], rhs = v[j | wj];
                v[j] = __fadd_rn(lhs, rhs);
                v[j | wj] = __fsub_rn(lhs, rhs);
            }
    }
#pragma unroll
    for (int j = 0; j < J; ++j) v[j] = __fmul_rn(v[j], scale);
}

struct SignEncodeArgs {
    int kind;                    // 0 rows as given, 1 database rows minus their list's centroid, 2 (query, probe) residuals
    const void* rows;            // kind 0/2: fp32 [n][dim] (kind 2: the queries); kind 1: u8 or fp32 rows
    int elem_bytes;              // kind 1: 1 or 4
    long long n;                 // rows / states to encode
    const float* centroids;      // kind 1/2
    const long long* offsets;    // kind 1: [nlist + 1]
    const int* probes;           // kind 2: [n]
    int nlist, nprobe, dim, padded;
    uint32_t seed;
    long long row_offset;        // kind 1: global row of rows[0]
    float* rotated;              // [n][padded] or null
    uint32_t* codes;             // [.][padded / 32] or null
    float* norms;                // kind 0/2: sqrt(sum x^2); kind 1: L1 scale
    float* norm_sq;              // kind 0/2: sum x^2
};

template <int J>
__global__ void __launch_bounds__(256) k_sign_encode(const SignEncodeArgs a) {
    const int lane = threadIdx.x & 31;
    const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const float scale = rsqrtf((float)a.padded);   // on the device from a run-time value, as the reference's kernel takes it
    // A warp takes a run of consecutive rows: consecutive database rows mostly share a list, whose bounds are then at hand.
    const long long per_warp = (a.n + nwarps - 1) / nwarps;
    const long long r_end = min(a.n, (warp0 + 1) * per_warp);
    int held_list = 0;
    long long held_beg = 0, held_end = -1;
    for (long long r = warp0 * per_warp; r < r_end; ++r) {
        long long out_row = r;
        const float* cen = nullptr;
        const float* src_f = nullptr;
        const unsigned char* src_b = nullptr;
        bool live = true;
        if (a.kind == 0) {
            src_f = static_cast<const float*>(a.rows) + (size_t)r * a.dim;
        } else if (a.kind == 1) {
            out_row = r + a.row_offset;
            if (out_row < held_beg || out_row >= held_end) {
                int lo = 0, hi = a.nlist;   // the list of the global row (turboquant_1bit_encode.cu:21-31)
                while (lo + 1 < hi) {
                    const int mid = lo + (hi - lo) / 2;
                    if (a.offsets[mid] <= out_row) lo = mid; else hi = mid;
                }
                held_list = lo; held_beg = a.offsets[lo]; held_end = a.offsets[lo + 1];
            }
            cen = a.centroids + (size_t)held_list * a.dim;
            if (a.elem_bytes == 1) src_b = static_cast<const unsigned char*>(a.rows) + (size_t)r * a.dim;
            else src_f = static_cast<const float*>(a.rows) + (size_t)r * a.dim;
        } else {
            const int list = a.probes[r];
            live = list >= 0 && list < a.nlist;
            src_f = static_cast<const float*>(a.rows) + (size_t)(r / a.nprobe) * a.dim;
            cen = a.centroids + (size_t)(live ? list : 0) * a.dim;
        }
        float v[J], stat[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int d = lane + 32 * j;
            float x = 0.f;
            if (live && d < a.dim) {
                x = src_b ? (float)src_b[d] : src_f[d];
                if (cen) x = __fsub_rn(x, cen[d]);
            }
            v[j] = x;
            stat[j] = __fmul_rn(x, x);
        }
        rotate_in_warp<J>(v, lane, a.seed, scale);
#pragma unroll
        for (int j = 0; j < J; ++j) {
            if (a.rotated) a.rotated[(size_t)out_row * (32 * J) + lane + 32 * j] = v[j];
            const unsigned word = __ballot_sync(kFull, v[j] >= 0.0f);
            if (a.codes && lane == 0) a.codes[(size_t)out_row * J + j] = word;
            if (a.kind == 1) stat[j] = fabsf(v[j]);
        }
        if (a.norms || a.norm_sq) {   // uniform
            const float sum = block_order_sum<J>(stat, lane);
            if (lane == 0) {
                if (a.kind == 1) {
                    if (a.norms) a.norms[out_row] = __fdiv_rn(sum, (float)(32 * J));
                } else {
                    if (a.norm_sq) a.norm_sq[out_row] = sum;
                    if (a.norms) a.norms[out_row] = __fsqrt_rn(sum);
                }
            }
        }
    }
}

// The same encoding with one row per THREAD, for padded_dim <= 128 and rows whose length is a multiple of four elements: the
// whole (zero padded) row sits in registers, every butterfly is two register operations and nothing is exchanged between
// lanes (the warp-per-row kernel above spends 49 shuffles per row).  Every value goes through the same operations on the
// same operands - the sign flip, the (lhs + rhs, lhs - rhs) pairs width by width, the scale, the two reduction trees of the
// statistic taken as register trees - so the bits are the same.  A thread reads its row with 16-byte (fp32) or 4-byte (u8)
// loads; the row is a run of whole sectors, read once.
constexpr int kLaneEncThreads = 128;

// What lane 0 of a warp would hold after the shuffle-down tree over t[0..32): t[p] += t[p + delta], delta = 16 .. 1.
__device__ __forceinline__ float tree32_regs(float (&t)[32]) {
#pragma unroll
    for (int delta = 16; delta > 0; delta >>= 1) {
#pragma unroll
        for (int p = 0; p < delta; ++p) t[p] = __fadd_rn(t[p], t[p + delta]);
    }
    return t[0];
}

template <int P>
__global__ void __launch_bounds__(kLaneEncThreads, 2) k_sign_encode_lane(const SignEncodeArgs a) {
    __shared__ uint32_t s_flip[P];   // 0x80000000 where the rotation flips the sign of dimension d
    for (int d = threadIdx.x; d < P; d += kLaneEncThreads) s_flip[d] = (sign_mix(a.seed ^ (uint32_t)d) & 1u) ? 0x80000000u : 0u;
    __syncthreads();
    const float scale = rsqrtf((float)a.padded);   // on the device from a run-time value, as the reference's kernel takes it
    const int dim4 = a.dim >> 2;
    // A thread takes a run of consecutive rows: consecutive database rows mostly share a list, whose bounds are then at hand
    // (the search is 16 dependent loads).
    const long long threads = (long long)gridDim.x * kLaneEncThreads;
    const long long per_thread = (a.n + threads - 1) / threads;
    const long long r_begin = ((long long)blockIdx.x * kLaneEncThreads + threadIdx.x) * per_thread;
    const long long r_end = min(a.n, r_begin + per_thread);
    int held_list = 0;
    long long held_beg = 0, held_end = -1;
    const bool bytes16 = (a.dim & 15) == 0 && (reinterpret_cast<uintptr_t>(a.rows) & 15) == 0;   // u8 rows in 16-byte loads
    for (long long r = r_begin; r < r_end; ++r) {
        long long out_row = r;
        const float* cen = nullptr;
        const float* src_f = nullptr;
        const unsigned char* src_b = nullptr;
        bool live = true;
        if (a.kind == 0) {
            src_f = static_cast<const float*>(a.rows) + (size_t)r * a.dim;
        } else if (a.kind == 1) {
            out_row = r + a.row_offset;
            if (out_row < held_beg || out_row >= held_end) {
                int lo = 0, hi = a.nlist;   // the list of the global row (turboquant_1bit_encode.cu:21-31)
                while (lo + 1 < hi) {
                    const int mid = lo + (hi - lo) / 2;
                    if (a.offsets[mid] <= out_row) lo = mid; else hi = mid;
                }
                held_list = lo; held_beg = a.offsets[lo]; held_end = a.offsets[lo + 1];
            }
            cen = a.centroids + (size_t)held_list * a.dim;
            if (a.elem_bytes == 1) src_b = static_cast<const unsigned char*>(a.rows) + (size_t)r * a.dim;
            else src_f = static_cast<const float*>(a.rows) + (size_t)r * a.dim;
        } else {
            const int list = a.probes[r];
            live = list >= 0 && list < a.nlist;
            src_f = static_cast<const float*>(a.rows) + (size_t)(r / a.nprobe) * a.dim;
            cen = a.centroids + (size_t)(live ? list : 0) * a.dim;
        }
        float v[P];
        uint4 packed = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int d4 = 0; d4 < P / 4; ++d4) {
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live && d4 < dim4) {
                if (src_b) {
                    uint32_t word;
                    if (bytes16) {   // uniform; the 16-byte load of group d4 / 4 serves four passes of this loop
                        if ((d4 & 3) == 0) packed = __ldg(reinterpret_cast<const uint4*>(src_b) + (d4 >> 2));
                        word = (d4 & 3) == 0 ? packed.x : (d4 & 3) == 1 ? packed.y : (d4 & 3) == 2 ? packed.z : packed.w;
                    } else {
                        word = __ldg(reinterpret_cast<const uint32_t*>(src_b) + d4);
                    }
                    x = make_float4((float)(word & 255u), (float)((word >> 8) & 255u), (float)((word >> 16) & 255u), (float)(word >> 24));
                } else {
                    x = __ldg(reinterpret_cast<const float4*>(src_f) + d4);
                }
                if (cen) {
                    const float4 c = __ldg(reinterpret_cast<const float4*>(cen) + d4);
                    x.x = __fsub_rn(x.x, c.x); x.y = __fsub_rn(x.y, c.y); x.z = __fsub_rn(x.z, c.z); x.w = __fsub_rn(x.w, c.w);
                }
            }
            v[4 * d4] = x.x; v[4 * d4 + 1] = x.y; v[4 * d4 + 2] = x.z; v[4 * d4 + 3] = x.w;
        }
        float sum = 0.f;
        if (a.kind != 1 && (a.norms || a.norm_sq)) {   // sum of squares of the row as given, group trees then the tree over groups
            float g[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) g[i] = 0.f;
#pragma unroll
            for (int w = 0; w < P / 32; ++w) {
                float t[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) t[i] = __fmul_rn(v[32 * w + i], v[32 * w + i]);
                g[w] = tree32_regs(t);
            }
            sum = tree32_regs(g);
        }
#pragma unroll
        for (int d = 0; d < P; ++d) v[d] = __uint_as_float(__float_as_uint(v[d]) ^ s_flip[d]);
#pragma unroll
        for (int width = 1; width < P; width <<= 1) {
#pragma unroll
            for (int t = 0; t < P / 2; ++t) {
                const int left = (t / width) * (width << 1) + (t % width), right = left + width;
                const float lhs = v[left], rhs = v[right];
                v[left] = __fadd_rn(lhs, rhs);
                v[right] = __fsub_rn(lhs, rhs);
            }
        }
#pragma unroll
        for (int d = 0; d < P; ++d) v[d] = __fmul_rn(v[d], scale);
        if (a.rotated) {
            float4* out = reinterpret_cast<float4*>(a.rotated + (size_t)out_row * P);
#pragma unroll
            for (int d4 = 0; d4 < P / 4; ++d4) out[d4] = make_float4(v[4 * d4], v[4 * d4 + 1], v[4 * d4 + 2], v[4 * d4 + 3]);
        }
        if (a.codes) {
#pragma unroll
            for (int w = 0; w < P / 32; ++w) {
                uint32_t word = 0u;
#pragma unroll
                for (int b = 0; b < 32; ++b) word |= v[32 * w + b] >= 0.0f ? (1u << b) : 0u;
                a.codes[(size_t)out_row * (P / 32) + w] = word;
            }
        }
        if (a.kind == 1) {
            if (a.norms) {
                float g[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) g[i] = 0.f;
#pragma unroll
                for (int w = 0; w < P / 32; ++w) {
                    float t[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) t[i] = fabsf(v[32 * w + i]);
                    g[w] = tree32_regs(t);
                }
                a.norms[out_row] = __fdiv_rn(tree32_regs(g), (float)P);
            }
        } else {
            if (a.norm_sq) a.norm_sq[out_row] = sum;
            if (a.norms) a.norms[out_row] = __fsqrt_rn(sum);
        }
    }
}

__global__ void k_sign_scale(int padded, float* out) { *out = rsqrtf((float)padded); }

// ---- candidate search ------------------------------------------------------------------------------------------

constexpr int kScanThreads = 256;
constexpr int kScanRows = 4;                      // rows per thread per step
constexpr int kScanStep = kScanThreads * kScanRows;
constexpr int kSignMaxCandidates = 8192;
constexpr int kMergeMaxKeys = 16384;

struct SignScanArgs {
    const float* states;          // float states [nq * nprobe][dim]
    const float* norm_sq;         // [nq * nprobe]
    const uint32_t* state_codes;  // sign-coded states [nq * nprobe][dim / 32]
    const float* norms;           // [nq * nprobe]
    const uint32_t* codes;        // [rows][dim / 32]
    const float* row_params;      // [rows]: reconstruction scale (float states) or norm (sign-coded states)
    const long long* offsets;     // [nlist + 1]
    const int* probes;            // [nq][nprobe]
    int nlist, nq, nprobe, dim, k, kp2, cap, split;
    int seg;                      // waiting rows per warp (float states)
    uint64_t* partial;            // [nq][split][k] when split > 1
    int* rows_out;                // [nq][k]
    float* dist_out;              // [nq][k] or null
};

template <int W> struct CodeWords { uint32_t w[W]; };

template <int W>
__device__ __forceinline__ CodeWords<W> load_code(const uint32_t* __restrict__ codes, long long row) {
    CodeWords<W> c;
    if constexpr (W == 1) {
        c.w[0] = __ldg(codes + row);
    } else if constexpr (W == 2) {
        const uint2 t = __ldg(reinterpret_cast<const uint2*>(codes) + row);
        c.w[0] = t.x; c.w[1] = t.y;
    } else {
#pragma unroll
        for (int i = 0; i < W / 4; ++i) {
            const uint4 t = __ldg(reinterpret_cast<const uint4*>(codes) + row * (W / 4) + i);
            c.w[4 * i] = t.x; c.w[4 * i + 1] = t.y; c.w[4 * i + 2] = t.z; c.w[4 * i + 3] = t.w;
        }
    }
    return c;
}

// dot + v when the sign bit is set, dot - v when it is clear: one bit test into a predicate and two predicated adds.  Building
// +-v with a shift and an exclusive-or instead costs two integer operations per dimension, which run at half the rate of the
// adds; measured, this form is the faster of the two by a few percent.
__device__ __forceinline__ float sign_step(float dot, float v, uint32_t word, uint32_t mask) {
    asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\t"
        "and.b32 t, %1, %2;\n\t"
        "setp.ne.u32 p, t, 0;\n\t"
        "@p add.rn.f32 %0, %0, %3;\n\t"
        "@!p sub.rn.f32 %0, %0, %3;\n\t}"
        : "+f"(dot)
        : "r"(word), "r"(mask), "f"(v));
    return dot;
}

// Shared scratch of the selection: a 256-bin histogram, the warp sums of its scan, and a few words.
struct SignSelectScratch {
    int hist[256];
    int warp_sums[32];
    int bucket, need, moved, filled;
    unsigned long long differ;
};

// Cuts the buffer back to its k smallest keys, keys[0..k) in no particular order, and moves the cutoff to the k-th smallest.
// A radix selection over the bytes of the keys (most significant first, bytes that all keys share skipped) finds the k-th
// key in a few passes over the buffer; keys beyond position k that stay are parked in `spill` and dropped into the places of
// keys within the first k that go.  A full sort of the buffer here cost two thirds of the instructions of the popcount scan
// and a fifth of those of the float scan.  Called by all threads of the CTA (blockDim.x == 256).
__device__ __forceinline__ void sign_compact(uint64_t* keys, uint64_t* spill, int k, int* s_cnt, unsigned long long* s_thr,
                                             SignSelectScratch* sc) {
    const int n = *s_cnt;
    const int tid = threadIdx.x;
    __syncthreads();
    if (n <= k) return;   // uniform
    if (tid == 0) sc->differ = 0ull;
    __syncthreads();
    const uint64_t first = keys[0];
    uint64_t diff = 0;
    for (int i = tid; i < n; i += kScanThreads) diff |= keys[i] ^ first;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) diff |= __shfl_xor_sync(kFull, diff, o);
    if ((tid & 31) == 0 && diff) atomicOr(&sc->differ, (unsigned long long)diff);
    __syncthreads();
    const unsigned long long differ = sc->differ;
    // keys are distinct unless a query names a list twice; all equal: any k of them will do
    int shift = differ ? 56 - 8 * (__clzll((long long)differ) / 8) : -8;
    uint64_t prefix = shift >= 0 && shift < 56 ? first & (~0ull << (shift + 8)) : 0ull;
    int need = k;
    for (; shift >= 0; shift -= 8) {
        sc->hist[tid] = 0;
        __syncthreads();
        const uint64_t above = shift == 56 ? 0ull : ~0ull << (shift + 8);
        for (int i = tid; i < n; i += kScanThreads) {
            const uint64_t key = keys[i];
            if ((key & above) == prefix) atomicAdd(&sc->hist[(int)((key >> shift) & 255u)], 1);
        }
        __syncthreads();
        const int c = sc->hist[tid];
        const int before = block_exclusive_scan(c, sc->warp_sums, nullptr);
        if (before < need && need <= before + c) { sc->bucket = tid; sc->need = need - before; }
        __syncthreads();
        prefix |= (uint64_t)sc->bucket << shift;
        need = sc->need;
        __syncthreads();
    }
    const uint64_t kth = differ ? prefix : first;
    if (tid == 0) { sc->moved = 0; sc->filled = 0; }
    __syncthreads();
    // keys below the k-th first, then keys equal to it (more than one only when a query names a list twice): the places that
    // come free go to the parked keys in this order
    for (int pass = 0; pass < 2; ++pass) {
        for (int i = k + tid; i < n; i += kScanThreads) {
            const uint64_t key = keys[i];
            if (pass == 0 ? key < kth : key == kth) {
                const int pos = atomicAdd(&sc->moved, 1);
                if (pos < k) spill[pos] = key;
            }
        }
        __syncthreads();
    }
    const int moved = sc->moved < k ? sc->moved : k;
    for (int j = tid; j < k; j += kScanThreads) {
        if (keys[j] > kth) {
            const int pos = atomicAdd(&sc->filled, 1);
            keys[j] = pos < moved ? spill[pos] : KEY_MAX;   // pos < moved always, for distinct keys
        }
    }
    if (tid == 0) { *s_cnt = k; *s_thr = kth; }
    __syncthreads();
}

// The kept keys in ascending order in keys[0..n), n = min(held, k).
__device__ __forceinline__ int sign_finish(uint64_t* keys, uint64_t* spill, int k, int kp2, int* s_cnt, unsigned long long* s_thr,
                                           SignSelectScratch* sc) {
    sign_compact(keys, spill, k, s_cnt, s_thr, sc);
    const int n = *s_cnt;
    __syncthreads();
    for (int i = n + threadIdx.x; i < kp2; i += kScanThreads) keys[i] = KEY_MAX;
    __syncthreads();
    block_bitonic_sort(keys, kp2);
    return n;
}

// The exact scores of up to kScanRows rows per thread, each against the float state `state[r]` points to (global memory: the
// rows of a thread may belong to different probes): one chain over d = 0..dim-1 per row, the chains interleaved.
template <int W, bool WIDE>   // WIDE: the states are 16-byte aligned
__device__ __forceinline__ void exact_float_scores(const CodeWords<W> (&c)[kScanRows], const float (&param)[kScanRows],
                                                   const float* const (&state)[kScanRows], const float (&norm_sq)[kScanRows],
                                                   float (&score)[kScanRows]) {
    float dot[kScanRows];
#pragma unroll
    for (int r = 0; r < kScanRows; ++r) dot[r] = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
#pragma unroll
        for (int bit = 0; bit < 32; bit += 4) {
            float4 v[kScanRows];
#pragma unroll
            for (int r = 0; r < kScanRows; ++r) {
                const float* x = state[r] + 32 * w + bit;
                if (WIDE) v[r] = __ldg(reinterpret_cast<const float4*>(x));
                else v[r] = make_float4(__ldg(x), __ldg(x + 1), __ldg(x + 2), __ldg(x + 3));
            }
#pragma unroll
            for (int r = 0; r < kScanRows; ++r) dot[r] = sign_step(dot[r], v[r].x, c[r].w[w], 1u << bit);
#pragma unroll
            for (int r = 0; r < kScanRows; ++r) dot[r] = sign_step(dot[r], v[r].y, c[r].w[w], 2u << bit);
#pragma unroll
            for (int r = 0; r < kScanRows; ++r) dot[r] = sign_step(dot[r], v[r].z, c[r].w[w], 4u << bit);
#pragma unroll
            for (int r = 0; r < kScanRows; ++r) dot[r] = sign_step(dot[r], v[r].w, c[r].w[w], 8u << bit);
        }
    }
    const float dimf = (float)(32 * W);
#pragma unroll
    for (int r = 0; r < kScanRows; ++r) {
        const float s = param[r];
        score[r] = __fmaf_rn(-__fmul_rn(2.0f, s), dot[r], __fmaf_rn(__fmul_rn(dimf, s), s, norm_sq[r]));
    }
}

constexpr int kUnitRows = 64, kStepUnits = 2;   // rows a warp takes at a time, and how often between two looks at the queue

// The filter's dot products, on the integer tensor cores.  A row's sign bits b_d are bytes of the left operand: a code word masked with
// 0x01010101 << p holds four of them as 0 or 2^p, p < 4, and the word shifted right by 4 the other half, so an operand register costs
// one mask.  The state is two columns of bytes, w_d = 256 hi_d + lo_d = state[d] / (2^p delta) to the nearest, p = d mod 4, and
//   sum +-state[d] = delta (2 (256 sum b 2^p hi + sum b 2^p lo) - sum 2^p w)   within  delta / 2 (1 + 2 + 4 + 8) dim / 4.
// The sums are exact whole numbers.  All four column pairs of mma.m16n8k32 hold the same two columns: after four tiles of 16 rows
// every thread picks the tile of its own and has two rows.
// Which bits make which K slots is free as long as the state's bytes follow: thread t of a quad takes word t (padded_dim 128; its half
// of word t / 2 for 64, a quarter of the only word for 32, words t and t + 4 for 256), byte positions p and p + 1 of it per step.
__device__ __forceinline__ void imma_16832(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <int W> __device__ __forceinline__ int slot_word(int s, int t) { return W >= 4 ? t + 4 * (s >> 2) : (W == 2 ? t >> 1 : 0); }
template <int W> __device__ __forceinline__ int slot_bit(int s, int t) { return W >= 4 ? 2 * (s & 3) : (W == 2 ? 4 * (t & 1) + 2 * s : 2 * t); }
// out[0], out[1]: sum b 2^p w of rows base + 16 t + g and + 8 (t, g: lane % 4, lane / 4); rows past `last`, the last of all, repeat it.
template <int W>
__device__ __forceinline__ void tile_dots(const uint32_t* __restrict__ codes, int base, int last, const uint2 (&b)[W], int (&out)[2]) {
    constexpr int WPT = W >= 4 ? W / 4 : 1;
    const int lane = threadIdx.x & 31, t = lane & 3, g = lane >> 2;
    uint32_t x[4][2][WPT];
    if (base + kUnitRows - 1 <= last) {   // warp-uniform; one address, for padded_dim 128 consecutive words in every load
        const uint32_t* code = codes + (size_t)(base + g) * W + slot_word<W>(0, t);
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int i = 0; i < WPT; ++i) x[j >> 1][j & 1][i] = __ldg(code + 8 * j * W + 4 * i);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int i = 0; i < WPT; ++i) x[j >> 1][j & 1][i] = __ldg(codes + (size_t)min(base + 8 * j + g, last) * W + slot_word<W>(4 * i, t));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int acc[4] = {0, 0, 0, 0};
#pragma unroll
        for (int s = 0; s < W; ++s) {
            const int p = slot_bit<W>(s, t), i = W >= 4 ? s >> 2 : 0;
            const uint32_t u = x[j][0][i] >> (p & 4), v = x[j][1][i] >> (p & 4);
            const uint32_t m0 = 0x01010101u << (p & 3), m1 = m0 << 1;
            imma_16832(acc, u & m0, v & m0, u & m1, v & m1, b[s].x, b[s].y);
        }
        if (t == j) { out[0] = 256 * acc[0] + acc[1]; out[1] = 256 * acc[2] + acc[3]; }
    }
}

// The kept keys to the query's output, or to its slice's place for k_sign_merge.
__device__ __forceinline__ void sign_output(const SignScanArgs& a, int q, int slice, const uint64_t* keys, int n) {
    if (a.split > 1) {
        uint64_t* out = a.partial + ((size_t)q * a.split + slice) * a.k;
        for (int i = threadIdx.x; i < a.k; i += kScanThreads) out[i] = i < n ? keys[i] : KEY_MAX;
    } else {
        for (int i = threadIdx.x; i < a.k; i += kScanThreads) {
            a.rows_out[(size_t)q * a.k + i] = i < n ? (int)key_idx(keys[i]) : -1;
            if (a.dist_out) a.dist_out[(size_t)q * a.k + i] = i < n ? key_dist(keys[i]) : FLT_MAX;
        }
    }
}

// Sign-coded states: every row's score is a popcount; keys below the cutoff go to the buffer.  One CTA per (query, slice of probes).
template <int W>
__global__ void __launch_bounds__(kScanThreads, W > 4 ? 2 : 6) k_sign_scan_codes(const SignScanArgs a) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    uint64_t* keys = reinterpret_cast<uint64_t*>(s_raw);
    uint64_t* spill = keys + a.cap;   // k keys
    __shared__ SignSelectScratch s_sel;
    __shared__ int s_cnt;
    __shared__ unsigned long long s_thr;
    const int q = blockIdx.x / a.split, slice = blockIdx.x % a.split;
    const int tid = threadIdx.x;
    const float dimf = (float)(32 * W);
    if (tid == 0) { s_cnt = 0; s_thr = KEY_MAX; }
    __syncthreads();
    for (int p = slice; p < a.nprobe; p += a.split) {
        const long long st = (long long)q * a.nprobe + p;
        const int list = a.probes[st];
        if (list < 0 || list >= a.nlist) continue;   // uniform
        uint32_t qcode[W];   // the state's sign words, the same in every thread
#pragma unroll
        for (int w = 0; w < W; ++w) qcode[w] = __ldg(a.state_codes + (size_t)st * W + w);
        const float qparam = a.norms[st];
        const long long beg = a.offsets[list], end = a.offsets[list + 1];
        for (long long row0 = beg; row0 < end; row0 += kScanStep) {
            const int held = s_cnt;   // settled: the previous step ended with a barrier
            __syncthreads();          // ... and nobody appends before everybody has read it
            if (held > a.cap - kScanStep) sign_compact(keys, spill, a.k, &s_cnt, &s_thr, &s_sel);   // uniform
            const unsigned long long thr = s_thr;
            CodeWords<W> c[kScanRows];
            float param[kScanRows];
            bool ok[kScanRows];
            long long rows[kScanRows];
#pragma unroll
            for (int r = 0; r < kScanRows; ++r) {
                rows[r] = row0 + r * kScanThreads + tid;
                ok[r] = rows[r] < end;
                if (ok[r]) { c[r] = load_code<W>(a.codes, rows[r]); param[r] = __ldg(a.row_params + rows[r]); }
                else {
#pragma unroll
                    for (int w = 0; w < W; ++w) c[r].w[w] = 0u;
                    param[r] = 0.f;
                }
            }
#pragma unroll
            for (int r = 0; r < kScanRows; ++r) {
                if (!ok[r]) continue;
                int h = 0;
#pragma unroll
                for (int w = 0; w < W; ++w) h += __popc(qcode[w] ^ c[r].w[w]);
                const float cosine = __fdiv_rn(__fsub_rn(dimf, __fmul_rn(2.0f, (float)h)), dimf);
                const float dn = param[r];
                const float score = __fmaf_rn(-__fmul_rn(__fmul_rn(2.0f, qparam), dn), cosine, __fmaf_rn(dn, dn, __fmul_rn(qparam, qparam)));
                const uint64_t key = make_key(score, (uint32_t)rows[r]);
                if (key < thr) keys[atomicAdd(&s_cnt, 1)] = key;   // room for a whole step was checked above
            }
            __syncthreads();
        }
    }
    __syncthreads();
    sign_output(a, q, slice, keys, sign_finish(keys, spill, a.k, a.kp2, &s_cnt, &s_thr, &s_sel));
}

// Float states.  One CTA per (query, slice of probes); its probes are taken kProbeChunk at a time, their states' bytes and bounds laid
// out in shared memory together (a warp per state), and the chunk's rows are dealt to the warps in units of 64 of one list.
// A row first gets a bound: rough - slack <= exact score <= rough + slack, rough from the filter's dot product.  Rows whose
// lower bound is not above the cut wait, (bound, row, probe), in their warp's part of the queue.  The cut never is below the k-th
// smallest exact score: k waiting rows have upper bounds, lower + 2 x the largest slack seen, of at most it.  When a warp's part
// runs full the cut is moved down (a histogram of the bounds finds a value that k of them do not exceed) and what lies above it goes;
// only if that does not make room - many equal scores, or a k beyond the queue - the waiting rows are scored exactly, into the key
// buffer, whose k-th key is a cut too.  What still waits at the end, little more than k rows, gets the exact chain.
//
// Slack: with A = sum |state[d]| and delta = max |state| / 32,500, the filter's dot is within 1.875 dim delta of the true sum (above), and
// the exact chain too rounds: every partial sum is at most A in magnitude and each of its dim <= 256 roundings at most 2^-24 of it,
// less than 2^-15 A in all; a few more come from the multiplications by delta.  Taken: 2 dim delta + 2^-14 A on the dot and
// 2^-20 relative on the final multiply-adds.
//
// The earlier form scored rows from a table of partial sums (32 look-ups of 8 warp instructions per row and warp) and, its cut coming from
// exact keys alone, sent a third of all rows through the chain.  4,000 queries x 32 of 2,048 lists, 2M rows, k = 512: 1,556 -> 1,041 us.
constexpr int kProbeChunk = 32;
constexpr int kScanWarps = kScanThreads / 32;
template <int W> struct ProbeChunk { static constexpr int value = W > 4 ? kProbeChunk / 2 : kProbeChunk; };

struct SignProbe { int beg, end, probe; float delta2, offset, slack, norm_sq; };   // dot = delta2 x (sum of bytes) + offset
struct WarpBounds { float lo, hi, slack, kth; int n; };

template <int W>
__global__ void __launch_bounds__(kScanThreads, W > 4 ? 2 : 4) k_sign_scan_float(const SignScanArgs a) {
    constexpr int CHUNK = ProbeChunk<W>::value, DIM = 32 * W;
    extern __shared__ __align__(16) unsigned char s_raw[];
    uint64_t* keys = reinterpret_cast<uint64_t*>(s_raw);
    uint64_t* spill = keys + a.cap;                                              // k keys
    int8_t* s_bytes = reinterpret_cast<int8_t*>(spill + ((a.k + 1) & ~1));       // [CHUNK][2][DIM]: high and low bytes, in slot order
    float* q_low = reinterpret_cast<float*>(s_bytes + CHUNK * 2 * DIM);          // the waiting rows, a.seg per warp
    uint32_t* q_row = reinterpret_cast<uint32_t*>(q_low + kScanWarps * a.seg);
    uint16_t* q_probe = reinterpret_cast<uint16_t*>(q_row + kScanWarps * a.seg);
    __shared__ SignSelectScratch s_sel;
    __shared__ SignProbe s_probe[CHUNK];
    __shared__ WarpBounds s_bounds[kScanWarps];
    __shared__ int s_cnt;
    __shared__ unsigned long long s_thr;
    const int q = blockIdx.x / a.split, slice = blockIdx.x % a.split;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t = lane & 3, g = lane >> 2;
    const float dimf = (float)DIM;
    float* w_low = q_low + warp * a.seg;   // this warp's
    uint32_t* w_row = q_row + warp * a.seg;
    uint16_t* w_probe = q_probe + warp * a.seg;
    if (tid == 0) { s_cnt = 0; s_thr = KEY_MAX; }
    __syncthreads();
    int waiting = 0;            // rows in this warp's part
    float cut = __int_as_float(0x7f800000);   // the same in every thread
    float max_slack = 0.f, low_min = cut, low_max = -cut;   // over the rows this lane has queued

    // Moves the cut down and drops the waiting rows above it.  Called by all threads after a barrier.
    auto prune = [&]() {
        float lo = low_min, hi = low_max, slack = max_slack;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(kFull, lo, o)); hi = fmaxf(hi, __shfl_xor_sync(kFull, hi, o));
            slack = fmaxf(slack, __shfl_xor_sync(kFull, slack, o));
        }
        if (lane == 0) { WarpBounds& b = s_bounds[warp]; b.lo = lo; b.hi = hi; b.slack = slack; b.n = waiting; }
        s_sel.hist[tid] = 0;
        if (tid == 0) s_sel.bucket = -1;
        __syncthreads();
        int n = 0;
#pragma unroll
        for (int i = 0; i < kScanWarps; ++i) {
            const WarpBounds b = s_bounds[i];
            lo = fminf(lo, b.lo); hi = fmaxf(hi, b.hi); slack = fmaxf(slack, b.slack); n += b.n;
        }
        hi = fminf(hi, cut);   // of those that wait
        if (n < a.k) return;   // uniform
        const float scale = 255.0f / (hi - lo);   // no spread, or one beyond float: everything in bin 0
        auto bin = [&](float x) { return max(0, min(255, __float2int_rz((x - lo) * scale))); };
        for (int i = lane; i < waiting; i += 32) {
            const float x = w_low[i];
            if (fabsf(x) < __int_as_float(0x7f800000)) atomicAdd(&s_sel.hist[bin(x)], 1);
        }
        __syncthreads();
        const int c = s_sel.hist[tid];
        const int before = block_exclusive_scan(c, s_sel.warp_sums, nullptr);
        if (before < a.k && a.k <= before + c) s_sel.bucket = tid;
        __syncthreads();
        const int bucket = s_sel.bucket;
        if (bucket < 0) return;   // uniform; fewer than k numbers
        float kth = -__int_as_float(0x7f800000);
        for (int i = lane; i < waiting; i += 32) {
            const float x = w_low[i];
            if (fabsf(x) < __int_as_float(0x7f800000) && bin(x) <= bucket) kth = fmaxf(kth, x);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) kth = fmaxf(kth, __shfl_xor_sync(kFull, kth, o));
        if (lane == 0) s_bounds[warp].kth = kth;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kScanWarps; ++i) kth = fmaxf(kth, s_bounds[i].kth);
        cut = fminf(cut, kth + 2.0f * slack);
        int kept = 0;
        for (int i0 = 0; i0 < waiting; i0 += 32) {
            const int i = i0 + lane;
            const bool in = i < waiting;
            const float x = in ? w_low[i] : 0.f;
            const uint32_t row = in ? w_row[i] : 0u;
            const uint16_t pr = in ? w_probe[i] : (uint16_t)0;
            const bool keep = in && !(x > cut);
            const unsigned mask = __ballot_sync(kFull, keep);   // everyone has read before anyone writes, at or before i
            if (keep) {
                const int at = kept + __popc(mask & ((1u << lane) - 1u));
                w_low[at] = x; w_row[at] = row; w_probe[at] = pr;
            }
            kept += __popc(mask);
            __syncwarp();
        }
        waiting = kept;
    };

    // Exact scores of all waiting rows, up to 1,024 per round.  Called by all threads after a barrier.
    auto work_off = [&]() {
        if (lane == 0) s_bounds[warp].n = waiting;
        __syncthreads();
        int all = 0;
#pragma unroll
        for (int i = 0; i < kScanWarps; ++i) all += s_bounds[i].n;
        const bool wide = reinterpret_cast<uintptr_t>(a.states) % 16 == 0;
#pragma unroll 1
        for (int done = 0; done < all; done += kScanStep) {
            const int held = s_cnt;
            __syncthreads();
            if (held > a.cap - kScanStep) sign_compact(keys, spill, a.k, &s_cnt, &s_thr, &s_sel);   // uniform
            const unsigned long long thr = s_thr;
            CodeWords<W> c[kScanRows];
            float param[kScanRows], norm_sq[kScanRows], score[kScanRows];
            const float* state[kScanRows];
            uint32_t row[kScanRows];
            bool ok[kScanRows];
#pragma unroll
            for (int r = 0; r < kScanRows; ++r) {
                int at = done + kScanRows * tid + r;   // four consecutive rows per thread: whole warps work or rest
                ok[r] = at < all;
                row[r] = 0u; param[r] = 0.f; norm_sq[r] = 0.f; state[r] = a.states;
#pragma unroll
                for (int w = 0; w < W; ++w) c[r].w[w] = 0u;
                if (ok[r]) {
                    int part = 0;
                    while (at >= s_bounds[part].n) { at -= s_bounds[part].n; ++part; }
                    at += part * a.seg;
                    row[r] = q_row[at];
                    const long long st = (long long)q * a.nprobe + q_probe[at];
                    c[r] = load_code<W>(a.codes, row[r]);
                    param[r] = __ldg(a.row_params + row[r]);
                    norm_sq[r] = __ldg(a.norm_sq + st);
                    state[r] = a.states + (size_t)st * DIM;
                }
            }
            if (ok[0]) {
                if (wide) exact_float_scores<W, true>(c, param, state, norm_sq, score);
                else exact_float_scores<W, false>(c, param, state, norm_sq, score);
#pragma unroll
                for (int r = 0; r < kScanRows; ++r) {
                    if (!ok[r]) continue;
                    const uint64_t key = make_key(score[r], row[r]);
                    if (key < thr) keys[atomicAdd(&s_cnt, 1)] = key;   // room for a whole round was made above
                }
            }
            __syncthreads();
        }
        waiting = 0;
        if (s_thr != KEY_MAX) cut = fminf(cut, key_dist(s_thr));
    };

    const int probes = (a.nprobe - slice + a.split - 1) / a.split;   // of this slice
    const int last = (int)a.offsets[a.nlist] - 1;
#pragma unroll 1
    for (int c0 = 0; c0 < probes; c0 += CHUNK) {
        const int np = min(CHUNK, probes - c0);
        __syncthreads();
        for (int i = warp; i < np; i += kScanWarps) {
            const int p = slice + (c0 + i) * a.split;
            const long long st = (long long)q * a.nprobe + p;
            const int list = a.probes[st];
            if (list < 0 || list >= a.nlist) {   // warp-uniform
                if (lane == 0) { s_probe[i].beg = 0; s_probe[i].end = 0; }
                continue;
            }
            float x[W], abs_sum = 0.f, top = 0.f;   // abs_sum: rounded up a little
#pragma unroll
            for (int j = 0; j < W; ++j) { x[j] = __ldg(a.states + (size_t)st * DIM + lane + 32 * j); abs_sum += fabsf(x[j]); top = fmaxf(top, fabsf(x[j])); }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) { abs_sum += __shfl_xor_sync(kFull, abs_sum, o); top = fmaxf(top, __shfl_xor_sync(kFull, top, o)); }
            abs_sum *= 1.001f;
            const float delta = fmaxf(top, 1e-30f) * (1.0f / 32500.0f);   // never so small that the division leaves its range
            const float unit = delta * (float)(1 << (lane & 3));
            int part = 0;
            int8_t* out = s_bytes + i * 2 * DIM + 4 * (lane & 7) + (lane >> 3);   // slot order: the four bits of a byte position side by side
#pragma unroll
            for (int j = 0; j < W; ++j) {
                const int v = __float2int_rn(__fdividef(x[j], unit));
                const int lo = (int)(int8_t)(v & 255), hi = (int)(int8_t)((v - lo) >> 8);
                out[32 * j] = (int8_t)hi;
                out[32 * j + DIM] = (int8_t)lo;
                part += (256 * hi + lo) << (lane & 3);
            }
            part = __reduce_add_sync(kFull, part);
            if (lane == 0)
                s_probe[i] = SignProbe{(int)a.offsets[list], (int)a.offsets[list + 1], p, 2.0f * delta, -delta * (float)part,
                                       2.0f * (abs_sum * (1.0f / 16384.0f + 1.0f / 1048576.0f) + 2.0f * dimf * delta), __ldg(a.norm_sq + st)};
        }
        __syncthreads();
        const int units = lane < np ? (s_probe[lane < CHUNK ? lane : 0].end - s_probe[lane < CHUNK ? lane : 0].beg + kUnitRows - 1) / kUnitRows : 0;
        int upto = units;   // units of this lane's probe and those before it
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, upto, o);
            if (lane >= o) upto += v;
        }
        const int total = __shfl_sync(kFull, upto, 31);
#pragma unroll 1
        for (int u0 = 0; u0 < total; u0 += kStepUnits * kScanWarps) {
#pragma unroll 1
            for (int h = 0; h < kStepUnits; ++h) {
                const int u = u0 + h * kScanWarps + warp;
                if (u >= total) break;   // warp-uniform
                const int i = __popc(__ballot_sync(kFull, upto <= u));
                const SignProbe pr = s_probe[i];
                const int base = pr.beg + (u - __shfl_sync(kFull, upto - units, i)) * kUnitRows;
                const int mine = base + 16 * t + g;
                float param[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) param[r] = __ldg(a.row_params + min(mine + 8 * r, last));
                uint2 b[W];   // even columns: high bytes, odd ones: low bytes
                const uint2* col = reinterpret_cast<const uint2*>(s_bytes + (2 * i + (g & 1)) * DIM);
#pragma unroll
                for (int s = 0; s < W; ++s) b[s] = col[slot_word<W>(s, t) * 4 + slot_bit<W>(s, t) / 2];
                int dots[2];
                tile_dots<W>(a.codes, base, last, b, dots);
                float low[2], slack[2];
                bool wait[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float s = param[r];
                    const float base_score = __fmaf_rn(__fmul_rn(dimf, s), s, pr.norm_sq);
                    const float rough = __fmaf_rn(-2.0f * s, __fmaf_rn(pr.delta2, (float)dots[r], pr.offset), base_score);
                    slack[r] = fabsf(s) * pr.slack + fabsf(base_score) * (1.0f / 1048576.0f);
                    low[r] = rough - slack[r];
                    wait[r] = mine + 8 * r < pr.end && !(low[r] > cut);   // NaN waits too
                }
                if (!__any_sync(kFull, wait[0] || wait[1])) continue;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const unsigned mask = __ballot_sync(kFull, wait[r]);
                    if (wait[r]) {
                        const int at = waiting + __popc(mask & ((1u << lane) - 1u));   // room for two units was left
                        w_low[at] = low[r]; w_row[at] = (uint32_t)(mine + 8 * r); w_probe[at] = (uint16_t)pr.probe;
                        max_slack = fmaxf(max_slack, slack[r]); low_min = fminf(low_min, low[r]); low_max = fmaxf(low_max, low[r]);
                    }
                    waiting += __popc(mask);
                }
            }
            if (__syncthreads_or(waiting > a.seg - kStepUnits * kUnitRows)) {
                prune();
                if (__syncthreads_or(waiting > a.seg - kStepUnits * kUnitRows)) work_off();
            }
        }
    }
    __syncthreads();
    prune();
    __syncthreads();
    work_off();
    __syncthreads();
    sign_output(a, q, slice, keys, sign_finish(keys, spill, a.k, a.kp2, &s_cnt, &s_thr, &s_sel));
}

__global__ void __launch_bounds__(kScanThreads) k_sign_merge(const uint64_t* __restrict__ partial, int split, int k, int cap,
                                                             int* __restrict__ rows_out, float* __restrict__ dist_out) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    uint64_t* keys = reinterpret_cast<uint64_t*>(s_raw);
    const int q = blockIdx.x, n = split * k;
    for (int i = threadIdx.x; i < cap; i += blockDim.x) keys[i] = i < n ? partial[(size_t)q * n + i] : KEY_MAX;
    __syncthreads();
    block_bitonic_sort(keys, cap);
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        const uint64_t key = keys[i];
        rows_out[(size_t)q * k + i] = key == KEY_MAX ? -1 : (int)key_idx(key);
        if (dist_out) dist_out[(size_t)q * k + i] = key == KEY_MAX ? FLT_MAX : key_dist(key);
    }
}

int pow2_at_least(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

template <int J>
psb_status run_encode(const SignEncodeArgs& a, int sm_count, cudaStream_t s) {
    const long long ctas = std::min<long long>((a.n + 7) / 8, (long long)sm_count * 16);
    k_sign_encode<J><<<(unsigned)ctas, 256, 0, s>>>(a);
    PSB_LAUNCH_CHECK();
    count_launch();
    return PSB_OK;
}

template <int P>
psb_status run_encode_lane(const SignEncodeArgs& a, int sm_count, cudaStream_t s) {
    const long long ctas = std::min<long long>((a.n + kLaneEncThreads - 1) / kLaneEncThreads, (long long)sm_count * 8);
    k_sign_encode_lane<P><<<(unsigned)ctas, kLaneEncThreads, 0, s>>>(a);
    PSB_LAUNCH_CHECK();
    count_launch();
    return PSB_OK;
}

psb_status dispatch_encode(const SignEncodeArgs& args, int padded, int sm_count, cudaStream_t s) {
    if (args.n <= 0) return PSB_OK;
    SignEncodeArgs a = args;
    a.padded = padded;
    // one row per thread where the row fits the registers and its loads can be 16 (fp32) / 4 (u8) bytes wide
    const bool u8 = a.kind == 1 && a.elem_bytes == 1;
    const bool wide = a.dim % 4 == 0 && reinterpret_cast<uintptr_t>(a.rows) % (u8 ? 4 : 16) == 0 &&
                      (!a.centroids || reinterpret_cast<uintptr_t>(a.centroids) % 16 == 0) &&
                      (!a.rotated || reinterpret_cast<uintptr_t>(a.rotated) % 16 == 0);
    if (wide && padded <= 128) {
        switch (padded) {
            case 32: return run_encode_lane<32>(a, sm_count, s);
            case 64: return run_encode_lane<64>(a, sm_count, s);
            case 128: return run_encode_lane<128>(a, sm_count, s);
        }
    }
    switch (padded) {
        case 32: return run_encode<1>(a, sm_count, s);
        case 64: return run_encode<2>(a, sm_count, s);
        case 128: return run_encode<4>(a, sm_count, s);
        case 256: return run_encode<8>(a, sm_count, s);
    }
    return fail(PSB_INVALID_ARGUMENT, "padded_dim must be 32, 64, 128 or 256");
}

template <int W>
psb_status run_scan(int mode, SignScanArgs& a, cudaStream_t s) {
    size_t smem = sizeof(uint64_t) * ((size_t)a.cap + ((a.k + 1) & ~1));
    auto kernel = k_sign_scan_codes<W>;
    if (mode == 0) {
        kernel = k_sign_scan_float<W>;
        smem += (size_t)ProbeChunk<W>::value * 64 * W;
        // Room for k waiting rows and two full steps more, so that the bounds alone can move the cut; a k for which that does not fit
        // beside its key buffer (above 4,096) leaves the cut to the exact keys.
        const size_t per_row = kScanWarps * (sizeof(float) + sizeof(uint32_t) + sizeof(uint16_t));
        a.seg = ((a.k + 2 * kScanStep) / kScanWarps + 31) / 32 * 32;
        if (smem + a.seg * per_row > 222 * 1024) a.seg = 2 * kScanStep / kScanWarps;
        smem += a.seg * per_row;
    }
    PSB_TRY(prefer_max_shared(kernel));
    PSB_TRY(kernel_shared(reinterpret_cast<const void*>(kernel), smem));
    kernel<<<(unsigned)(a.nq * a.split), kScanThreads, smem, s>>>(a);
    PSB_LAUNCH_CHECK();
    count_launch();
    return PSB_OK;
}

psb_status dispatch_scan(int mode, SignScanArgs& a, cudaStream_t s) {
    switch (a.dim) {
        case 32: return run_scan<1>(mode, a, s);
        case 64: return run_scan<2>(mode, a, s);
        case 128: return run_scan<4>(mode, a, s);
        case 256: return run_scan<8>(mode, a, s);
    }
    return fail(PSB_INVALID_ARGUMENT, "padded_dim must be 32, 64, 128 or 256");
}

bool sign_shape_ok(int dim, int padded) {
    return dim > 0 && dim <= padded && (padded == 32 || padded == 64 || padded == 128 || padded == 256);
}

}  // namespace

int sign_padded_dim(int dim) {   // src/search/ivf_res_turboquant/ivf_res_turboquant_search.cu:24-29
    if (dim <= 0) return -1;
    int p = 32;
    while (p < dim) p <<= 1;
    return p > 256 ? -1 : p;
}

psb_status launch_sign_scale(int padded_dim, float* d_out, cudaStream_t s) {
    k_sign_scale<<<1, 1, 0, s>>>(padded_dim, d_out);
    PSB_LAUNCH_CHECK();
    count_launch();
    return PSB_OK;
}

psb_status launch_sign_rotate(const float* d_rows, long long n, int dim, int padded_dim, uint32_t seed, float* d_rotated,
                              uint32_t* d_codes, float* d_norms, float* d_norm_sq, int sm_count, cudaStream_t s) {
    if (!sign_shape_ok(dim, padded_dim)) return fail(PSB_INVALID_ARGUMENT, "sign codec: dim must be in 1..padded_dim, padded_dim 32, 64, 128 or 256");
    SignEncodeArgs a{};
    a.kind = 0; a.rows = d_rows; a.n = n; a.dim = dim; a.seed = seed;
    a.rotated = d_rotated; a.codes = d_codes; a.norms = d_norms; a.norm_sq = d_norm_sq;
    return dispatch_encode(a, padded_dim, sm_count, s);
}

psb_status launch_sign_encode_database(const void* d_rows, int elem_bytes, long long n, const float* d_centroids,
                                       const long long* d_offsets, int nlist, int dim, int padded_dim, uint32_t seed,
                                       long long row_offset, uint32_t* d_codes, float* d_scales, int sm_count, cudaStream_t s) {
    if (!sign_shape_ok(dim, padded_dim)) return fail(PSB_INVALID_ARGUMENT, "sign codec: dim must be in 1..padded_dim, padded_dim 32, 64, 128 or 256");
    SignEncodeArgs a{};
    a.kind = 1; a.rows = d_rows; a.elem_bytes = elem_bytes; a.n = n; a.centroids = d_centroids; a.offsets = d_offsets;
    a.nlist = nlist; a.dim = dim; a.seed = seed; a.row_offset = row_offset; a.codes = d_codes; a.norms = d_scales;
    return dispatch_encode(a, padded_dim, sm_count, s);
}

psb_status launch_sign_encode_queries(const float* d_queries, const float* d_centroids, const int* d_probes, int nq, int nprobe,
                                      int nlist, int dim, int padded_dim, uint32_t seed, float* d_states, float* d_norm_sq,
                                      uint32_t* d_state_codes, float* d_norms, int sm_count, cudaStream_t s) {
    if (!sign_shape_ok(dim, padded_dim)) return fail(PSB_INVALID_ARGUMENT, "sign codec: dim must be in 1..padded_dim, padded_dim 32, 64, 128 or 256");
    SignEncodeArgs a{};
    a.kind = 2; a.rows = d_queries; a.n = (long long)nq * nprobe; a.centroids = d_centroids; a.probes = d_probes;
    a.nlist = nlist; a.nprobe = nprobe; a.dim = dim; a.seed = seed;
    a.rotated = d_states; a.codes = d_state_codes; a.norms = d_norms; a.norm_sq = d_norm_sq;
    return dispatch_encode(a, padded_dim, sm_count, s);
}

// Few queries: the probes of one query go to several CTAs so that the grid covers the SMs twice over.
static int sign_split(int nq, int nprobe, int candidate_count, int sm_count) {
    int split = 1;
    if (nq < 2 * sm_count) split = std::min(nprobe, (2 * sm_count + nq - 1) / nq);
    return std::max(1, std::min(split, kMergeMaxKeys / pow2_at_least(candidate_count)));
}

size_t sign_partial_bytes(int nq, int nprobe, int candidate_count, int sm_count) {
    if (nq <= 0 || nprobe <= 0 || candidate_count <= 0 || candidate_count > kSignMaxCandidates) return 0;
    const int split = sign_split(nq, nprobe, candidate_count, sm_count);
    return split > 1 ? sizeof(uint64_t) * (size_t)nq * split * candidate_count : 0;
}

psb_status launch_sign_candidates(int mode, const float* d_states, const float* d_norm_sq, const uint32_t* d_state_codes,
                                  const float* d_norms, const uint32_t* d_codes, const float* d_row_params,
                                  const long long* d_offsets, int nlist, const int* d_probes, int nq, int nprobe, int padded_dim,
                                  int candidate_count, int* d_rows_out, float* d_dist_out, void* d_partial, int sm_count, cudaStream_t s) {
    if (!sign_shape_ok(padded_dim, padded_dim)) return fail(PSB_INVALID_ARGUMENT, "sign codec: padded_dim must be 32, 64, 128 or 256");
    if (nprobe > 65535) return fail(PSB_INVALID_ARGUMENT, "sign codec: at most 65,535 probes per query");
    if (candidate_count <= 0 || candidate_count > kSignMaxCandidates)
        return fail(PSB_INVALID_ARGUMENT, "sign codec: candidate_count must be in 1..8192");
    if (reinterpret_cast<uintptr_t>(d_codes) % 16) return fail(PSB_INVALID_ARGUMENT, "sign codec: the code array must be 16-byte aligned");
    if (nq <= 0) return PSB_OK;
    SignScanArgs a{};
    a.states = d_states; a.norm_sq = d_norm_sq; a.state_codes = d_state_codes; a.norms = d_norms;
    a.codes = d_codes; a.row_params = d_row_params; a.offsets = d_offsets; a.probes = d_probes;
    a.nlist = nlist; a.nq = nq; a.nprobe = nprobe; a.dim = padded_dim; a.k = candidate_count;
    const int kp2 = pow2_at_least(candidate_count);
    a.kp2 = kp2;
    a.cap = std::max(2 * kp2, 2 * kScanStep);   // a whole step always fits after a cut back to candidate_count
    const int split = sign_split(nq, nprobe, candidate_count, sm_count);
    a.split = split;
    a.rows_out = d_rows_out; a.dist_out = d_dist_out;
    uint64_t* partial = static_cast<uint64_t*>(d_partial);
    a.partial = split > 1 ? partial : nullptr;
    psb_status rc = dispatch_scan(mode, a, s);
    if (rc == PSB_OK && split > 1) {
        const int mcap = pow2_at_least(split * candidate_count);
        const size_t msmem = sizeof(uint64_t) * (size_t)mcap;
        cudaError_t e = cudaSuccess;
        rc = kernel_shared(reinterpret_cast<const void*>(k_sign_merge), msmem);
        if (rc == PSB_OK) {
            k_sign_merge<<<(unsigned)nq, kScanThreads, msmem, s>>>(partial, split, candidate_count, mcap, d_rows_out, d_dist_out);
            e = cudaGetLastError();
            count_launch();
        }
        if (e != cudaSuccess) rc = cuda_fail(e, "k_sign_merge", __FILE__, __LINE__);
    }
    return rc;
}

}  // namespace psb
