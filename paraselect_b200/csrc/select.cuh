// Block-wide selection of the k smallest (value, payload) keys of a row of values in memory.
#pragma once

#include "common.cuh"

namespace psb {
namespace sel {

constexpr int kMaxGroups = 2048;  // minima looked at
constexpr int kSegShared = 1024;  // probes whose segments the selections over lists keep in shared memory

// Entries the key buffer needs: a power of two that holds the keys gathered at the usual cut several times over.
inline int buffer_entries(int k) { return k <= 256 ? 1024 : (k <= 1024 ? 4096 : 8192); }
inline size_t shared_bytes(int k) { return (size_t)buffer_entries(k) * 8 + (size_t)kMaxGroups * 4; }

struct Words { unsigned int hist[256]; uint64_t prefix; unsigned int rank; int done, cnt; float cut; };

// The rank-th smallest of the words get(i, word) gives for i = 0..n-1 (false: none), most significant byte first; returns its rank
// among those equal to it.  At least `rank` words.  All threads of the block.
template <int kThreads, typename Get>
__device__ unsigned smallest_word(int n, unsigned rank, Get get, uint32_t* out, Words* w) {
    uint32_t prefix = 0, mask = 0;
    for (int shift = 24; shift >= 0; shift -= 8) {
        if (threadIdx.x < 256) w->hist[threadIdx.x] = 0;
        __syncthreads();
#pragma unroll 4
        for (int i = threadIdx.x; i < n; i += kThreads) {
            uint32_t word = 0;
            if (get(i, word) && (word & mask) == prefix) atomicAdd(&w->hist[(word >> shift) & 255u], 1u);
        }
        __syncthreads();
        if (threadIdx.x < 32) {   // eight bins a lane
            unsigned mine = 0;
            for (int j = 0; j < 8; ++j) mine += w->hist[threadIdx.x * 8 + j];
            unsigned upto = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const unsigned v = __shfl_up_sync(0xffffffffu, upto, o); if ((int)threadIdx.x >= o) upto += v; }
            unsigned before = upto - mine;
            if (before < rank && rank <= upto) {
                int j = 0;
                while (before + w->hist[threadIdx.x * 8 + j] < rank) before += w->hist[threadIdx.x * 8 + j++];
                w->prefix = prefix | (uint32_t)(threadIdx.x * 8 + j) << shift;
                w->rank = rank - before;
            }
        }
        __syncthreads();
        prefix = (uint32_t)w->prefix;
        rank = w->rank;
        mask |= 255u << shift;
        __syncthreads();
    }
    *out = prefix;
    return rank;
}

// A value with at least k of s_min[0..n-1] (infinite: none) at or below it and not many more, by bisection; infinity where fewer than k are finite.
// One warp; a share of R words at most in registers, or (R = 0) all read from shared memory in every round.  (A count by the whole block, with a
// barrier and one counter for its warps in every round, took four times as long.)
template <int R>
__device__ __forceinline__ float bound_of(const float* s_min, int n, int k) {
    const int lane = threadIdx.x & 31;
    const float inf = __int_as_float(0x7f800000);
    float v[R > 0 ? R : 1], lo = inf, hi = -inf;
    auto each = [&](auto&& f) {
        if constexpr (R > 0) {
#pragma unroll
            for (int r = 0; r < R; ++r) f(v[r]);
        } else {
            for (int i = lane; i < n; i += 32) f(s_min[i]);
        }
    };
    if constexpr (R > 0) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = r * 32 + lane < n ? s_min[r * 32 + lane] : inf;
    }
    each([&](float x) { lo = fminf(lo, x); if (x < inf) hi = fmaxf(hi, x); });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o)); hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o)); }
    auto count = [&](float at) {
        int c = 0;
        each([&](float x) { c += x <= at ? 1 : 0; });
        return (int)__reduce_add_sync(0xffffffffu, c);
    };
    if (!(lo < inf) || count(hi) < k) return inf;
    const int enough = k > 384 && k <= 512 ? k : k + (k >> 3);   // (there a few more make the sort one of 1,024: 200 blocks, 400 of 4,000 values 33 us, 28 so)
    for (int it = 0; it < 14; ++it) {
        const float mid = lo + 0.5f * (hi - lo);
        const int c = count(mid);
        if (c >= k) hi = mid; else lo = mid;
        if (c >= k && c <= enough) break;
    }
    return hi;
}

// Minima of every 32 values, left by the kernel that computed them (one warp each), bound a row's k-th smallest value as well as the minima
// of subsets do, and say which 32 values to look at again.
constexpr int kRun = 32;
constexpr int kRunQueries = 16;   // (they cost a large batch's scan more than they save its selection)
inline long long run_count(long long values) { return (values + kRun - 1) / kRun; }
// The warp's lanes hold the values of run r (+infinity: none).
__device__ __forceinline__ void store_run(float* __restrict__ runs, int r, float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) runs[r] = v;
}

// The first c keys of s_keys in ascending order, and nothing (KEY_MAX) in the places up to k.
template <int kThreads>
__device__ __forceinline__ void put_in_order(uint64_t* s_keys, int c, int k) {
    const int tid = threadIdx.x;
    if (c <= kThreads) {   // a key's place is the number of smaller ones
        const uint64_t mine = tid < c ? s_keys[tid] : KEY_MAX;
        int rank = 0;
        if ((tid & ~31) < c) {
#pragma unroll 4
            for (int j = 0; j < c; ++j) { const uint64_t o = s_keys[j]; rank += o < mine || (o == mine && j < tid) ? 1 : 0; }   // a key may occur twice
        }
        __syncthreads();
        if (tid < c) s_keys[rank] = mine;
        for (int i = c + tid; i < k; i += kThreads) s_keys[i] = KEY_MAX;
        __syncthreads();
    } else {
        const int np = next_pow2(c);
        for (int i = c + tid; i < np || i < k; i += kThreads) s_keys[i] = KEY_MAX;
        __syncthreads();
        block_bitonic_sort(s_keys, np);
    }
}

// Leaves the min(k, n) smallest keys (vals[i], payload(i)) of i = 0..n-1 at the front of s_keys, ascending, and returns their number.  s_keys
// [buffer], s_runs [kMaxGroups], one Words in shared memory; k <= buffer.  runs: the minima of every kRun values, or null.
// The k-th smallest of the minima of at least 2 k subsets of the values bounds the k-th smallest value from above.  Every thread takes the
// minima of a few strided subsets, and not much more than k values lie below that bound, whatever the order of the values; a second read
// gathers them, and they are put in order by rank or, above the block's size, by a bitonic sort.  With runs, the minima of these bound the k-th
// value first, and only runs below that bound are read: a run's values belong together - rows of one list - so the bound alone is a loose one.
// 18,750 distances, 20 wanted, four blocks of 1,024 threads: 12.6 us without runs and with payloads one by one -> 10.1; 14,300, 200 wanted, 333
// blocks of 256 (no runs) 32.6 -> 24; 256, 16 wanted, 1,000 blocks, which used to be ranked whole, 25 -> 4.8.
// A radix selection is left for the rows the bound does not serve: too many equal values, fewer than k comparable ones, or k above what the
// minima cover.
template <int kThreads, typename Payload>   // kThreads: the block's threads, 256 or more
__device__ int smallest(const float* __restrict__ vals, int n, int k, Payload payload, uint64_t* s_keys, int buffer, int* s_runs, Words* w,
                        const float* __restrict__ runs = nullptr) {
    constexpr int PER = kMaxGroups / kThreads;
    const int tid = threadIdx.x, lane = tid & 31;
    const float inf = __int_as_float(0x7f800000);
    const int keep = k < n ? k : n, nruns = (n + kRun - 1) / kRun;
    const int per = (2 * k + kThreads - 1) / kThreads;   // subsets per thread
    float* s_min = reinterpret_cast<float*>(s_keys);     // [kMaxGroups]: the keys come later
    auto bound = [&](int groups) {   // of s_min
        __syncthreads();
        if (tid < 32) {
            const float at = groups <= kThreads ? bound_of<kThreads / 32>(s_min, groups, k) : bound_of<0>(s_min, groups, k);
            if (lane == 0) w->cut = at;
        }
        __syncthreads();
        return w->cut;
    };
    if (tid == 0) { w->cnt = 0; w->done = 0; w->cut = inf; }
    bool some = false;      // only the runs of s_runs are looked at
    int looked = n;
    if (runs && nruns >= 2 * k && nruns <= kMaxGroups) {
        for (int r = tid; r < nruns; r += kThreads) s_min[r] = runs[r];
        const float at = bound(nruns);
        if (at < inf) {
            for (int r = tid; r < nruns; r += kThreads)
                if (s_min[r] <= at) s_runs[atomicAdd(&w->done, 1)] = r;
            __syncthreads();
            some = true;
            looked = w->done * kRun;
        }
    }
    // The bound pays with four values for each wanted; with fewer, where it halves the sort: it leaves k to 9/8 k where every value is a subset, else up to half as
    // many more.  Of 600 values 256 wanted, 1,900 blocks of 256: without 92 us, with it 59; of 1,024 900 31 with, 22 without.
    const bool worth = looked > 4 * k ? looked >= 96 : looked > 2 * kThreads && next_pow2(looked) > next_pow2(k + (per * kThreads >= looked ? k >> 3 : k >> 1));
    auto gather = [&](auto index) {   // index(e): the place of the e-th value looked at, n or more for none
        float cut = inf;
        if (worth && per <= PER) {
            if (per == 1) {
                float m = inf;
#pragma unroll 8
                for (int e = tid; e < looked; e += kThreads) { const int i = index(e); if (i < n) m = fminf(m, vals[i]); }
                s_min[tid] = m;
            } else {
                for (int g = 0; g < per; ++g) {
                    float m = inf;
#pragma unroll 4
                    for (int e = tid + g * kThreads; e < looked; e += per * kThreads) { const int i = index(e); if (i < n) m = fminf(m, vals[i]); }
                    s_min[g * kThreads + tid] = m;
                }
            }
            cut = bound(per * kThreads);
        } else {
            __syncthreads();
        }
        if (cut == inf && looked > buffer) return cut;
#pragma unroll 8
        for (int e = tid; e < looked; e += kThreads) {
            const int i = index(e);
            const float v = i < n ? vals[i] : inf;
            if (cut == inf ? i < n : v <= cut) {
                const int pos = atomicAdd(&w->cnt, 1);
                if (pos < buffer) s_keys[pos] = make_key(v, (uint32_t)i);
            }
        }
        return cut;
    };
    const float cut = some ? gather([&](int e) { return s_runs[e / kRun] * kRun + e % kRun; }) : gather([](int e) { return e; });
    __syncthreads();
    int c = w->cnt;
    // Payloads, which may be a search and two loads each, for all kept values at once.
    if (c >= keep && c <= buffer)
        for (int e = tid; e < c; e += kThreads) s_keys[e] = (s_keys[e] & ~0xffffffffull) | (uint32_t)payload((int)key_idx(s_keys[e]));
    __syncthreads();
    if (c < keep || c > buffer) {
        // The keep-th smallest value by radix over the values up to the cut, then all below it and of the equal ones those with the
        // smallest payloads.  Rows of one code have one distance, so this happens; payloads, a search each, are asked of the chosen only
        // (whole keys, eight passes with a payload per value: 980 us for one row of 62,500 in a batch that takes 110).
        const bool all = c < keep;
        auto taken = [&](float v) { return all || cut == inf || v <= cut; };
        if (tid == 0) { w->cnt = 0; w->done = 0; }
        __syncthreads();
        if (keep == n) {
            for (int i = tid; i < n; i += kThreads) s_keys[i] = make_key(vals[i], payload(i));
            c = n;
        } else {
            uint32_t value = 0;
            const unsigned rank = smallest_word<kThreads>(n, (unsigned)keep, [&](int i, uint32_t& word) {
                const float v = vals[i];
                word = (uint32_t)(make_key(v, 0u) >> 32);
                return taken(v);
            }, &value, w);
#pragma unroll 4
            for (int i = tid; i < n; i += kThreads) {
                const float v = vals[i];
                const uint32_t word = (uint32_t)(make_key(v, 0u) >> 32);
                if (word < value) { const int pos = atomicAdd(&w->cnt, 1); if (pos < buffer) s_keys[pos] = make_key(v, payload(i)); }
                else if (word == value) atomicAdd(&w->done, 1);
            }
            __syncthreads();
            uint32_t last = 0xffffffffu;   // the largest payload wanted of the equal ones
            if (w->cnt + w->done > buffer)
                smallest_word<kThreads>(n, rank, [&](int i, uint32_t& word) {
                    if ((uint32_t)(make_key(vals[i], 0u) >> 32) != value) return false;
                    word = (uint32_t)payload(i);
                    return true;
                }, &last, w);
            __syncthreads();
#pragma unroll 4
            for (int i = tid; i < n; i += kThreads) {
                const float v = vals[i];
                if ((uint32_t)(make_key(v, 0u) >> 32) != value) continue;
                const uint32_t x = (uint32_t)payload(i);
                if (x <= last) { const int pos = atomicAdd(&w->cnt, 1); if (pos < buffer) s_keys[pos] = make_key(v, x); }
            }
            __syncthreads();
            c = w->cnt < buffer ? w->cnt : buffer;
        }
        __syncthreads();
    }
    put_in_order<kThreads>(s_keys, c, k);
    return keep;
}

}  // namespace sel
}  // namespace psb
