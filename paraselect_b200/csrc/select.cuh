// Block-wide selection of the k smallest (value, payload) keys of a row of values in memory.
#pragma once

#include "common.cuh"

namespace psb {
namespace sel {

constexpr int kMaxGroups = 2048;  // group minima

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

// Leaves the min(k, n) smallest keys (vals[i], payload(i)) of i = 0..n-1 at the front of s_keys, ascending, and returns their number.  s_keys [buffer], s_min [kMaxGroups], one Words in shared memory; k <= buffer.
//
// Reads the values twice.  First every thread takes the minima of a few of its strided subsets; the k-th smallest of all these
// minima - there are at least 2 k of them - bounds the k-th smallest value from above, and not much more than k values lie below
// it.  One warp finds it by bisection (14 rounds or until exactly k lie below; a little high does no harm).  Then the values up to
// that cut are gathered and put in order by rank or, above 256, by a bitonic sort.  A radix selection is left for
// the rows the cut does not serve: too many equal values, fewer than k comparable ones, or k above what the group minima cover.
template <int kThreads, typename Payload>   // kThreads: the block's threads, 256 or more
__device__ int smallest(const float* __restrict__ vals, int n, int k, Payload payload, uint64_t* s_keys, int buffer, float* s_min, Words* w) {
    const int tid = threadIdx.x, lane = tid & 31;
    const float inf = __int_as_float(0x7f800000);
    const int keep = k < n ? k : n;
    int per = (2 * k + kThreads - 1) / kThreads;   // subsets per thread
    if (tid == 0) { w->cnt = 0; w->cut = inf; }
    if (n > 2 * kThreads && per <= kMaxGroups / kThreads) {
        if (per == 1) {
            float m = inf;
#pragma unroll 8
            for (int i = tid; i < n; i += kThreads) m = fminf(m, vals[i]);
            s_min[tid] = m;
        } else {
            for (int g = 0; g < per; ++g) {
                float m = inf;
#pragma unroll 4
                for (int i = tid + g * kThreads; i < n; i += per * kThreads) m = fminf(m, vals[i]);
                s_min[g * kThreads + tid] = m;
            }
        }
        __syncthreads();
        if (tid < 32) {
            const int groups = per * kThreads;
            float mn = inf, mx = -inf;
            for (int i = lane; i < groups; i += 32) { const float v = s_min[i]; mn = fminf(mn, v); if (v < inf) mx = fmaxf(mx, v); }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) { mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o)); mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o)); }
            float lo = mn, hi = mx;
            int c = groups;
            for (int it = 0; it < 14 && mn < inf; ++it) {
                const float mid = lo + 0.5f * (hi - lo);
                c = 0;
                for (int i = lane; i < groups; i += 32) c += s_min[i] <= mid ? 1 : 0;
                c = __reduce_add_sync(0xffffffffu, c);
                if (c >= k) hi = mid; else lo = mid;
                if (c == k) break;
            }
            c = 0;
            for (int i = lane; i < groups; i += 32) c += s_min[i] <= hi ? 1 : 0;
            c = __reduce_add_sync(0xffffffffu, c);
            if (lane == 0) w->cut = c >= k && mn < inf ? hi : inf;
        }
    }
    __syncthreads();
    const float cut = w->cut;
    if (cut < inf || n <= buffer) {
#pragma unroll 8
        for (int i = tid; i < n; i += kThreads) {
            const float v = vals[i];
            if (cut == inf || v <= cut) {
                const int pos = atomicAdd(&w->cnt, 1);
                if (pos < buffer) s_keys[pos] = make_key(v, payload(i));
            }
        }
    }
    __syncthreads();
    int c = w->cnt;
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
    return keep;
}

}  // namespace sel
}  // namespace psb
