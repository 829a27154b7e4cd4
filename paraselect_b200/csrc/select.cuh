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

// Leaves the min(k, n) smallest keys (vals[i], payload(i)) of i = 0..n-1 at the front of s_keys, ascending, and returns their number.  s_keys [buffer], s_min [kMaxGroups], one Words in shared memory; k <= buffer.
//
// Reads the values twice.  First every thread takes the minima of a few of its strided subsets; the k-th smallest of all these
// minima - there are at least 2 k of them - bounds the k-th smallest value from above, and not much more than k values lie below
// it.  One warp finds it by bisection (14 rounds or until exactly k lie below; a little high does no harm).  Then the values up to
// that cut are gathered and put in order by rank or, above 256, by a bitonic sort.  A radix selection over the whole keys
// (up to eight passes with a histogram each, 12 us for 1,024 values and one row) is left for the rows the cut does not serve: too
// many equal values, fewer than k comparable ones, or k above what the group minima cover.
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
    if (c < keep || c > buffer) {   // radix selection over the whole keys, most significant byte first
        if (tid == 0) { w->prefix = 0; w->rank = (unsigned)keep; w->done = keep == n ? 1 : 0; w->cnt = 0; }
        uint64_t mask = 0;
        __syncthreads();
        for (int pass = 7; pass >= 0; --pass) {
            const int shift = pass * 8;
            if (tid < 256) w->hist[tid] = 0;
            __syncthreads();
            if (w->done) break;
            const uint64_t prefix = w->prefix;
            for (int i = tid; i < n; i += kThreads) {
                const uint64_t key = make_key(vals[i], payload(i));
                if ((key & mask) == prefix) atomicAdd(&w->hist[(key >> shift) & 255], 1u);
            }
            __syncthreads();
            if (tid == 0) {
                unsigned cum = 0;
                const unsigned rank = w->rank;
                for (int b = 0; b < 256; ++b) {
                    const unsigned h = w->hist[b];
                    if (cum + h >= rank) {
                        w->prefix = prefix | ((uint64_t)b << shift);
                        w->rank = rank - cum;
                        if (h == rank - cum) w->done = 1;  // the whole bucket is selected
                        break;
                    }
                    cum += h;
                }
            }
            mask |= 255ull << shift;
            __syncthreads();
        }
        __syncthreads();
        const uint64_t most = keep == n ? KEY_MAX : (w->prefix | ~mask);   // keys <= most are exactly the smallest
        for (int i = tid; i < n; i += kThreads) {
            const uint64_t key = make_key(vals[i], payload(i));
            if (key <= most) { const int pos = atomicAdd(&w->cnt, 1); if (pos < buffer) s_keys[pos] = key; }
        }
        __syncthreads();
        c = w->cnt;
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
