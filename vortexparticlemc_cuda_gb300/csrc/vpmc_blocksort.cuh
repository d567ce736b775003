// vpmc_blocksort.cuh -- stable sort of a small set of keys inside one CTA.
//
// A sort of a few thousand keys through global memory is a dozen launches of one
// or a few CTAs each, 3 us and more apiece.  Here one CTA counts the keys in
// shared memory, scans the counts (which are the keys' first places), places the
// indices and puts each key's few members in index order.  A set with a crowded
// key (more than kCrowd members, whose ordering would be quadratic) takes LSD
// radix passes over single words (key << index bits) | index instead.
#pragma once

#include "vpmc_internal.cuh"

namespace vpmc {

constexpr int kSmallThreads = 1024;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr long kSmallN = 16384;            // two word buffers of 64 KB
constexpr int kCrowd = 64;
constexpr size_t kSmallSmem = 224 * 1024;

// 16-bit counters of nk keys, two a word, one word of padding in 33
inline size_t small_count_words(long nk) { return (size_t(nk) + 2) / 2 + (size_t(nk) + 2) / 64 + 2; }
inline size_t small_sort_smem(long n, long nk) {
    // radix: words in flight, the per-(digit, warp) counters of an 8-bit pass, the ranks
    const size_t radix = (2 * size_t(n) + 256 * (kSmallWarps + 1)) * sizeof(uint32_t) + 2 * size_t(n) + 16;
    const size_t count = 4 * size_t(n) + 4 * small_count_words(nk) + 2 * size_t(n) + 16;
    return radix > count ? radix : count;
}
inline bool small_sort_fits(long n, long nk) {
    return n > 0 && n <= kSmallN && bits_for(uint64_t(n)) + bits_for(uint64_t(nk)) <= 32 && small_sort_smem(n, nk) <= kSmallSmem;
}

#ifdef __CUDACC__
// The valid lanes of the warp whose digit of `bits` <= 8 bits equals this lane's, by
// a ballot a bit: match.any costs several times the six to eight ballots.
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, bool valid, int bits) {
    uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll 4
    for (int b = 0; b < bits; ++b) {
        const bool set = (d >> b) & 1u;
        const uint32_t on = __ballot_sync(0xffffffffu, set);
        peers &= set ? on : ~on;
    }
    return peers;
}

// One radix pass over the digit of `bits` bits at `shift`, from `in` to `out`;
// cnt: 256 x 33 words, rk: n ranks.  Each warp owns a contiguous part of the
// input.
static __device__ __noinline__ void small_radix_pass(const uint32_t* in, uint32_t* out, int n, int shift, int bits,
                                              uint32_t* cnt, uint16_t* rk) {
    const int D = 1 << bits;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int i = tid; i < D * (kSmallWarps + 1); i += kSmallThreads) cnt[i] = 0u;
    __syncthreads();
    const int per = ((n + kSmallThreads - 1) / kSmallThreads) * 32;   // words a warp
    const int e0 = w * per, e1 = e0 + per;
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
#pragma unroll 1
    for (int e = e0 + lane; e < e1; e += 32) {
        const bool valid = e < n;
        const uint32_t d = valid ? (in[e] >> shift) & uint32_t(D - 1) : 0u;
        const uint32_t peers = digit_peers(d, valid, bits), before = __popc(peers & lt);
        uint32_t* c = cnt + d * (kSmallWarps + 1) + w;
        const uint32_t base = *c;
        __syncwarp();
        if (valid) {
            if (before == 0u) *c = base + __popc(peers);
            rk[e] = uint16_t(base + before);
        }
        __syncwarp();
    }
    __syncthreads();
    // exclusive scan over (digit, warp): warp w takes the digits w, w + 32, ... (32
    // counters each), then the digits' totals are scanned
    __shared__ uint32_t s_dig[256];
#pragma unroll 1
    for (int d = w; d < D; d += kSmallWarps) {
        const uint32_t v = cnt[d * (kSmallWarps + 1) + lane];
        uint32_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        cnt[d * (kSmallWarps + 1) + lane] = inc - v;
        if (lane == 31) s_dig[d] = inc;
    }
    __syncthreads();
    if (w == 0) {
        uint32_t run = 0u;
#pragma unroll 1
        for (int d0 = 0; d0 < D; d0 += 32) {
            const uint32_t v = d0 + lane < D ? s_dig[d0 + lane] : 0u;
            uint32_t inc = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += t;
            }
            if (d0 + lane < D) s_dig[d0 + lane] = run + inc - v;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int e = e0 + lane; e < e1 && e < n; e += 32) {
        const uint32_t k = in[e], d = (k >> shift) & uint32_t(D - 1);
        out[s_dig[d] + cnt[d * (kSmallWarps + 1) + w] + rk[e]] = k;
    }
    __syncthreads();
}

// The n keys (< nk) in buf[0..n) sorted stably: perm[slot] = index, start[k] = the
// first slot of key k for k < nk.  buf: small_sort_smem(n, nk) bytes.
__device__ __forceinline__ int count_word(uint32_t k) {
    const uint32_t w = k >> 1;
    return int(w + (w >> 5));   // 32 words and one of padding: a thread's run of words starts in its own bank
}
__device__ __forceinline__ void small_sort(uint32_t* buf, int n, int nk, int ibits, uint32_t* __restrict__ perm,
                                           uint32_t* __restrict__ start) {
    __shared__ uint32_t s_warp[kSmallWarps];
    __shared__ int s_crowd;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    uint32_t* key = buf;
    uint32_t* cnt = buf + n;
    const int words = nk / 2 + 1;                       // counter words in use
    const int padded = words + (words >> 5) + 1;
    uint16_t* order = reinterpret_cast<uint16_t*>(cnt + padded);
    const uint16_t* cnt16 = reinterpret_cast<const uint16_t*>(cnt);
    for (int i = tid; i < padded; i += kSmallThreads) cnt[i] = 0u;
    if (tid == 0) s_crowd = 0;
    __syncthreads();
    uint32_t most = 0u;
    for (int i = tid; i < n; i += kSmallThreads) {
        const uint32_t k = key[i], sh = (k & 1u) * 16u;
        most = max(most, (atomicAdd(&cnt[count_word(k)], 1u << sh) >> sh) & 0xffffu);
    }
    if (most >= uint32_t(kCrowd)) s_crowd = 1;
    __syncthreads();
    const bool crowd = s_crowd != 0;
    // exclusive scan of the counters: each thread a run of whole words
    const int per = (words + kSmallThreads - 1) / kSmallThreads, w0 = min(words, tid * per), w1 = min(words, w0 + per);
    uint32_t sum = 0u;
    for (int i = w0; i < w1; ++i) {
        const uint32_t v = cnt[i + (i >> 5)];
        sum += (v & 0xffffu) + (v >> 16);
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    if (w == 0) {
        uint32_t t = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        s_warp[lane] = t;
    }
    __syncthreads();
    uint32_t run = inc - sum + (w > 0 ? s_warp[w - 1] : 0u);
    for (int i = w0; i < w1; ++i) {
        const uint32_t v = cnt[i + (i >> 5)], a = v & 0xffffu;
        cnt[i + (i >> 5)] = run | ((run + a) << 16);
        run += a + (v >> 16);
    }
    __syncthreads();
    for (int k = tid; k < nk; k += kSmallThreads) start[k] = cnt16[2 * count_word(k) + (k & 1)];
    if (!crowd) {
        __syncthreads();   // the starts are out before the places move them
        for (int i = tid; i < n; i += kSmallThreads) {
            const uint32_t k = key[i], sh = (k & 1u) * 16u;
            order[(atomicAdd(&cnt[count_word(k)], 1u << sh) >> sh) & 0xffffu] = uint16_t(i);
        }
        __syncthreads();
        // each counter now holds its key's end, the one before it its first place
        for (int s = tid; s < n; s += kSmallThreads) {
            const uint32_t i = order[s], k = key[i];
            const int lo = k ? cnt16[2 * count_word(k - 1u) + ((k - 1u) & 1u)] : 0, hi = cnt16[2 * count_word(k) + (k & 1u)];
            int r = lo;
            for (int j = lo; j < hi; ++j) r += order[j] < i ? 1 : 0;
            perm[r] = i;
        }
        return;
    }
    __syncthreads();
    const int kbits = 32 - __clz(nk > 1 ? nk - 1 : 1);
    const int passes = (kbits + 7) / 8, dbits = (kbits + passes - 1) / passes;
    uint32_t *a = buf, *b = buf + n, *dig = buf + 2 * n;
    uint16_t* rk = reinterpret_cast<uint16_t*>(dig + 256 * (kSmallWarps + 1));
    for (int i = tid; i < n; i += kSmallThreads) a[i] = (a[i] << ibits) | uint32_t(i);
    __syncthreads();
#pragma unroll 1
    for (int p = 0; p < passes; ++p) {
        // the last pass's digit may reach past the key: those bits are zero
        small_radix_pass(a, b, n, ibits + p * dbits, dbits, dig, rk);
        uint32_t* t = a;
        a = b;
        b = t;
    }
    for (int i = tid; i < n; i += kSmallThreads) perm[i] = a[i] & ((1u << ibits) - 1u);
}

// The first of the n ascending keys that is >= k.
__device__ __forceinline__ uint32_t lower_bound_key(const uint32_t* __restrict__ keys, uint32_t n, uint32_t k) {
    uint32_t lo = 0u, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (keys[mid] < k) lo = mid + 1u; else hi = mid;
    }
    return lo;
}
#endif

}  // namespace vpmc
