// vpmc_sort.cu -- exclusive scan, stable LSD radix sort.
//
// Design: reduce-then-scan everywhere (no inter-block spin waits).  The radix
// sort is the classic three-kernel pass (tile digit histograms, one scan of the
// [digit][tile] count matrix, stable scatter); within a tile, ranks come from
// ballots over 32 consecutive keys, warp-private digit counters and a
// cross-warp prefix, so equal keys keep their input order.  A tile is put in
// order in shared memory and written as runs of equal digits: pairs stored one
// by one touch eight times the sectors.  (match.any for the ballots, and single
// stores, took 41 us a pass at 2.1 M pairs, this form 15 us.)  Stability is
// what makes the spatial hash bit-identical to the reference's sequential
// counting sort (src/cpu/hash.cpp:36-48).
#include "vpmc_blocksort.cuh"

namespace vpmc {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;   // 4096

constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
// keys a thread: 8 (tiles of 4096) from kSortBig keys on, below it 4, so that
// more SMs take part
constexpr long kSortBig = 1L << 20;
int sort_items(long n) { return n >= kSortBig ? 8 : 4; }
long sort_tiles(long n) { return (n + long(kSortThreads) * sort_items(n) - 1) / (long(kSortThreads) * sort_items(n)); }

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix, *total receives the block sum.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* warp_tot, uint32_t* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        uint32_t w = lane < nw ? warp_tot[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < nw) warp_tot[lane] = wi - w;
        if (lane == nw - 1) warp_tot[32] = wi;
    }
    __syncthreads();
    const uint32_t res = warp_tot[wid] + inc - v;
    *total = warp_tot[32];
    __syncthreads();
    return res;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(const uint32_t* __restrict__ in, long n,
                                                              uint32_t* __restrict__ sums) {
    __shared__ uint32_t wt[33];
    const long base = long(blockIdx.x) * kScanTile;
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const long e = base + long(i) * kScanThreads + threadIdx.x;
        if (e < n) s += in[e];
    }
    uint32_t tot;
    (void)block_exclusive(s, wt, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const uint32_t* in, uint32_t* out, long n,
                                                             const uint32_t* __restrict__ offs,
                                                             int write_total) {
    __shared__ uint32_t wt[33];
    const long base = long(blockIdx.x) * kScanTile + long(threadIdx.x) * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const long e = base + i;
        v[i] = e < n ? in[e] : 0u;
        s += v[i];
    }
    uint32_t tot;
    uint32_t run = block_exclusive(s, wt, &tot) + (offs ? offs[blockIdx.x] : 0u);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const long e = base + i;
        if (e < n) out[e] = run;
        run += v[i];
        if (write_total && e == n - 1) out[n] = run;
    }
}

// Up to kSmallScan elements by one CTA of 1024 threads, in place of the three
// launches of the tiled scan (each 3 us and more).  A warp takes a contiguous part,
// in coalesced rows of 32 (a contiguous part per thread touches a sector per
// element: 32,768 elements took 37 us that way, 9 us this way).
constexpr int kSmallScan = 32768;

__global__ void __launch_bounds__(1024) k_scan_small(const uint32_t* in, uint32_t* out, int n, int write_total) {
    __shared__ uint32_t s_warp[32];
    constexpr int kRows = kSmallScan / 1024;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int rows = (n + 1023) / 1024, base = w * rows * 32 + lane;
    uint32_t v[kRows], s = 0;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        v[r] = r < rows && base + r * 32 < n ? in[base + r * 32] : 0u;
        s += v[r];
    }
    s = __reduce_add_sync(0xffffffffu, s);
    if (lane == 0) s_warp[w] = s;
    __syncthreads();
    if (w == 0) {
        const uint32_t t = s_warp[lane];
        uint32_t inc = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        s_warp[lane] = inc - t;
        if (lane == 31 && write_total) out[n] = inc;
    }
    __syncthreads();
    uint32_t run = s_warp[w];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        if (r >= rows) break;
        uint32_t inc = v[r];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (base + r * 32 < n) out[base + r * 32] = run + inc - v[r];
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
}

template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads) k_radix_upsweep(const uint32_t* __restrict__ keys, long n,
                                                                int shift, uint32_t mask,
                                                                uint32_t* __restrict__ counts, int ntiles) {
    __shared__ uint32_t hist[256];
    if (threadIdx.x < 256) hist[threadIdx.x] = 0;
    const long base = long(blockIdx.x) * (kSortThreads * ITEMS);
    uint32_t k[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const long e = base + long(i) * kSortThreads + threadIdx.x;
        k[i] = e < n ? keys[e] : 0u;
    }
    __syncthreads();
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const bool valid = base + long(i) * kSortThreads + threadIdx.x < n;
        const uint32_t d = (k[i] >> shift) & mask;
        const uint32_t peers = digit_peers(d, valid, __popc(mask));
        if (valid && (peers & lt) == 0u) atomicAdd(&hist[d], uint32_t(__popc(peers)));
    }
    __syncthreads();
    if (threadIdx.x <= mask) counts[long(threadIdx.x) * ntiles + blockIdx.x] = hist[threadIdx.x];
}

template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads) k_radix_downsweep(
    const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
    uint32_t* __restrict__ vout, long n, int shift, uint32_t mask, const uint32_t* __restrict__ offs,
    int ntiles) {
    constexpr int kTile = kSortThreads * ITEMS;
    __shared__ __align__(4) uint16_t wh[kSortWarps][256];   // counts and places inside the tile (<= 4096)
    __shared__ uint32_t sk[kTile], sv[kTile];
    __shared__ uint32_t goff[256];   // global place of a digit's first key, less its place in the tile
    __shared__ uint32_t wt[33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long t0 = long(blockIdx.x) * kTile, base = t0 + long(w) * (32 * ITEMS);
    uint32_t k[ITEMS], v[ITEMS], lr[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const long e = base + long(r) * 32 + lane;
        k[r] = e < n ? kin[e] : 0u;
        v[r] = e < n ? (vin ? vin[e] : uint32_t(e)) : 0u;
    }
    for (int i = threadIdx.x; i < kSortWarps * 128; i += kSortThreads) reinterpret_cast<uint32_t*>(&wh[0][0])[i] = 0;
    __syncthreads();
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const bool valid = base + long(r) * 32 + lane < n;
        const uint32_t d = (k[r] >> shift) & mask;
        const uint32_t peers = digit_peers(d, valid, __popc(mask));
        const uint32_t rank = __popc(peers & lt);
        const uint32_t b = valid ? wh[w][d] : 0u;
        __syncwarp();
        if (valid && rank == 0) wh[w][d] = uint16_t(b + __popc(peers));
        __syncwarp();
        lr[r] = b + rank;
    }
    __syncthreads();
    // per digit: the warps' first places inside the tile, and the tile's place in the output
    uint32_t c = 0;
    if (threadIdx.x <= mask)
#pragma unroll
        for (int q = 0; q < kSortWarps; ++q) c += wh[q][threadIdx.x];
    uint32_t tot;
    uint32_t run = block_exclusive(c, wt, &tot);
    if (threadIdx.x <= mask) {
        goff[threadIdx.x] = offs[long(threadIdx.x) * ntiles + blockIdx.x] - run;
#pragma unroll
        for (int q = 0; q < kSortWarps; ++q) {
            const uint32_t t = wh[q][threadIdx.x];
            wh[q][threadIdx.x] = uint16_t(run);
            run += t;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        if (base + long(r) * 32 + lane >= n) continue;
        const uint32_t p = wh[w][(k[r] >> shift) & mask] + lr[r];
        sk[p] = k[r];
        sv[p] = v[r];
    }
    __syncthreads();
    const int cnt = int(min(long(kTile), n - t0));
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const int i = r * kSortThreads + int(threadIdx.x);
        if (i >= cnt) break;
        const uint32_t key = sk[i];
        const uint32_t p = goff[(key >> shift) & mask] + uint32_t(i);
        kout[p] = key;
        vout[p] = sv[i];
    }
}

template <int ITEMS>
int radix_pass(vpmc_context* ctx, const uint32_t* kc, const uint32_t* vc, uint32_t* ko, uint32_t* vo, long n, int shift,
               uint32_t mask, const RadixScratch& rs) {
    const int ntiles = int(sort_tiles(n));
    VPMC_LAUNCH(k_radix_upsweep<ITEMS>, unsigned(ntiles), kSortThreads, 0, ctx->stream, kc, n, shift, mask, rs.counts,
                ntiles);
    VPMC_TRY(exclusive_scan(ctx, rs.counts, rs.counts, long(mask + 1) * ntiles, rs.scan_tmp, false));
    VPMC_LAUNCH(k_radix_downsweep<ITEMS>, unsigned(ntiles), kSortThreads, 0, ctx->stream, kc, vc, ko, vo, n, shift, mask,
                rs.counts, ntiles);
    return VPMC_OK;
}

}  // namespace

size_t scan_tmp_elems(long n) {
    const long nb = (n + kScanTile - 1) / kScanTile;
    if (nb <= 1) return 0;
    return size_t(2 * nb) + scan_tmp_elems(nb) + 64;
}

int exclusive_scan(vpmc_context* ctx, const uint32_t* in, uint32_t* out, long n, uint32_t* tmp,
                   bool write_total) {
    if (n <= 0) {
        if (write_total) VPMC_CUDA(cudaMemsetAsync(out, 0, sizeof(uint32_t), ctx->stream));
        return VPMC_OK;
    }
    if (n <= kSmallScan) {
        VPMC_LAUNCH(k_scan_small, 1, 1024, 0, ctx->stream, in, out, int(n), write_total ? 1 : 0);
        return VPMC_OK;
    }
    const long nb = (n + kScanTile - 1) / kScanTile;
    uint32_t* sums = tmp;
    uint32_t* offs = tmp + nb;
    VPMC_LAUNCH(k_scan_reduce, unsigned(nb), kScanThreads, 0, ctx->stream, in, n, sums);
    VPMC_TRY(exclusive_scan(ctx, sums, offs, nb, tmp + 2 * nb, false));
    VPMC_LAUNCH(k_scan_apply, unsigned(nb), kScanThreads, 0, ctx->stream, in, out, n, offs,
                write_total ? 1 : 0);
    return VPMC_OK;
}

size_t radix_counts_elems(long n) { return size_t(256) * size_t(n < 1 ? 1 : sort_tiles(n)); }

void carve_radix(Carver& c, long n, RadixScratch* rs) {
    const size_t m = size_t(n < 1 ? 1 : n);
    rs->kbuf[0] = c.take<uint32_t>(m);
    rs->kbuf[1] = c.take<uint32_t>(m);
    rs->vbuf[0] = c.take<uint32_t>(m);
    rs->vbuf[1] = c.take<uint32_t>(m);
    const size_t ce = radix_counts_elems(n);
    rs->counts = c.take<uint32_t>(ce);
    rs->scan_tmp = c.take<uint32_t>(scan_tmp_elems(long(ce)) + 1);
}

int radix_sort(vpmc_context* ctx, const uint32_t* keys_in, const uint32_t* vals_in, long n, int key_bits,
               const RadixScratch& rs, uint32_t** keys_out, uint32_t** vals_out) {
    if (key_bits < 1) key_bits = 1;
    if (key_bits > 32) return VPMC_ERR_INVALID;
    const int passes = (key_bits + 7) / 8;
    const int dbits = (key_bits + passes - 1) / passes;
    const uint32_t mask = (dbits >= 32) ? 0xffffffffu : ((1u << dbits) - 1u);
    const uint32_t* kc = keys_in;
    const uint32_t* vc = vals_in;
    *keys_out = rs.kbuf[0];
    *vals_out = rs.vbuf[0];
    if (n <= 0) return VPMC_OK;
    for (int p = 0; p < passes; ++p) {
        const int shift = p * dbits;
        uint32_t* ko = rs.kbuf[p & 1];
        uint32_t* vo = rs.vbuf[p & 1];
        if (sort_items(n) == 8) VPMC_TRY(radix_pass<8>(ctx, kc, vc, ko, vo, n, shift, mask, rs));
        else VPMC_TRY(radix_pass<4>(ctx, kc, vc, ko, vo, n, shift, mask, rs));
        kc = ko;
        vc = vo;
    }
    *keys_out = const_cast<uint32_t*>(kc);
    *vals_out = const_cast<uint32_t*>(vc);
    return VPMC_OK;
}

}  // namespace vpmc
