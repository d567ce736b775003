// vpmc_grid.cu -- evaluation grid: planning, stable build, query binning and
// the field-evaluation kernel (the hot loop of queries, MIS samples and SpMV).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "vpmc_blocksort.cuh"
#include "vpmc_grid.cuh"
#include "vpmc_wide.cuh"

namespace vpmc {

namespace {

constexpr int kEvalThreads = 32;
constexpr int kMaxK = 8;
constexpr int kMaxPieces = 2 * (2 * kMaxK + 1);
constexpr int kCandCap = 208;                  // candidates staged per batch (6.5 KB: 24 one-warp CTAs fill an SM's shared memory)
constexpr uint32_t kWaitLimit = VPMC_WAIT_LIMIT_DEFAULT;   // drain wait of an aborted CTA (always the full cap)

__device__ __forceinline__ int inst_of_particle(const GridInst* inst, int n_inst, long i) {
    int lo = 0, hi = n_inst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (inst[mid].p_begin <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ int inst_of_bin(const GridInst* inst, int n_inst, uint32_t b) {
    int lo = 0, hi = n_inst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (uint32_t(inst[mid].bin_base) <= b) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Wrap into [0, L) the way the reference does (p - floor(p/L)*L).
__device__ __forceinline__ float wrapf(float p, float L) { return p - floorf(p / L) * L; }

// Candidate key of particle i: (bin, sub-row), or nbins rows when it is in no set.
__device__ __forceinline__ uint32_t grid_key(const float2* __restrict__ pos, const float* __restrict__ omega, long i,
                                             const GridInst* __restrict__ inst, int n_inst, int set_mode,
                                             uint32_t nbins, int rows) {
    float2 p = pos[i];
    const float w = omega ? omega[i] : 1.f;
    const GridInst& G = inst[inst_of_particle(inst, n_inst, i)];
    int set = 0;
    bool use = true;
    switch (set_mode) {
        case SET_SIGN_SPLIT: set = w > 0.f ? 0 : 1; use = w != 0.f; break;
        case SET_POS_ONLY: use = w > 0.f; break;
        case SET_NEG_ONLY: use = w < 0.f; break;
        default: break;
    }
    if (!use) return nbins * uint32_t(rows);
    if (G.periodic) { p.x = wrapf(p.x, G.Lx); p.y = wrapf(p.y, G.Ly); }
    const int cx = min(max(floor_int(p.x * G.inv_sx), 0), G.gx - 1);
    const int cy = min(max(floor_int(p.y * G.inv_sy), 0), G.gy - 1);
    const uint32_t bin = uint32_t(G.bin_base) + uint32_t(set) * uint32_t(G.gx * G.gy) + uint32_t(cx * G.gy + cy);
    // sub-row of the cell (nested: clamped into the cell's own rows)
    const int r = min(max(floor_int(p.y * G.inv_sy * float(rows)) - cy * rows, 0), rows - 1);
    return bin * uint32_t(rows) + uint32_t(r);
}

__global__ void k_grid_keys(const float2* __restrict__ pos, const float* __restrict__ omega, long n,
                            const GridInst* __restrict__ inst, int n_inst, int set_mode, uint32_t nbins, int rows,
                            uint32_t* __restrict__ keys) {
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x)
        keys[i] = grid_key(pos, omega, i, inst, n_inst, set_mode, nbins, rows);
}

// A small grid (see vpmc_blocksort.cuh): keys, sort and ranges in one launch of one
// CTA, where the general build takes a launch for the keys, three a digit and one
// for the ranges.  64^2 particles, 65,536 sub-rows: 18.9 us; the whole step 239 -> 182 us.
__global__ void __launch_bounds__(kSmallThreads) k_grid_small(const float2* __restrict__ pos,
                                                              const float* __restrict__ omega, int n,
                                                              const GridInst* __restrict__ inst, int n_inst,
                                                              int set_mode, uint32_t nbins, int rows, int ibits,
                                                              uint32_t* start, uint32_t* __restrict__ cstart,
                                                              uint32_t* __restrict__ perm) {
    extern __shared__ uint32_t words[];
#pragma unroll 2
    for (int i = threadIdx.x; i < n; i += kSmallThreads)
        words[i] = grid_key(pos, omega, i, inst, n_inst, set_mode, nbins, rows);
    const int nsub = int(nbins) * rows;
    small_sort(words, n, nsub + 1, ibits, perm, start);
    if (rows > 1) {
        __syncthreads();   // start is read back by the threads of this CTA
        for (uint32_t b = threadIdx.x; b <= nbins; b += kSmallThreads) cstart[b] = start[size_t(b) * rows];
    }
}

// First candidate of every sub-row (and of every bin): the first sorted key >= k,
// searched between the bounds of the block's span of consecutive keys (few
// candidates).  Counting the keys with an atomic each and scanning the counts moves
// 16 bytes a sub-row and takes five launches; this writes 4.  A long span shares
// the two full searches (14.5 M sub-rows: 212 us with spans of 256, 101 us with 4096).
__global__ void __launch_bounds__(256) k_grid_starts(const uint32_t* __restrict__ keys, uint32_t n, long nsub, int rows,
                                                     int span, uint32_t* __restrict__ start,
                                                     uint32_t* __restrict__ cstart) {
    __shared__ uint32_t s_b[2];
    for (long k0 = long(blockIdx.x) * span; k0 <= nsub; k0 += long(gridDim.x) * span) {
        if (threadIdx.x < 2)
            s_b[threadIdx.x] = lower_bound_key(keys, n, uint32_t(min(nsub, k0 + long(threadIdx.x) * (span - 1))));
        __syncthreads();
        const uint32_t lo = s_b[0], hi = s_b[1];
        for (long k = k0 + threadIdx.x; k <= nsub && k < k0 + span; k += 256) {
            const uint32_t s = lo + lower_bound_key(keys + lo, hi - lo, uint32_t(k));
            start[k] = s;
            if (rows > 1 && k % rows == 0) cstart[k / rows] = s;
        }
        __syncthreads();
    }
}

__global__ void k_grid_gather(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ start, long n,
                              uint32_t nbins, const float2* __restrict__ pos, const float* __restrict__ omega,
                              const GridInst* __restrict__ inst, int n_inst, int set_mode,
                              Cand* __restrict__ cand, float4* __restrict__ cand4) {
    const long nv = start[nbins];
    for (long p = long(blockIdx.x) * blockDim.x + threadIdx.x; p < nv && p < n; p += long(gridDim.x) * blockDim.x) {
        const uint32_t i = perm[p];
        const GridInst G = inst[inst_of_particle(inst, n_inst, i)];
        float2 q = pos[i];
        if (G.periodic) { q.x = wrapf(q.x, G.Lx); q.y = wrapf(q.y, G.Ly); }
        const float w = omega ? omega[i] : 1.f;
        // weight 2 sigma |omega| (or 2 sigma omega), FP32 hi part + remainder
        const double wd = double(set_mode == SET_ONE_SIGNED ? w : fabsf(w)) * (80.0 / (7.0 * kPiD * double(G.hw) * G.hw));
        const float wt = float(wd);
        if (cand) cand[p] = Cand{q.x, q.x, q.y, q.y, wt, wt, float(wd - double(wt)), 0.f};
        if (cand4) cand4[p] = make_float4(q.x, q.y, wt, 0.f);
    }
}

// Deformed records: metric G = F^-T F^-1 of F = [[F.x, F.y], [F.z, F.w]]
// (the inverse the reference applies, include/vorticity_query.cuh:52-63,
// divides the adjugate by det F), formed in FP64.
__global__ void k_grid_gather_f(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ start, long n,
                                uint32_t nbins, const float2* __restrict__ pos, const float* __restrict__ omega,
                                const float4* __restrict__ F, const GridInst* __restrict__ inst, int n_inst,
                                int set_mode, CandF* __restrict__ cand) {
    const long nv = start[nbins];
    for (long p = long(blockIdx.x) * blockDim.x + threadIdx.x; p < nv && p < n; p += long(gridDim.x) * blockDim.x) {
        const uint32_t i = perm[p];
        const GridInst G = inst[inst_of_particle(inst, n_inst, i)];
        float2 q = pos[i];
        if (G.periodic) { q.x = wrapf(q.x, G.Lx); q.y = wrapf(q.y, G.Ly); }
        const float w = omega ? omega[i] : 1.f;
        const double wd = double(set_mode == SET_ONE_SIGNED ? w : fabsf(w)) * (80.0 / (7.0 * kPiD * double(G.hw) * G.hw));
        const float wt = float(wd);
        const float4 f = F[i];
        const double det = double(f.x) * f.w - double(f.y) * f.z;
        const double id2 = 1.0 / (det * det);
        CandF r;
        r.f[0] = q.x;
        r.f[1] = q.y;
        r.f[2] = float((double(f.w) * f.w + double(f.z) * f.z) * id2);
        r.f[3] = float(-(double(f.w) * f.y + double(f.z) * f.x) * id2);
        r.f[4] = float((double(f.y) * f.y + double(f.x) * f.x) * id2);
        r.f[5] = wt;
        r.f[6] = float(wd - double(wt));
#pragma unroll
        for (int k = 7; k < 16; ++k) r.f[k] = 0.f;
        cand[p] = r;
    }
}

__global__ void k_sigma(const float4* __restrict__ F, long n, unsigned* __restrict__ out) {
    unsigned m = 0u;
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x) {
        const float4 f = F[i];
        const float sm = sigma_max(f);
        const float det = f.x * f.w - f.y * f.z;
        // non-negative floats order as their bit patterns; degenerate F -> +inf
        m = max(m, (sm == sm && sm <= 3.0e38f && det > 0.f) ? __float_as_uint(sm) : 0x7f800000u);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__global__ void k_grid_weights(const double* __restrict__ x, long n, double scale, Cand* __restrict__ cand) {
    for (long p = long(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += long(gridDim.x) * blockDim.x) {
        const double v = x[p] * scale;
        const float hi = float(v);
        cand[p].w = hi;
        cand[p].w2 = hi;
        cand[p].wl = float(v - double(hi));
    }
}

__global__ void k_bin_points(const float2* __restrict__ pts, long M, const GridInst* __restrict__ inst,
                             int set, int field9, uint32_t* __restrict__ qbin, uint32_t* __restrict__ qcount) {
    for (long m = long(blockIdx.x) * blockDim.x + threadIdx.x; m < M; m += long(gridDim.x) * blockDim.x) {
        const GridInst G = inst[0];
        float2 p = pts[m];
        uint32_t b = kNoBin;
        bool ok = p.x == p.x && p.y == p.y;
        if (ok && G.periodic) {
            const float kx = floorf(p.x / G.Lx), ky = floorf(p.y / G.Ly);
            if (field9 && (fabsf(kx) > 2.f || fabsf(ky) > 2.f)) ok = false;
            p.x = p.x - kx * G.Lx;
            p.y = p.y - ky * G.Ly;
        } else if (ok) {
            ok = !(p.x < 0.f || p.x > G.Lx || p.y < 0.f || p.y > G.Ly);
        }
        if (ok) {
            const int cx = min(max(floor_int(p.x * G.inv_sx), 0), G.gx - 1);
            const int cy = min(max(floor_int(p.y * G.inv_sy), 0), G.gy - 1);
            b = uint32_t(G.bin_base) + uint32_t(set) * uint32_t(G.gx * G.gy) + uint32_t(cx * G.gy + cy);
            atomicAdd(&qcount[b], 1u);
        }
        qbin[m] = b;
    }
}

__global__ void k_scatter_points(const float2* __restrict__ pts, long M, const GridInst* __restrict__ inst,
                                 int n_inst, const uint32_t* __restrict__ qbin, const uint32_t* __restrict__ qstart,
                                 uint32_t* __restrict__ qfill, QRec* __restrict__ qrec) {
    for (long m = long(blockIdx.x) * blockDim.x + threadIdx.x; m < M; m += long(gridDim.x) * blockDim.x) {
        const uint32_t b = qbin[m];
        if (b == kNoBin) continue;
        const GridInst G = inst[inst_of_bin(inst, n_inst, b)];
        float2 p = pts[m];
        uint32_t fl = (2u) | (2u << 3);
        if (G.periodic) {
            const float kx = floorf(p.x / G.Lx), ky = floorf(p.y / G.Ly);
            p.x = p.x - kx * G.Lx;
            p.y = p.y - ky * G.Ly;
            const int ikx = min(max(int(kx), -2), 2), iky = min(max(int(ky), -2), 2);
            fl = uint32_t(ikx + 2) | (uint32_t(iky + 2) << 3);
        }
        const uint32_t slot = atomicAdd(&qfill[b], 1u);
        qrec[qstart[b] + slot] = QRec{p.x, p.y, uint32_t(m), fl};
    }
}

// Direct placement of binned samples: the generator counted them per (bin,
// sub-cell) and kept each one's rank there, so a sample's slot is its bin's start
// plus the counts of the sub-cells before its own plus its rank.  One pass over
// the samples instead of three, for as long as the records (16 bytes, stored in
// no order) and the counters stay in L2; beyond, the staged passes below.
__global__ void k_place_direct(const float2* __restrict__ pts, long M, const GridInst* __restrict__ inst, int n_inst,
                               const uint32_t* __restrict__ qbin, const uint32_t* __restrict__ qrank,
                               const uint32_t* __restrict__ qstart, const uint32_t* __restrict__ qsub,
                               QRec* __restrict__ qrec) {
    for (long m = long(blockIdx.x) * blockDim.x + threadIdx.x; m < M; m += long(gridDim.x) * blockDim.x) {
        const uint32_t b = qbin[m];
        if (b == kNoBin) continue;
        const uint32_t rk = qrank[m], sub = rk & 15u;
        float2 p = pts[m];
        const uint4* c4 = reinterpret_cast<const uint4*>(qsub + size_t(b) * 16);
        uint32_t slot = qstart[b] + (rk >> 4);
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            if (4u * i >= sub) break;
            const uint4 c = c4[i];
            slot += c.x + (4u * i + 1u < sub ? c.y : 0u) + (4u * i + 2u < sub ? c.z : 0u) + (4u * i + 3u < sub ? c.w : 0u);
        }
        const GridInst& G = inst[n_inst == 1 ? 0 : inst_of_bin(inst, n_inst, b)];
        uint32_t fl = (2u) | (2u << 3);
        if (G.periodic) {
            const float kx = floorf(p.x / G.Lx), ky = floorf(p.y / G.Ly);
            p.x = p.x - kx * G.Lx;
            p.y = p.y - ky * G.Ly;
            const int ikx = min(max(int(kx), -2), 2), iky = min(max(int(ky), -2), 2);
            fl = uint32_t(ikx + 2) | (uint32_t(iky + 2) << 3);
        }
        qrec[slot] = QRec{p.x, p.y, uint32_t(m), fl};
    }
}

// Samples per bin from the counts per (bin, sub-cell).
__global__ void k_bin_totals(const uint32_t* __restrict__ qsub, long nbins, uint32_t* __restrict__ qcount) {
    for (long b = long(blockIdx.x) * blockDim.x + threadIdx.x; b < nbins; b += long(gridDim.x) * blockDim.x) {
        uint32_t t = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 c = reinterpret_cast<const uint4*>(qsub)[4 * b + i];
            t += c.x + c.y + c.z + c.w;
        }
        qcount[b] = t;
    }
}

// Placement of binned samples (three streaming passes).  Writing a 16-byte
// record straight to its final slot touches a different DRAM sector per
// sample (the bins of consecutive samples are unrelated).  Instead:
//   pass 1 (k_scatter_coarse): each CTA moves its tile of samples into runs
//     per super-bin (2^S consecutive bins; one global atomic per CTA and
//     super-bin) as {unwrapped point, sample id, bin};
//   pass 2 (k_scatter_window): the super-bin segments into runs per window
//     (2^W consecutive bins, ~1-2k samples), placed at the window's first
//     slot qstart[w << W];
//   pass 3 (k_scatter_assemble): one CTA per window gives every record its
//     slot from shared-memory counters started at qstart of its bin, builds
//     the window in shared memory (wrapping the point, deriving its image
//     flags) and writes it out as one contiguous block.
// The order of queries inside a bin is not fixed by this; no result depends
// on it (each query's field value is its own fixed-order sum).
constexpr int kPlaceThreads = 512;
constexpr int kPlaceTile = 8;                                // records per thread per tile
constexpr int kTileRecs = kPlaceThreads * kPlaceTile;        // 4096 records = 64 KB staged per tile
constexpr int kTargetSuper = 512;                            // super-bins per grid
constexpr int kWinMax = 2048;                                // windows one tile may sort in shared memory
constexpr int kAsmPer = 8;                                   // records per thread of a window that fits
constexpr int kWinBinsMax = 64;                             // bins per window at most

// Exclusive prefix sum of v[0..n) in place (shared memory, n small), block
// of kPlaceThreads; returns the total.
__device__ __forceinline__ uint32_t block_scan_excl(uint32_t* v, int n, uint32_t* s_warp) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int per = (n + kPlaceThreads - 1) / kPlaceThreads;
    const int b = min(n, tid * per), e = min(n, b + per);
    uint32_t sum = 0;
    for (int i = b; i < e; ++i) sum += v[i];
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t t = lane < kPlaceThreads / 32 ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < kPlaceThreads / 32) s_warp[lane] = t;
    }
    __syncthreads();
    uint32_t run = (x - sum) + (wid > 0 ? s_warp[wid - 1] : 0u);
    for (int i = b; i < e; ++i) {
        const uint32_t c = v[i];
        v[i] = run;
        run += c;
    }
    const uint32_t total = s_warp[kPlaceThreads / 32 - 1];
    __syncthreads();
    return total;
}

// Pass 1: each tile of samples counting-sorted by super-bin in shared memory,
// one global reservation per (tile, super-bin), then written out as
// contiguous runs (coalesced stores).
__global__ void __launch_bounds__(kPlaceThreads) k_scatter_coarse(const float2* __restrict__ pts, long M,
                                                                 const uint32_t* __restrict__ qbin,
                                                                 const uint32_t* __restrict__ qstart, int shift,
                                                                 int nsuper, uint32_t* __restrict__ super_fill,
                                                                 uint4* __restrict__ tmp) {
    extern __shared__ __align__(16) uint4 srec[];   // kTileRecs
    __shared__ uint32_t hist[kTargetSuper], loff[kTargetSuper], s_warp[32];
    __shared__ long long goff[kTargetSuper];
    // the tile's bins and points are loaded one tile ahead (while the previous
    // tile is written out)
    uint32_t bb[kPlaceTile], lr[kPlaceTile];
    float2 pp[kPlaceTile];
    auto load_tile = [&](long t) {
#pragma unroll
        for (int j = 0; j < kPlaceTile; ++j) {
            const long m = t + long(j) * kPlaceThreads + threadIdx.x;
            bb[j] = m < M ? qbin[m] : kNoBin;
            pp[j] = m < M ? pts[m] : make_float2(0.f, 0.f);   // unwrapped: pass 3 wraps it
        }
    };
    long t0 = long(blockIdx.x) * kTileRecs;
    if (t0 >= M) return;
    load_tile(t0);
    for (;;) {
        for (int k = threadIdx.x; k < nsuper; k += kPlaceThreads) hist[k] = 0u;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPlaceTile; ++j)
            if (bb[j] != kNoBin) lr[j] = atomicAdd(&hist[bb[j] >> shift], 1u);
        __syncthreads();
        for (int k = threadIdx.x; k < nsuper; k += kPlaceThreads) loff[k] = hist[k];
        __syncthreads();
        const uint32_t ntile = block_scan_excl(loff, nsuper, s_warp);
        for (int k = threadIdx.x; k < nsuper; k += kPlaceThreads) {
            const uint32_t c = hist[k];
            goff[k] = c ? (long long)(qstart[uint32_t(k) << shift] + atomicAdd(&super_fill[k], c)) - loff[k] : 0;
        }
#pragma unroll
        for (int j = 0; j < kPlaceTile; ++j) {
            if (bb[j] == kNoBin) continue;
            const long m = t0 + long(j) * kPlaceThreads + threadIdx.x;
            srec[loff[bb[j] >> shift] + lr[j]] = make_uint4(__float_as_uint(pp[j].x), __float_as_uint(pp[j].y),
                                                            uint32_t(m), bb[j]);
        }
        __syncthreads();
        const long tn = t0 + long(gridDim.x) * kTileRecs;
        if (tn < M) load_tile(tn);
        for (uint32_t i = threadIdx.x; i < ntile; i += kPlaceThreads) {
            const uint4 r = srec[i];
            tmp[goff[r.w >> shift] + i] = r;
        }
        __syncthreads();
        if (tn >= M) break;
        t0 = tn;
    }
}

// Query record of a placed sample: wrapped point and image flags (Lx, Ly: the
// domain of its instance, (0, 0) where it is not periodic).
__device__ __forceinline__ QRec make_qrec(uint4 r, float2 L) {
    float2 p = make_float2(__uint_as_float(r.x), __uint_as_float(r.y));
    uint32_t fl = (2u) | (2u << 3);
    if (L.x > 0.f) {
        const float kx = floorf(p.x / L.x), ky = floorf(p.y / L.y);
        p.x = p.x - kx * L.x;
        p.y = p.y - ky * L.y;
        const int ikx = min(max(int(kx), -2), 2), iky = min(max(int(ky), -2), 2);
        fl = uint32_t(ikx + 2) | (uint32_t(iky + 2) << 3);
    }
    return QRec{p.x, p.y, r.z, fl};
}
__device__ __forceinline__ float2 wrap_lengths(const GridInst& G) {
    return G.periodic ? make_float2(G.Lx, G.Ly) : make_float2(0.f, 0.f);
}

// Pass 2: the same per tile of the super-bin-grouped records, by window
// (2^W consecutive bins), placed from the window's first slot qstart[w << W].
// A tile spanning more windows than the shared-memory counters hold (one
// across many sparse super-bins) reserves per record instead.
__global__ void __launch_bounds__(kPlaceThreads) k_scatter_window(const uint4* __restrict__ tmp,
                                                                 const uint32_t* __restrict__ total, long M,
                                                                 int wshift, const uint32_t* __restrict__ qstart,
                                                                 uint32_t* __restrict__ win_fill,
                                                                 uint4* __restrict__ tmp2) {
    extern __shared__ __align__(16) uint4 srec[];   // kTileRecs
    __shared__ uint32_t hist[kWinMax], loff[kWinMax], s_warp[32];
    __shared__ long long goff[kWinMax];
    __shared__ uint32_t s_lo, s_hi;
    const long n = min(long(*total), M);
    // records loaded one tile ahead (while the previous tile is written out)
    uint4 r[kPlaceTile];
    auto load_tile = [&](long t) {
#pragma unroll
        for (int j = 0; j < kPlaceTile; ++j) {
            const long i = t + long(j) * kPlaceThreads + threadIdx.x;
            r[j] = i < n ? tmp[i] : make_uint4(0u, 0u, 0u, kNoBin);
        }
    };
    long t0 = long(blockIdx.x) * kTileRecs;
    if (t0 >= n) return;
    if (threadIdx.x == 0) { s_lo = 0xffffffffu; s_hi = 0u; }
    load_tile(t0);
    __syncthreads();
    for (;;) {
        uint32_t lo = 0xffffffffu, hi = 0u;
#pragma unroll
        for (int j = 0; j < kPlaceTile; ++j)
            if (r[j].w != kNoBin) { lo = min(lo, r[j].w >> wshift); hi = max(hi, r[j].w >> wshift); }
        atomicMin(&s_lo, lo);
        atomicMax(&s_hi, hi);
        __syncthreads();
        const uint32_t wlo = s_lo, span = s_hi >= s_lo ? s_hi - s_lo + 1u : 0u;
        const long tn = t0 + long(gridDim.x) * kTileRecs;
        if (span > uint32_t(kWinMax)) {
#pragma unroll
            for (int j = 0; j < kPlaceTile; ++j) {
                if (r[j].w == kNoBin) continue;
                const uint32_t w = r[j].w >> wshift;
                tmp2[qstart[w << wshift] + atomicAdd(&win_fill[w], 1u)] = r[j];
            }
            __syncthreads();
            if (threadIdx.x == 0) { s_lo = 0xffffffffu; s_hi = 0u; }
            if (tn < n) load_tile(tn);
            __syncthreads();
            if (tn >= n) break;
            t0 = tn;
            continue;
        }
        for (uint32_t k = threadIdx.x; k < span; k += kPlaceThreads) hist[k] = 0u;
        __syncthreads();
        uint32_t lr[kPlaceTile];
#pragma unroll
        for (int j = 0; j < kPlaceTile; ++j)
            if (r[j].w != kNoBin) lr[j] = atomicAdd(&hist[(r[j].w >> wshift) - wlo], 1u);
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < span; k += kPlaceThreads) loff[k] = hist[k];
        __syncthreads();
        const uint32_t ntile = block_scan_excl(loff, int(span), s_warp);
        for (uint32_t k = threadIdx.x; k < span; k += kPlaceThreads) {
            const uint32_t c = hist[k];
            goff[k] = c ? (long long)(qstart[(wlo + k) << wshift] + atomicAdd(&win_fill[wlo + k], c)) - loff[k] : 0;
        }
#pragma unroll
        for (int j = 0; j < kPlaceTile; ++j)
            if (r[j].w != kNoBin) srec[loff[(r[j].w >> wshift) - wlo] + lr[j]] = r[j];
        __syncthreads();
        if (threadIdx.x == 0) { s_lo = 0xffffffffu; s_hi = 0u; }
        if (tn < n) load_tile(tn);
        for (uint32_t i = threadIdx.x; i < ntile; i += kPlaceThreads) {
            const uint4 q = srec[i];
            tmp2[goff[(q.w >> wshift) - wlo] + i] = q;
        }
        __syncthreads();
        if (tn >= n) break;
        t0 = tn;
    }
}

// Pass 3: one window per CTA: every record gets its slot from shared-memory
// counters started at qstart of its bin, the window is built in shared memory
// and written out as one contiguous block (an over-full window is counted and
// placed from global memory, 8 records a thread in flight).  The chain of a window
// (load, rank, scan, place, store, and a barrier after each) bounds it, so many small
// CTAs share an SM: 128 threads where the bins hold up to 512 records, 256 up to
// 1,024, else 512.  What a record needs of its instance is looked up once a bin.
// 67 M samples in 668 a bin: 797 us with 512 threads, 610 with 256; 195 M samples of
// 24 instances around vortices: 3.09 ms with 512 threads and
// over-full windows in any order, 2.14 with 128 and all windows ordered (which takes
// 8 % from the evaluation after it).  Bulk copies of the windows in and out, one or
// two windows ahead, measured the same as these loads.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_scatter_assemble(const uint4* __restrict__ tmp2, long nbins, int wshift,
                                                            const uint32_t* __restrict__ qstart,
                                                            const GridInst* __restrict__ inst, int n_inst,
                                                            QRec* __restrict__ qrec, uint32_t* __restrict__ sstart) {
    constexpr int kCap = THREADS * kAsmPer;
    extern __shared__ __align__(16) QRec buf[];   // kCap records
    __shared__ uint32_t cnt[kWinBinsMax];
    __shared__ uint32_t sub[kSubCells * kWinBinsMax];   // per (sub-cell, bin of the window): count, then first slot
    __shared__ float4 corg[kWinBinsMax];                 // per bin of the window: its cell, for subcell_key
    __shared__ float2 wrap[kWinBinsMax];                 // and its instance's periodic lengths
    const long nwin = ((nbins - 1) >> wshift) + 1;
    long w = blockIdx.x;
    if (w >= nwin) return;
    if (sstart && w == 0 && threadIdx.x == 0) sstart[size_t(nbins) * kSubCells] = qstart[nbins];
    // window w's bounds and (when it fits) its records: loaded one window ahead,
    // so the loads overlap the previous window's write-out
    long b0 = w << wshift, b1 = min(nbins, b0 + (1L << wshift));
    uint32_t start = qstart[b0], nw = qstart[b1] - start;
    uint4 r[kAsmPer];
    auto load_records = [&](uint32_t st, uint32_t n) {
#pragma unroll
        for (int j = 0; j < kAsmPer; ++j) {
            const uint32_t k = threadIdx.x + uint32_t(j) * uint32_t(THREADS);
            if (k < n) r[j] = tmp2[st + k];
        }
    };
    auto load_window = [&](uint32_t st, uint32_t n) {
        if (n <= uint32_t(kCap)) load_records(st, n);
    };
    load_window(start, nw);
    for (;;) {
        const bool fits = nw <= uint32_t(kCap);
        const uint32_t nb = uint32_t(b1 - b0);
        for (long b = b0 + threadIdx.x; b < b1; b += THREADS) {
            cnt[b - b0] = qstart[b];
            const GridInst& G = inst[n_inst == 1 ? 0 : inst_of_bin(inst, n_inst, uint32_t(b))];
            const uint32_t cell = (uint32_t(b) - uint32_t(G.bin_base)) % uint32_t(G.gx * G.gy);
            corg[b - b0] = make_float4(float(int(cell) / G.gy), float(int(cell) % G.gy), G.inv_sx, G.inv_sy);
            wrap[b - b0] = wrap_lengths(G);
        }
        for (uint32_t i = threadIdx.x; i < uint32_t(kSubCells) * nb; i += THREADS) sub[i] = 0u;
        __syncthreads();
        // inside each bin the records are ordered by sub-cell, so that consecutive
        // queries of a bin lie close together
        uint32_t kr[kAsmPer];   // bin in the window | sub-cell << 8 | rank within (sub-cell, bin) << 12
        if (fits) {
#pragma unroll
            for (int j = 0; j < kAsmPer; ++j) {
                const uint32_t k = threadIdx.x + uint32_t(j) * uint32_t(THREADS);
                if (k >= nw) break;
                const uint32_t bl = r[j].w - uint32_t(b0);
                const QRec q = make_qrec(r[j], wrap[bl]);
                const uint32_t key = subcell_key(q.x, q.y, corg[bl]);
                kr[j] = bl | (key << 8) | (atomicAdd(&sub[key * nb + bl], 1u) << 12);
                r[j] = make_uint4(__float_as_uint(q.x), __float_as_uint(q.y), q.id, q.flags);
            }
        } else {   // a window that does not fit is counted, then placed, from global memory
            for (uint32_t k0 = 0; k0 < nw; k0 += uint32_t(kCap)) {
                load_records(start + k0, nw - k0);
#pragma unroll
                for (int j = 0; j < kAsmPer; ++j) {
                    if (k0 + threadIdx.x + uint32_t(j) * uint32_t(THREADS) >= nw) break;
                    const uint32_t bl = r[j].w - uint32_t(b0);
                    const QRec q = make_qrec(r[j], wrap[bl]);
                    atomicAdd(&sub[subcell_key(q.x, q.y, corg[bl]) * nb + bl], 1u);
                }
            }
        }
        __syncthreads();
        // each bin's 16 sub-cell counters -> first slots: a warp takes two bins
        // per pass, one counter per lane, a scan inside each 16-lane half
        {
            const uint32_t lane = threadIdx.x & 31u, c = lane & 15u;
            for (uint32_t b = (threadIdx.x >> 5) * 2u + (lane >> 4); b < ((nb + 1u) & ~1u); b += THREADS / 16) {
                const bool live = b < nb;
                const uint32_t n = live ? sub[c * nb + b] : 0u;
                uint32_t incl = n;
#pragma unroll
                for (int o = 1; o < 16; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o, 16);
                    if (c >= uint32_t(o)) incl += y;
                }
                if (live) {
                    sub[c * nb + b] = cnt[b] + incl - n;
                    if (sstart) sstart[(size_t(b0) + b) * kSubCells + c] = cnt[b] + incl - n;
                }
            }
        }
        __syncthreads();
        if (fits) {
#pragma unroll
            for (int j = 0; j < kAsmPer; ++j) {
                const uint32_t k = threadIdx.x + uint32_t(j) * uint32_t(THREADS);
                if (k >= nw) break;
                const uint32_t slot = sub[((kr[j] >> 8) & 15u) * nb + (kr[j] & 255u)] + (kr[j] >> 12);
                buf[slot - start] = QRec{__uint_as_float(r[j].x), __uint_as_float(r[j].y), r[j].z, r[j].w};
            }
        } else {
            for (uint32_t k0 = 0; k0 < nw; k0 += uint32_t(kCap)) {
                load_records(start + k0, nw - k0);
#pragma unroll
                for (int j = 0; j < kAsmPer; ++j) {
                    if (k0 + threadIdx.x + uint32_t(j) * uint32_t(THREADS) >= nw) break;
                    const uint32_t bl = r[j].w - uint32_t(b0);
                    const QRec q = make_qrec(r[j], wrap[bl]);
                    qrec[atomicAdd(&sub[subcell_key(q.x, q.y, corg[bl]) * nb + bl], 1u)] = q;
                }
            }
        }
        __syncthreads();
        // the next window's bounds and records go out before this one is written
        const long wn = w + gridDim.x;
        long nb0 = 0, nb1 = 0;
        uint32_t nstart = 0, nnw = 0;
        if (wn < nwin) {
            nb0 = wn << wshift;
            nb1 = min(nbins, nb0 + (1L << wshift));
            nstart = qstart[nb0];
            nnw = qstart[nb1] - nstart;
            load_window(nstart, nnw);
        }
        if (fits)
            for (uint32_t k = threadIdx.x; k < nw; k += THREADS) qrec[start + k] = buf[k];
        __syncthreads();
        if (wn >= nwin) break;
        w = wn;
        b0 = nb0;
        b1 = nb1;
        start = nstart;
        nw = nnw;
    }
}

// skip: bins of boxed instances get no items here.
__global__ void k_items_count(const uint32_t* __restrict__ qstart, long nbins, int chunk,
                              const GridInst* __restrict__ inst, int n_inst, int skip, uint32_t* __restrict__ per_bin) {
    for (long b = long(blockIdx.x) * blockDim.x + threadIdx.x; b < nbins; b += long(gridDim.x) * blockDim.x) {
        uint32_t c = qstart[b + 1] - qstart[b];
        if (skip && inst[inst_of_bin(inst, n_inst, uint32_t(b))].nb) c = 0u;
        per_bin[b] = (c + chunk - 1) / chunk;
    }
}

// First slot of each (bin, sub-cell) from the counts and the bins' starts.
__global__ void k_sub_starts(const uint32_t* __restrict__ qsub, const uint32_t* __restrict__ qstart, long nbins,
                             uint32_t* __restrict__ sstart) {
    for (long b = long(blockIdx.x) * blockDim.x + threadIdx.x; b < nbins; b += long(gridDim.x) * blockDim.x) {
        uint32_t s = qstart[b];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 c = reinterpret_cast<const uint4*>(qsub)[4 * b + i];
            reinterpret_cast<uint4*>(sstart)[4 * b + i] = make_uint4(s, s + c.x, s + c.x + c.y, s + c.x + c.y + c.z);
            s += c.x + c.y + c.z + c.w;
        }
        if (b == nbins - 1) sstart[nbins * kSubCells] = s;
    }
}

// Items of the boxes (aligned groups of sub-cells) of boxed instances.
__global__ void k_box_count(const uint32_t* __restrict__ sstart, long nbins, const GridInst* __restrict__ inst, int n_inst,
                            uint32_t* __restrict__ per_bin) {
    for (long b = long(blockIdx.x) * blockDim.x + threadIdx.x; b < nbins; b += long(gridDim.x) * blockDim.x) {
        const int nb = inst[n_inst == 1 ? 0 : inst_of_bin(inst, n_inst, uint32_t(b))].nb;
        uint32_t t = 0u;
        if (nb) {
            const int per = kSubCells / (nb * nb);
            for (int s = 0; s < kSubCells; s += per)
                t += (sstart[b * kSubCells + s + per] - sstart[b * kSubCells + s] + kBoxChunk - 1) / kBoxChunk;
        }
        per_bin[b] = t;
    }
}
__global__ void k_box_fill(const uint32_t* __restrict__ sstart, long nbins, const uint32_t* __restrict__ item_start,
                           const GridInst* __restrict__ inst, int n_inst, Item* __restrict__ items,
                           uint32_t* __restrict__ n_items, uint32_t* __restrict__ counter, long max_items) {
    for (long b = long(blockIdx.x) * blockDim.x + threadIdx.x; b < nbins; b += long(gridDim.x) * blockDim.x) {
        const uint32_t ib = n_inst == 1 ? 0u : uint32_t(inst_of_bin(inst, n_inst, uint32_t(b)));
        const int nb = inst[ib].nb;
        if (!nb) continue;
        const int per = kSubCells / (nb * nb);
        uint32_t it = item_start[b];
        for (int s = 0; s < kSubCells; s += per) {
            const uint32_t q0 = sstart[b * kSubCells + s], c = sstart[b * kSubCells + s + per] - q0;
            for (uint32_t o = 0; o < c; o += kBoxChunk, ++it)
                if (it < max_items)
                    items[it] = Item{uint32_t(b), q0 + o, min(uint32_t(kBoxChunk), c - o) | (uint32_t(s / per) << 16), ib};
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const uint32_t t = item_start[nbins];
        *n_items = t < max_items ? t : uint32_t(max_items);
        *counter = 0;
    }
}

__global__ void k_items_fill(const uint32_t* __restrict__ qstart, long nbins, int chunk,
                             const uint32_t* __restrict__ item_start, const GridInst* __restrict__ inst,
                             int n_inst, int skip, Item* __restrict__ items, uint32_t* __restrict__ n_items,
                             uint32_t* __restrict__ counter, long max_items) {
    for (long b = long(blockIdx.x) * blockDim.x + threadIdx.x; b < nbins; b += long(gridDim.x) * blockDim.x) {
        const uint32_t q0 = qstart[b], c = qstart[b + 1] - q0;
        uint32_t it = item_start[b];
        const uint32_t ib = uint32_t(inst_of_bin(inst, n_inst, uint32_t(b)));
        if (skip && inst[ib].nb) continue;
        for (uint32_t o = 0; o < c; o += chunk, ++it)
            if (it < max_items) items[it] = Item{uint32_t(b), q0 + o, min(uint32_t(chunk), c - o), ib};
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const uint32_t t = item_start[nbins];
        *n_items = t < max_items ? t : uint32_t(max_items);
        *counter = 0;
    }
}

// Few bins and items: the items (and with qsub first the bins' totals and starts) in
// one launch of one CTA.  (8,192 bins of 3,000 samples: 428 us in one CTA, 27 us in
// the general three launches.)
bool items_in_one(long nbins, long queries) { return nbins <= 4096 && queries <= (1L << 19); }

__device__ __forceinline__ uint32_t scan_1024(uint32_t v, uint32_t* s_warp, uint32_t* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    __syncthreads();   // s_warp may still be read from the previous scan
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
    *total = s_warp[31];
    return inc - v + (w > 0 ? s_warp[w - 1] : 0u);
}

__global__ void __launch_bounds__(1024) k_items_small(const uint32_t* __restrict__ qsub, uint32_t* qstart, int nbins,
                                                      int chunk, const GridInst* __restrict__ inst, int n_inst, int skip,
                                                      Item* __restrict__ items, uint32_t* __restrict__ n_items,
                                                      uint32_t* __restrict__ counter, long max_items) {
    __shared__ uint32_t s_warp[32];
    const int per = (nbins + 1023) / 1024, b0 = min(nbins, int(threadIdx.x) * per), b1 = min(nbins, b0 + per);
    uint32_t total = 0u;
    if (qsub) {
        const uint4* c4 = reinterpret_cast<const uint4*>(qsub);
        auto bin_total = [&](int b) {
            uint32_t t = 0u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 c = c4[4 * b + i];
                t += c.x + c.y + c.z + c.w;
            }
            return t;
        };
        uint32_t sum = 0u;
        for (int b = b0; b < b1; ++b) sum += bin_total(b);
        uint32_t run = scan_1024(sum, s_warp, &total);
        for (int b = b0; b < b1; ++b) {
            qstart[b] = run;
            run += bin_total(b);
        }
        if (threadIdx.x == 0) qstart[nbins] = total;
        __syncthreads();   // the starts are read back by the threads of this CTA
    }
    auto boxed = [&](int b) { return skip && inst[n_inst > 1 ? inst_of_bin(inst, n_inst, uint32_t(b)) : 0].nb != 0; };
    uint32_t sum = 0u;
    for (int b = b0; b < b1; ++b)
        if (!boxed(b)) sum += (qstart[b + 1] - qstart[b] + uint32_t(chunk) - 1u) / uint32_t(chunk);
    uint32_t it = scan_1024(sum, s_warp, &total);
    for (int b = b0; b < b1; ++b) {
        if (boxed(b)) continue;
        const uint32_t q0 = qstart[b], c = qstart[b + 1] - q0;
        const uint32_t ib = c && n_inst > 1 ? uint32_t(inst_of_bin(inst, n_inst, uint32_t(b))) : 0u;
        for (uint32_t o = 0; o < c; o += uint32_t(chunk), ++it)
            if (it < max_items) items[it] = Item{uint32_t(b), q0 + o, min(uint32_t(chunk), c - o), ib};
    }
    if (threadIdx.x == 0) {
        *n_items = total < max_items ? total : uint32_t(max_items);
        *counter = 0;
    }
}

// ---------------------------------------------------------------- eval kernel
struct Piece {
    uint32_t gstart, cnt;   // candidate run in global memory
    float qdx, qdy;         // offset added to the query point (folds the periodic image)
    uint32_t b0;            // index into the sub-row starts of the run's first sub-row
    float x0, y0;           // bin-local left edge of the run's column, lower edge of its first sub-row
    int16_t nr;             // sub-rows in the run
    int8_t mx, my;          // image index of the run (for FIELD9)
};
struct BatchPiece {
    uint32_t soff, cnt, gstart;
    int piece;
};

struct EvalArgs {
    const GridInst* inst;
    const uint32_t* cstart;   // candidate range per sub-row (rows per cell: `rows`)
    int rows;
    const Cand* cand;
    const CandF* candf;
    const QRec* qrec;
    const Item* items;
    const uint32_t* n_items;
    uint32_t* counter;
    float* out_f32;
    double* out_f64;
    unsigned* flags;
    uint32_t wait_limit;      // polls of a staging wait before the kernel gives up
    const double* qweight;    // SCAT modes: the weight of each query (by id)
};

// The same sum for deformed kernels: s2 from the expanded metric form, its
// coefficients pre-scaled by kappa (5 packed FMAs instead of 3), the spline as above.
template <int NPR, int NPMAX>
__device__ __forceinline__ void packed_run_f(const CandF* __restrict__ cs, int cnt, const f2x (&QXX)[NPMAX],
                                             const f2x (&QXY)[NPMAX], const f2x (&QYY)[NPMAX],
                                             const f2x (&QX)[NPMAX], const f2x (&QY)[NPMAX], f2x (&P)[NPMAX]) {
    const f2x HALF = pk2(0.5f, 0.5f);
#pragma unroll 2
    for (int c = 0; c < cnt; ++c) {
        const ulonglong2* rec = reinterpret_cast<const ulonglong2*>(cs[c].f);
        const ulonglong2 R0 = rec[0];   // kappa (g11), kappa (2 g12)
        const ulonglong2 R1 = rec[1];   // kappa (g22), kappa (a)
        const ulonglong2 R2 = rec[2];   // kappa (b), kappa (e)
        const ulonglong2 R3 = rec[3];   // (w), (0)
#pragma unroll
        for (int pr = 0; pr < NPR; ++pr) {
            f2x s2 = fma2(R0.x, QXX[pr], R2.y);
            s2 = fma2(R0.y, QXY[pr], s2);
            s2 = fma2(R1.x, QYY[pr], s2);
            s2 = fma2(R1.y, QX[pr], s2);
            s2 = fma2(R2.x, QY[pr], s2);
            float ra, rb;
            up2(s2, ra, rb);
            const float sa = sqrt_approx(fabsf(ra)), sb = sqrt_approx(fabsf(rb));
            const f2x t = pk2(__saturatef(fmaf(-kInvSqrt3, sa, 1.f)), __saturatef(fmaf(-kInvSqrt3, sb, 1.f)));
            const f2x in = fma2(s2, t, HALF);
            const f2x t3 = mul2(mul2(t, t), t);
            float ia, ib, ta, tb;
            up2(in, ia, ib);
            up2(t3, ta, tb);
            P[pr] = fma2(R3.x, pk2(fminf(ia, ta), fminf(ib, tb)), P[pr]);
        }
    }
}

// s + e += x with s the running sum and e the running sum of its rounding errors
// (Knuth's TwoSum; the products are formed with __fmul_rn so no FMA contraction
// can fold them into the sum and break the exact error term).
__device__ __forceinline__ void two_sum_acc(float& s, float& e, float x) {
    const float t = __fadd_rn(s, x);
    const float bp = __fsub_rn(t, s);
    e = __fadd_rn(e, __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(x, bp)));
    s = t;
}

// The same for two sums at once.
__device__ __forceinline__ void two_sum_acc2(f2x& s, f2x& e, f2x x) {
    const f2x t = add2(s, x), bp = sub2(t, s);
    e = add2(e, add2(sub2(s, sub2(t, bp)), sub2(x, bp)));
    s = t;
}

// W / 2 sigma of the cubic spline and its r-derivative over r, divided by -3 / h, for
// FP32 pairs without a branch: one reciprocal square root gives r and 1 / r; with
// t = (1 - r/h)+ the value is min(1/2 - 3 (r/h)^2 t, t^3) (see packed_run) and the
// derivative's pieces are (3 t - 1) / h inside r <= h / 2 (t >= 1/2) and t^2 / r
// beyond, both exactly zero outside the support.  r2 > 0 (the caller adds 1e-30).
__device__ __forceinline__ void spline_vdr_f32(float r2, float ih, float kap, float& v, float& dr) {
    const float rs = wide::rsqrt_est(r2);
    const float t = __saturatef(fmaf(-ih, r2 * rs, 1.f));
    const float t2 = t * t;
    v = fminf(fmaf(kap * r2, t, 0.5f), t2 * t);
    dr = t >= 0.5f ? fmaf(3.f * ih, t, -ih) : t2 * rs;
}

// Images a sample may pair through (unbiased law): bit (sx + 1) * 3 + (sy + 1)
// is set when a run shifted by image (sx, sy) pairs the sample in unwrapped tile
// k with source image k + s inside {-1, 0, 1}^2 (flags: bits 0-2 kx + 2, 3-5 ky + 2).
__device__ __forceinline__ uint32_t image_mask9(uint32_t flags) {
    const int kx = int(flags & 7u) - 2, ky = int((flags >> 3) & 7u) - 2;
    uint32_t m = 0u;
#pragma unroll
    for (int sx = -1; sx <= 1; ++sx)
#pragma unroll
        for (int sy = -1; sy <= 1; ++sy)
            if (kx + sx >= -1 && kx + sx <= 1 && ky + sy >= -1 && ky + sy <= 1) m |= 1u << ((sx + 1) * 3 + (sy + 1));
    return m;
}

// The transposed sums of one staged batch, from the sample side (SCAT modes).
// The item's samples sit in s_sq (x, y, weight hi, weight lo; image masks in
// s_sqm); the batch's particles are staged back to back in s_cand.  Lane l
// takes staged particles l, l + 32, ... (whatever run each lies in), sums over
// all the item's samples the terms a_s W(|x_p - y_s|) and a_s dW/dx_p in the
// pair's image, and adds them to out[3 slot + {0, 1, 2}] with one FP64 atomic
// each, slot = the particle's candidate index.  The pair is the one the GRAD
// modes form with the roles of query and candidate swapped: the sample seen
// through the run's image is y + qdx, so x_p - y_s = (c - qdx) - q.
template <typename ST, bool K9>
__device__ __forceinline__ void scat_batch(const Cand* __restrict__ s_cand, const BatchPiece* s_bp,
                                           const Piece* s_pc, int nbp, const uint2* s_rng, const float4* s_sq,
                                           const uint16_t* s_sqm, int nq, const GridInst& G,
                                           double* __restrict__ out) {
    constexpr bool k32 = std::is_same<ST, float>::value;
    const int lane = threadIdx.x & 31;
    const ST hw = ST(G.hw), ih = ST(1) / hw;
    const ST A = ST(3) * ih * ih * ih, B = ST(-3) * ih * ih;
    // the particles of the runs' parts within reach, one after the other
    uint32_t total = 0u, off = 0u;
    for (int k = 0; k < nbp; ++k) total += s_rng[k].y - s_rng[k].x;
    int b = 0;
    for (uint32_t i = uint32_t(lane); i < total; i += 32u) {
        while (i - off >= s_rng[b].y - s_rng[b].x) {
            off += s_rng[b].y - s_rng[b].x;
            ++b;
        }
        const uint32_t at = s_rng[b].x + (i - off);
        const BatchPiece bp = s_bp[b];
        const Piece pc = s_pc[bp.piece];
        const Cand cv = s_cand[bp.soff + at];
        const uint32_t pbit = uint32_t((pc.mx + 1) * 3 + (pc.my + 1));
        const ST cx = ST(cv.x) - ST(pc.qdx), cy = ST(cv.y) - ST(pc.qdy);
        double gv, ggx, ggy;
        if constexpr (k32) {
            float sv = 0.f, ev = 0.f;   // the sums and their error terms
            f2x sg = pk2(0.f, 0.f), eg = sg;
            const f2x C = pk2(cx, cy);
            const float kap = G.B, m3ih = -3.f * ih;
            const uint32_t bit = 1u << pbit;
            // branch-free: a pair outside the support or the sample's images adds
            // exact zeros, which leave the compensated sums unchanged
#pragma unroll 4
            for (int j = 0; j < nq; ++j) {
                const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(&s_sq[j]);   // (x, y), (weight, images)
                float w, m, dx, dy;
                up2(q.y, w, m);
                if (K9) w = (__float_as_uint(m) & bit) ? w : 0.f;
                const f2x d = sub2(C, q.x);   // x_p - y_s
                up2(d, dx, dy);
                float v, dr;
                spline_vdr_f32(fmaf(dx, dx, fmaf(dy, dy, 1e-30f)), ih, kap, v, dr);
                const float wdr = __fmul_rn(__fmul_rn(w, m3ih), dr);
                two_sum_acc(sv, ev, __fmul_rn(w, v));
                two_sum_acc2(sg, eg, mul2(pk2(wdr, wdr), d));
            }
            gv = double(sv) + double(ev);
            float gx, gy, hx, hy;
            up2(sg, gx, gy);
            up2(eg, hx, hy);
            ggx = double(gx) + double(hx);
            ggy = double(gy) + double(hy);
        } else {
            gv = ggx = ggy = 0.0;
            for (int j = 0; j < nq; ++j) {
                if (K9 && !((uint32_t(s_sqm[j]) >> pbit) & 1u)) continue;
                const float4 q = s_sq[j];
                const double dx = cx - double(q.x), dy = cy - double(q.y);   // x_p - y_s
                const double r2 = dx * dx + dy * dy;
                const double r = sqrt(r2);
                if (r >= hw) continue;
                const double t = 1.0 - ih * r;
                double v, dr;   // W / 2 sigma and its r-derivative over r
                if (r <= 0.5 * hw) {
                    v = 0.5 + r2 * (A * r + B);
                    dr = 3.0 * A * r + 2.0 * B;
                } else {
                    v = t * t * t;
                    dr = -3.0 * t * t * ih / r;
                }
                const double w = double(q.z) + double(q.w);
                gv += w * v;
                ggx += w * dr * dx;
                ggy += w * dr * dy;
            }
        }
        if (gv != 0.0 || ggx != 0.0 || ggy != 0.0) {
            double* o = out + 3 * (size_t(bp.gstart) + size_t(at));
            atomicAdd(o, gv);
            atomicAdd(o + 1, ggx);
            atomicAdd(o + 2, ggy);
        }
    }
}

// Value and gradient sums of NJ queries over one staged run, FP32 pairs; the
// gradient in units of -3 / h.
template <int NJ>
__device__ __forceinline__ void grad32_run(const Cand* __restrict__ cs, int cnt, const f2x* pxy, const GridInst& G,
                                           float* pv, f2x* pg) {
    const float ih = G.inv_hw, kap = G.B;
#pragma unroll 2
    for (int c = 0; c < cnt; ++c) {
        const float4 xy = *reinterpret_cast<const float4*>(&cs[c].x);   // x, x, y, y
        const f2x C = pk2(xy.x, xy.z);
        const float w = cs[c].w;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const f2x d = sub2(pxy[j], C);   // q - c
            float dx, dy, v, dr;             // zeros outside the support
            up2(d, dx, dy);
            spline_vdr_f32(fmaf(dx, dx, fmaf(dy, dy, 1e-30f)), ih, kap, v, dr);
            const float wdr = w * dr;
            pv[j] = fmaf(w, v, pv[j]);
            pg[j] = fma2(pk2(wdr, wdr), d, pg[j]);
        }
    }
}
// One query's sum over one staged run to FP64 precision on the FP32 pipe (see
// vpmc_wide.cuh): records {xh, xl, yh, yl, w, ., wl, .} already shifted by the
// run's image.  LOW: some difference may need a second float.  A pair's error is
// below 1e-20 of W(0) (the FP64 form's: 3.5e-16), at ~190 FP32 instructions for a
// pair inside the support, 10 outside.
template <bool LOW>
__device__ __forceinline__ void wide_run(const Cand* __restrict__ cs, int cnt, float qx, float qy, float h, float lim,
                                         const wide::W3& half_h3, wide::W3& acc) {
    for (int c = 0; c < cnt; ++c) {
        const float4 p = *reinterpret_cast<const float4*>(&cs[c].x);
        float xh, xl = 0.f, yh, yl = 0.f;
        if (LOW) {
            float e;
            wide::two_sum(p.x, -qx, xh, e);
            wide::fast_two_sum(xh, wide::add(e, p.y), xh, xl);
            wide::two_sum(p.z, -qy, yh, e);
            wide::fast_two_sum(yh, wide::add(e, p.w), yh, yl);
        } else {
            xh = p.x - qx;
            yh = p.z - qy;
        }
        if (fmaf(xh, xh, yh * yh) < lim) {
            const wide::W3 v = wide::spline_h3(wide::norm2<LOW>(xh, xl, yh, yl), h, half_h3);
            if (v.a > 0.f) wide::add_product(acc, cs[c].w, cs[c].wl, v);
        }
    }
}

// The packed FP32 kernels run one-warp CTAs, 24 per SM (their 6.5 KB staging
// buffers fit 24 times in shared memory; 85 registers a thread at most) with 4
// queries per thread, 16 per SM with 6 and 12 with 8.  One warp per CTA: no warp of an item
// waits at a barrier for another.
constexpr int eval_min_blocks(int mode, int qpt) {
    return (mode == EVAL_FIELD || mode == EVAL_FIELD9 || mode == EVAL_FIELD_F || mode == EVAL_FIELD9_F)
               ? (qpt == 4 ? 24 : qpt == 6 ? 16 : 12)
               : (mode == EVAL_FIELD64 || mode == EVAL_FIELD9_64) ? 20
               : (mode == EVAL_GRAD32 || mode == EVAL_GRAD9_32) ? 16 : 1;
}

template <int MODE, int QPT>
__global__ void __launch_bounds__(kEvalThreads, eval_min_blocks(MODE, QPT)) k_eval(EvalArgs a) {
    extern __shared__ __align__(128) Cand s_cand[];
    __shared__ Piece s_pc[kMaxPieces];
    __shared__ BatchPiece s_bp[kMaxPieces + 2];
    __shared__ uint2 s_rng[kEvalThreads / 32][kMaxPieces + 2];   // per warp: its part of each batch piece
    __shared__ float4 s_wb[kEvalThreads / 32];                    // per warp: query bounding box (x0, x1, y0, y1)
    __shared__ int s_np, s_nbp, s_cur_piece, s_abort, s_pre;
    __shared__ uint32_t s_cur_off, s_btot, s_item;
    __shared__ float s_ox, s_oy;
    __shared__ __align__(8) uint64_t s_bar;
    constexpr bool kScat = eval_scat(MODE);
    constexpr int kScatQ = kScat ? kEvalThreads * QPT : 1;   // an item's queries (make_items' chunk)
    __shared__ float4 s_sq[kScatQ];
    __shared__ uint16_t s_sqm[kScatQ];

    constexpr bool kF64 = MODE == EVAL_SPMV64;
    constexpr bool kComp = MODE == EVAL_SPMV32;
    constexpr bool kField64 = MODE == EVAL_FIELD64 || MODE == EVAL_FIELD9_64;
    constexpr bool kTrim = kField64 || MODE == EVAL_GRAD32 || MODE == EVAL_GRAD9_32 || kScat || MODE == EVAL_FIELD || MODE == EVAL_FIELD9 || MODE == EVAL_FIELD_F ||
                           MODE == EVAL_FIELD9_F;
    // FP64 field: the item's queries and sums, slot j 32 + lane
    constexpr int kF64Q = kField64 ? kEvalThreads * QPT : 1;
    __shared__ float4 s_fq[kF64Q];      // x, y, image flags, id
    __shared__ double s_fd[kF64Q];
    constexpr bool kGrad = eval_grad(MODE);
    constexpr bool kGrad32 = MODE == EVAL_GRAD32 || MODE == EVAL_GRAD9_32;
    constexpr bool kGrad9 = MODE == EVAL_GRAD9_64 || MODE == EVAL_GRAD9_32;
    constexpr bool kScat9 = MODE == EVAL_SCAT9_64 || MODE == EVAL_SCAT9_32;
    using ST = typename std::conditional<MODE == EVAL_SCAT32 || MODE == EVAL_SCAT9_32, float, double>::type;
    using GT = double;
    constexpr bool kDef = eval_deformed(MODE);
    constexpr bool kDefExc = MODE == EVAL_FIELD_F_EXC;
    constexpr bool kPacked = MODE == EVAL_FIELD || MODE == EVAL_FIELD9 || MODE == EVAL_FIELD_F || MODE == EVAL_FIELD9_F;
    constexpr bool kField9 = MODE == EVAL_FIELD9 || MODE == EVAL_FIELD9_64 || MODE == EVAL_FIELD9_F;
    constexpr uint32_t kRec = kDef ? uint32_t(sizeof(CandF)) : uint32_t(sizeof(Cand));
    constexpr int kCap = kDef ? kCandCap / 2 : kCandCap;   // records per staged batch
    CandF* const s_candf = reinterpret_cast<CandF*>(s_cand);
    constexpr int NP = QPT / 2;   // packed query pairs
    static_assert(!kPacked || (QPT % 2 == 0), "packed path needs an even query count");
    using Acc = typename std::conditional<kF64 || kField64 || kGrad, double, float>::type;

    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init(&s_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
        s_item = atomicAdd(a.counter, 1u);
    }
    __syncthreads();
    uint32_t phase = 0;

    for (;;) {
        const uint32_t item = s_item;
        if (item >= *a.n_items) break;
        // claim the next item now: the atomic's round trip hides behind this one
        uint32_t next_item = 0;
        if (tid == 0) next_item = atomicAdd(a.counter, 1u);
        const Item it = a.items[item];
        const GridInst G = a.inst[it.inst];
        // the item's queries form units of 64 (one packed pair per lane); the warps
        // take consecutive units, as evenly as the count allows (a partly filled
        // item leaves no warp idle while another holds two units more), and a
        // warp runs only the pairs it holds: npw = its units (warp-uniform)
        constexpr int kWarps = kEvalThreads / 32;
        const int nunits = (int(it.qcnt) + 63) >> 6;   // <= kWarps * QPT / 2
        const int u0 = ((tid >> 5) * nunits) / kWarps;
        const int npw = (((tid >> 5) + 1) * nunits) / kWarps - u0;

        if (tid < 32) {
            // the walk, one column per lane of warp 0 (2 k + 1 <= 17 columns): each
            // column gives up to two runs (a periodic column wrapping in y splits),
            // emitted in column order as a serial walk would
            const int lane = tid;
            const uint32_t local = it.bin - uint32_t(G.bin_base);
            const uint32_t ncell = uint32_t(G.gx * G.gy);
            const uint32_t set = local / ncell, cell = local % ncell;
            const int cx = int(cell) / G.gy, cy = int(cell) % G.gy;
            const int R = a.rows, gyR = G.gy * R;
            const uint32_t colbase = (uint32_t(G.bin_base) + set * ncell) * uint32_t(R);
            int gxx, sxi, r0[2], r1[2], syi[2];
            walk_column(G, cx, cy, R, lane, gxx, sxi, r0, r1, syi);
            uint32_t rs[2] = {0u, 0u}, re[2] = {0u, 0u};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (r0[h] <= r1[h]) {
                    const uint32_t b0 = colbase + uint32_t(gxx * gyR + r0[h]);
                    rs[h] = a.cstart[b0];
                    re[h] = a.cstart[b0 + uint32_t(r1[h] - r0[h]) + 1];
                }
            }
            const bool v0 = re[0] > rs[0], v1 = re[1] > rs[1];
            const unsigned m0 = __ballot_sync(0xffffffffu, v0), m1 = __ballot_sync(0xffffffffu, v1);
            const unsigned lt = (1u << lane) - 1u;
            const int pos = __popc(m0 & lt) + __popc(m1 & lt);   // <= 2 (2 k + 1) = kMaxPieces
            // bin centre (wrapped coordinates): origin of the local frame
            const float ocx = (float(cx) + 0.5f) / G.inv_sx, ocy = (float(cy) + 0.5f) / G.inv_sy;
            const float srow = 1.f / (G.inv_sy * float(R));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (!(h == 0 ? v0 : v1)) continue;
                Piece pc;
                pc.gstart = rs[h];
                pc.cnt = re[h] - rs[h];
                pc.qdx = -float(sxi) * G.Lx;
                pc.qdy = -float(syi[h]) * G.Ly;
                pc.b0 = colbase + uint32_t(gxx * gyR + r0[h]);
                pc.x0 = float(gxx) / G.inv_sx - ocx - pc.qdx;
                pc.y0 = float(r0[h]) * srow - ocy - pc.qdy;
                pc.nr = int16_t(r1[h] - r0[h] + 1);
                pc.mx = int8_t(sxi);
                pc.my = int8_t(syi[h]);
                s_pc[pos + (h == 1 && v0 ? 1 : 0)] = pc;
            }
            // a walk that fits one batch is planned and its bulk copies issued here,
            // by the lanes that hold its runs (the previous item's reads of the
            // staging buffer ended at the item's closing barrier)
            const uint32_t c0 = v0 ? re[0] - rs[0] : 0u, c1 = v1 ? re[1] - rs[1] : 0u;
            uint32_t incl = c0 + c1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t tot_all = __shfl_sync(0xffffffffu, incl, 31);
            const uint32_t ex = incl - c0 - c1;   // staging offset of this lane's first run
            const bool one = tot_all > 0u && tot_all <= uint32_t(kCap);
            const int np = __popc(m0) + __popc(m1);
            if (one) {
                if (v0) s_bp[pos] = BatchPiece{ex, c0, rs[0], pos};
                if (v1) s_bp[pos + (v0 ? 1 : 0)] = BatchPiece{ex + c0, c1, rs[1], pos + (v0 ? 1 : 0)};
                if (lane == 0) {
                    fence_proxy_async_smem();
                    mbar_arrive_expect_tx(&s_bar, tot_all * kRec);
                }
                __syncwarp();
                fence_proxy_async_smem();
                const char* gsrc = kDef ? reinterpret_cast<const char*>(a.candf) : reinterpret_cast<const char*>(a.cand);
                if (v0)
                    bulk_g2s(reinterpret_cast<char*>(s_cand) + size_t(ex) * kRec, gsrc + size_t(rs[0]) * kRec,
                             c0 * kRec, &s_bar);
                if (v1)
                    bulk_g2s(reinterpret_cast<char*>(s_cand) + size_t(ex + c0) * kRec, gsrc + size_t(rs[1]) * kRec,
                             c1 * kRec, &s_bar);
            }
            if (lane == 0) {
                s_np = np;
                s_cur_piece = one ? np : 0;
                s_cur_off = 0;
                s_pre = one ? 1 : 0;
                s_nbp = one ? np : 0;
                s_btot = one ? tot_all : 0u;
                s_ox = ocx;
                s_oy = ocy;
            }
        }

        // this thread's queries
        float qx[QPT], qy[QPT];
        uint32_t qid[QPT];
        // image flags of the queries, 6 bits each (FIELD9)
        using QFlags = typename std::conditional<(6 * QPT > 32), unsigned long long, uint32_t>::type;
        QFlags qfl = 0;
        bool qv[QPT];
        Acc acc[QPT];
        float acc_c[QPT];
        double accg[kGrad && !kGrad32 ? QPT : 1][2];
        float sums[kGrad32 ? 3 * QPT : 1][3];   // value and gradient, three floats each
#pragma unroll
        for (int j = 0; j < QPT; ++j) {
            const uint32_t idx = uint32_t((u0 + (j >> 1)) * 64 + (j & 1) * 32 + (tid & 31));
            qv[j] = (j >> 1) < npw && idx < it.qcnt;
            QRec r = qv[j] ? a.qrec[it.qbeg + idx] : QRec{0.f, 0.f, 0u, (2u) | (2u << 3)};
            qx[j] = r.x;
            qy[j] = r.y;
            qid[j] = r.id;
            qfl |= QFlags(r.flags & 63u) << (6 * j);
            acc[j] = Acc(0);
            acc_c[j] = 0.f;
            if constexpr (kGrad && !kGrad32) accg[j][0] = accg[j][1] = 0.0;
            if constexpr (kGrad32)
                for (int k = 0; k < 9; ++k) sums[3 * j + k / 3][k % 3] = 0.f;
        }
        if constexpr (kScat) {
            // the item's samples with their weights a_s 2 sigma (FP32 hi + lo)
            const double sig2 = 80.0 / (7.0 * kPiD * double(G.hw) * double(G.hw));
            for (uint32_t k = uint32_t(tid); k < it.qcnt && k < uint32_t(kScatQ); k += kEvalThreads) {
                const QRec r = a.qrec[it.qbeg + k];
                const double w = a.qweight[r.id] * sig2;
                const float wh = float(w);
                // FP32 pairs use the weight's first float and the images, FP64 pairs all
                constexpr bool k32 = std::is_same<ST, float>::value;
                const uint32_t images = image_mask9(r.flags);
                s_sq[k] = make_float4(r.x, r.y, wh, k32 ? __uint_as_float(images) : float(w - double(wh)));
                s_sqm[k] = uint16_t(images);
            }
            if (tid == 0 && it.qcnt > uint32_t(kScatQ)) atomicOr(a.flags, FLAG_CAPACITY);
        }
        if constexpr (kField64) {
#pragma unroll
            for (int j = 0; j < QPT; ++j) {
                const int k = j * 32 + (tid & 31);
                const float nan = __int_as_float(0x7fffffff);   // an empty slot is near nothing
                s_fq[k] = make_float4(qv[j] ? qx[j] : nan, qv[j] ? qy[j] : nan,
                                      __uint_as_float(uint32_t(qfl >> (6 * j)) & 63u), __uint_as_float(qid[j]));
                s_fd[k] = 0.0;
            }
        }
        __syncthreads();
        if constexpr (kTrim) {
            // bounding box of this warp's queries in the bin's frame
            float bx0 = INFINITY, bx1 = -INFINITY, by0 = INFINITY, by1 = -INFINITY;
#pragma unroll
            for (int j = 0; j < QPT; ++j) {
                if (!qv[j]) continue;
                bx0 = fminf(bx0, qx[j]);
                bx1 = fmaxf(bx1, qx[j]);
                by0 = fminf(by0, qy[j]);
                by1 = fmaxf(by1, qy[j]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                bx0 = fminf(bx0, __shfl_xor_sync(0xffffffffu, bx0, o));
                bx1 = fmaxf(bx1, __shfl_xor_sync(0xffffffffu, bx1, o));
                by0 = fminf(by0, __shfl_xor_sync(0xffffffffu, by0, o));
                by1 = fmaxf(by1, __shfl_xor_sync(0xffffffffu, by1, o));
            }
            if ((tid & 31) == 0) s_wb[tid >> 5] = make_float4(bx0 - s_ox, bx1 - s_ox, by0 - s_oy, by1 - s_oy);
            // the warp's lanes read the box below, possibly before any CTA barrier
            // (a first batch issued with the walk skips the planning barrier)
            __syncwarp();
        }

        for (;;) {
            // s_pre: this batch was planned and issued with the walk (read after a
            // barrier, cleared by thread 0 once every thread is past the next one)
            if (!s_pre) {
            if (tid == 0) {
                // next batch: whole or partial pieces up to the staging capacity
                int pc = s_cur_piece;
                uint32_t po = s_cur_off, tot = 0;
                int nb = 0;
                while (pc < s_np && tot < uint32_t(kCap) && nb < kMaxPieces + 2) {
                    const uint32_t rem = s_pc[pc].cnt - po;
                    const uint32_t take = min(rem, uint32_t(kCap) - tot);
                    s_bp[nb++] = BatchPiece{tot, take, s_pc[pc].gstart + po, pc};
                    tot += take;
                    po += take;
                    if (po == s_pc[pc].cnt) { ++pc; po = 0; }
                }
                s_cur_piece = pc;
                s_cur_off = po;
                s_nbp = nb;
                s_btot = tot;
                if (tot > 0) {
                    fence_proxy_async_smem();
                    mbar_arrive_expect_tx(&s_bar, tot * kRec);
                    const char* gsrc = kDef ? reinterpret_cast<const char*>(a.candf)
                                            : reinterpret_cast<const char*>(a.cand);
                    for (int b = 0; b < nb; ++b)
                        bulk_g2s(reinterpret_cast<char*>(s_cand) + size_t(s_bp[b].soff) * kRec,
                                 gsrc + size_t(s_bp[b].gstart) * kRec, s_bp[b].cnt * kRec, &s_bar);
                }
            }
            __syncthreads();
            }
            if (s_btot == 0) break;
            if constexpr (kTrim) {
                // this warp's part of each staged run: the sub-rows within reach of
                // its queries' bounding box (reach widened by 0.1%, sub-row bounds by
                // 1% of a sub-row, so no pair with a non-zero term is dropped: the
                // sums equal those over the whole runs).  The sub-row starts are read
                // while the bulk copy is in flight.
                if (npw > 0) {
                    const int wid = tid >> 5;
                    const float4 bb = s_wb[wid];
                    const float sxw = 1.f / G.inv_sx, inv_srow = G.inv_sy * float(a.rows);
                    const float rm = G.reach * 1.001f;
                    for (int b = tid & 31; b < s_nbp; b += 32) {
                        const BatchPiece bp = s_bp[b];
                        const Piece pc = s_pc[bp.piece];
                        uint32_t lo = 0u, hi = 0u;
                        const float dxw = fmaxf(0.f, fmaxf(pc.x0 - bb.y, bb.x - (pc.x0 + sxw)));
                        if (dxw < rm) {
                            const float dy = sqrtf(fmaf(rm, rm, -dxw * dxw));
                            const int ilo = max(int(floorf(fmaf(bb.z - dy - pc.y0, inv_srow, -0.01f))), 0);
                            const int ihi = min(int(floorf(fmaf(bb.w + dy - pc.y0, inv_srow, 0.01f))), int(pc.nr) - 1);
                            if (ilo <= ihi) {
                                const uint32_t t0 = a.cstart[pc.b0 + uint32_t(ilo)];
                                const uint32_t t1 = a.cstart[pc.b0 + uint32_t(ihi) + 1u];
                                const uint32_t g0 = bp.gstart, g1 = bp.gstart + bp.cnt;
                                lo = min(max(t0, g0), g1) - g0;
                                hi = max(min(max(t1, g0), g1) - g0, lo);
                            }
                        }
                        s_rng[wid][b] = make_uint2(lo, hi);
                    }
                }
            }
            // each thread sees the copied bytes once its own wait completes; the
            // packed modes rewrite them first, so their barrier follows that pass
            if (!mbar_wait_bounded(&s_bar, phase, a.wait_limit)) atomicOr(&s_abort, 1);
            phase ^= 1u;
            if constexpr (!kPacked && !kField64) {
                __syncthreads();
                if (tid == 0) s_pre = 0;
                if (s_abort) break;
            }

            const int nbp = s_nbp;
            if constexpr (kScat)
                scat_batch<ST, kScat9>(s_cand, s_bp, s_pc, nbp, s_rng[0], s_sq, s_sqm, min(int(it.qcnt), kScatQ), G,
                                       a.out_f64);
            if constexpr (kPacked) {
                // staged candidates -> image-shifted, bin-local coordinates + kappa c2
                // (kappa = -3/h^2 scales every squared distance, see packed_run)
                const float kap = G.B;
                for (int b = 0; b < nbp; ++b) {
                    const BatchPiece bp = s_bp[b];
                    const Piece pc = s_pc[bp.piece];
                    const float ox = s_ox + pc.qdx, oy = s_oy + pc.qdy;
                    for (uint32_t c = threadIdx.x; c < bp.cnt; c += kEvalThreads) {
                        if constexpr (kDef) {
                            float* f = s_candf[bp.soff + c].f;
                            const float lx = f[0] - ox, ly = f[1] - oy;
                            const float g11 = f[2], g12 = f[3], g22 = f[4], w = f[5];
                            const float gx = fmaf(g11, lx, g12 * ly), gy = fmaf(g12, lx, g22 * ly);
                            const float e = kap * fmaf(lx, gx, ly * gy);
                            f[0] = kap * g11; f[1] = f[0];
                            f[2] = kap * (2.f * g12); f[3] = f[2];
                            f[4] = kap * g22; f[5] = f[4];
                            f[6] = kap * (-2.f * gx); f[7] = f[6];
                            f[8] = kap * (-2.f * gy); f[9] = f[8];
                            f[10] = e; f[11] = e;
                            f[12] = w; f[13] = w;
                            f[14] = 0.f; f[15] = 0.f;
                        } else {
                            Cand& cd = s_cand[bp.soff + c];
                            const float lx = cd.x - ox, ly = cd.y - oy;
                            const float c2 = kap * fmaf(lx, lx, ly * ly);
                            cd.x = lx;
                            cd.x2 = lx;
                            cd.y = ly;
                            cd.y2 = ly;
                            cd.wl = c2;
                            cd.pad = c2;
                        }
                    }
                }
                __syncthreads();
                if (tid == 0) s_pre = 0;
                if (s_abort) break;   // (a thread whose wait expired rewrote stale bytes: unused)
            }
            if constexpr (kField64) {
                static_assert(kEvalThreads == 32, "one warp an item");
                // candidates -> the image of their run, exactly (two floats); the weights'
                // range, and whether every difference within reach is one float
                const float h3 = 2.f * G.half_h3[0], near = G.reach * 1.01f;
                float most = 0.f, least = INFINITY;
                bool finite = true, exact = true;
                for (int b = 0; b < nbp; ++b) {
                    const BatchPiece bp = s_bp[b];
                    const Piece pc = s_pc[bp.piece];
                    for (uint32_t c = threadIdx.x; c < bp.cnt; c += kEvalThreads) {
                        Cand& cd = s_cand[bp.soff + c];
                        float xh, xl, yh, yl;
                        wide::two_sum(cd.x, -pc.qdx, xh, xl);
                        wide::two_sum(cd.y, -pc.qdy, yh, yl);
                        cd.x = xh;
                        cd.x2 = xl;
                        cd.y = yh;
                        cd.y2 = yl;
                        const float a = fabsf(cd.w);
                        finite = finite && a <= 3.0e38f;
                        most = fmaxf(most, a);
                        if (a > 0.f) least = fminf(least, a);
                        exact = exact && xl == 0.f && yl == 0.f && fabsf(xh) >= near && fabsf(yh) >= near;
                    }
                }
#pragma unroll
                for (int j = 0; j < QPT; ++j) exact = exact && (!qv[j] || (fabsf(qx[j]) >= near && fabsf(qy[j]) >= near));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
                    least = fminf(least, __shfl_xor_sync(0xffffffffu, least, o));
                }
                // weights times a power of two: the largest product h^3 w is about 1, and the
                // smallest keeps its three floats above the underflow
                const int ex = min(max(254 - int(__float_as_uint(most) >> 23) + 127 - int(__float_as_uint(h3) >> 23), 1), 253);
                const float scale = __uint_as_float(uint32_t(ex) << 23);
                const bool fits = __all_sync(0xffffffffu, finite) && G.hw >= 1e-6f && G.hw <= 1e6f &&
                                  (most == 0.f || (least * scale * h3 >= 1e-20f && most * scale * h3 <= 1e20f));
                exact = __all_sync(0xffffffffu, exact);
                __syncthreads();
                if (tid == 0) s_pre = 0;
                if (s_abort) break;   // (a thread whose wait expired rewrote stale bytes: unused)
                if (fits)
                    for (uint32_t c = threadIdx.x; c < s_btot; c += kEvalThreads) {
                        s_cand[c].w *= scale;
                        s_cand[c].wl *= scale;
                    }
                __syncthreads();
                const double unit = G.inv_h3 / double(scale);
                const float lim = G.hw * G.hw * 1.00001f;
                const wide::W3 half_h3{G.half_h3[0], G.half_h3[1], G.half_h3[2]};
#pragma unroll 1
                for (int j = 0; j < 2 * npw; ++j) {
                    const int k = j * 32 + (tid & 31);
                    const float4 q = s_fq[k];
                    const uint32_t fl = __float_as_uint(q.z);
                    wide::W3 acc3{0.f, 0.f, 0.f};
                    double accd = 0.0;
#pragma unroll 1
                    for (int b = 0; b < nbp; ++b) {
                        const uint2 rg = s_rng[0][b];
                        const BatchPiece bp = s_bp[b];
                        if (kField9) {
                            const Piece pc = s_pc[bp.piece];
                            const int mx = int(fl & 7u) - 2 + pc.mx, my = int((fl >> 3) & 7u) - 2 + pc.my;
                            if (!(mx >= -1 && mx <= 1 && my >= -1 && my <= 1)) continue;
                        }
                        const Cand* cs = s_cand + bp.soff + rg.x;
                        const int cnt = int(rg.y) - int(rg.x);
                        if (fits && exact) wide_run<false>(cs, cnt, q.x, q.y, G.hw, lim, half_h3, acc3);
                        else if (fits) wide_run<true>(cs, cnt, q.x, q.y, G.hw, lim, half_h3, acc3);
                        else {
                            const double ih = 1.0 / double(G.hw), A = 3.0 * ih * ih * ih, B = -3.0 * ih * ih;
                            const double px = q.x, py = q.y;
                            for (int c = 0; c < cnt; ++c) {
                                const Cand cv = cs[c];
                                const double dx = (double(cv.x) + double(cv.x2)) - px;
                                const double dy = (double(cv.y) + double(cv.y2)) - py;
                                const double r2 = dx * dx + dy * dy, r = sqrt(r2);
                                const double inner = 0.5 + r2 * (A * r + B), t = 1.0 - ih * r;
                                accd += (double(cv.w) + double(cv.wl)) * fmax(fmin(inner, t * t * t), 0.0);
                            }
                        }
                    }
                    if (fits) accd = ((double(acc3.a) + double(acc3.b)) + double(acc3.c)) * unit;
                    s_fd[k] += accd;
                }
            }
            for (int b = 0; b < (kScat || kField64 ? 0 : nbp); ++b) {
                const BatchPiece bp = s_bp[b];
                const Piece pc = s_pc[bp.piece];
                int cnt = int(bp.cnt);
                const int bfirst = b;
                if constexpr (kPacked) {
                    // staged runs sit back to back in shared memory, already in the
                    // bin's frame: consecutive runs under the same image mask are one
                    // sweep (each warp visits its own part of each run, in run order)
                    while (b + 1 < nbp) {
                        const Piece nx = s_pc[s_bp[b + 1].piece];
                        if (kField9 && (nx.mx != pc.mx || nx.my != pc.my)) break;
                        cnt += int(s_bp[b + 1].cnt);
                        ++b;
                    }
                }
                const Cand* cs = s_cand + bp.soff;
                Acc part[QPT];
                if constexpr (kPacked && kDef) {
                    // queries in the local frame: the monomials of the expanded metric form
                    f2x QXX[NP], QXY[NP], QYY[NP], QX[NP], QY[NP], P[NP];
#pragma unroll
                    for (int pr = 0; pr < NP; ++pr) {
                        const float ax = qx[2 * pr] - s_ox, bx = qx[2 * pr + 1] - s_ox;
                        const float ay = qy[2 * pr] - s_oy, by = qy[2 * pr + 1] - s_oy;
                        QXX[pr] = pk2(ax * ax, bx * bx);
                        QXY[pr] = pk2(ax * ay, bx * by);
                        QYY[pr] = pk2(ay * ay, by * by);
                        QX[pr] = pk2(ax, bx);
                        QY[pr] = pk2(ay, by);
                        P[pr] = pk2(0.f, 0.f);
                    }
                    for (int gb = bfirst; gb <= b && npw > 0; ++gb) {
                        const uint2 rg = s_rng[tid >> 5][gb];
                        const int n = int(rg.y) - int(rg.x);
                        if (n <= 0) continue;
                        const CandF* csf = s_candf + s_bp[gb].soff + rg.x;
                        if (npw == 1) packed_run_f<1, NP>(csf, n, QXX, QXY, QYY, QX, QY, P);
                        else if (NP >= 2 && npw == 2)
                            packed_run_f<(NP >= 2 ? 2 : 1), NP>(csf, n, QXX, QXY, QYY, QX, QY, P);
                        else packed_run_f<NP, NP>(csf, n, QXX, QXY, QYY, QX, QY, P);
                    }
#pragma unroll
                    for (int pr = 0; pr < NP; ++pr) {
                        float lo, hi;
                        up2(P[pr], lo, hi);
                        part[2 * pr] = lo;
                        part[2 * pr + 1] = hi;
                    }
                } else if constexpr (kPacked) {
                    // queries in the same local frame: -2 kappa q and kappa |q|^2
                    f2x QX[NP], QY[NP], Q2[NP], P[NP];
                    const float kap = G.B, m2k = -2.f * G.B;
#pragma unroll
                    for (int pr = 0; pr < NP; ++pr) {
                        const float ax = qx[2 * pr] - s_ox, bx = qx[2 * pr + 1] - s_ox;
                        const float ay = qy[2 * pr] - s_oy, by = qy[2 * pr + 1] - s_oy;
                        QX[pr] = pk2(m2k * ax, m2k * bx);
                        QY[pr] = pk2(m2k * ay, m2k * by);
                        Q2[pr] = pk2(kap * fmaf(ax, ax, ay * ay), kap * fmaf(bx, bx, by * by));
                        P[pr] = pk2(0.f, 0.f);
                    }
                    // a warp with few queries runs fewer pairs (none when it holds no query)
                    for (int gb = bfirst; gb <= b && npw > 0; ++gb) {
                        const uint2 rg = s_rng[tid >> 5][gb];
                        const int n = int(rg.y) - int(rg.x);
                        if (n <= 0) continue;
                        const Cand* c0 = s_cand + s_bp[gb].soff + rg.x;
                        if (npw == 1) packed_run<1, NP>(c0, n, QX, QY, Q2, P);
                        else if (NP >= 2 && npw == 2) packed_run<(NP >= 2 ? 2 : 1), NP>(c0, n, QX, QY, Q2, P);
                        else packed_run<NP, NP>(c0, n, QX, QY, Q2, P);
                    }
#pragma unroll
                    for (int pr = 0; pr < NP; ++pr) {
                        float lo, hi;
                        up2(P[pr], lo, hi);
                        part[2 * pr] = lo;
                        part[2 * pr + 1] = hi;
                    }
                } else if constexpr (kDefExc) {
                    // deformed kernels, differences taken directly (an exact zero
                    // for coincident points, so the centre test is reliable)
                    float px[QPT], py[QPT];
#pragma unroll
                    for (int j = 0; j < QPT; ++j) {
                        px[j] = qx[j] + pc.qdx;
                        py[j] = qy[j] + pc.qdy;
                        part[j] = Acc(0);
                    }
                    const float A = G.A, B = G.B, ih = G.inv_hw;
                    const CandF* csf = s_candf + bp.soff;
                    for (int c = 0; c < cnt; ++c) {
                        const float cx = csf[c].f[0], cy = csf[c].f[1];
                        const float g11 = csf[c].f[2], g12 = csf[c].f[3], g22 = csf[c].f[4], cw = csf[c].f[5];
#pragma unroll
                        for (int j = 0; j < QPT; ++j) {
                            const float dx = cx - px[j], dy = cy - py[j];
                            const float r2 = fmaf(g11 * dx, dx, fmaf(2.f * g12 * dx, dy, g22 * dy * dy));
                            const float r = sqrtf(fmaxf(r2, 0.f));
                            const float inner = fmaf(r2, fmaf(A, r, B), 0.5f);
                            const float t = fmaf(-ih, r, 1.0f);
                            float v = fmaxf(fminf(inner, t * t * t), 0.0f);
                            if (r < 1e-6f) v = 0.f;
                            part[j] = fmaf(cw, v, part[j]);
                        }
                    }
                } else if constexpr (kGrad32) {
                    const uint2 rg = s_rng[0][b];
                    f2x pxy[QPT], pg[QPT];
                    float pv[QPT];
                    const float m3ih = -3.f * G.inv_hw;
#pragma unroll
                    for (int j = 0; j < QPT; ++j) {
                        pxy[j] = pk2(qx[j] + pc.qdx, qy[j] + pc.qdy);
                        pg[j] = pk2(0.f, 0.f);
                        pv[j] = 0.f;
                    }
                    if (npw == 1) grad32_run<2>(cs + rg.x, int(rg.y) - int(rg.x), pxy, G, pv, pg);
                    else grad32_run<QPT>(cs + rg.x, int(rg.y) - int(rg.x), pxy, G, pv, pg);
#pragma unroll
                    for (int j = 0; j < QPT; ++j) {
                        bool use = (j >> 1) < npw;
                        if (kGrad9) {
                            const int mx = int(uint32_t(qfl >> (6 * j)) & 7u) - 2 + pc.mx;
                            const int my = int(uint32_t(qfl >> (6 * j + 3)) & 7u) - 2 + pc.my;
                            use = use && mx >= -1 && mx <= 1 && my >= -1 && my <= 1;
                        }
                        if (!use) continue;
                        float gx, gy;
                        up2(pg[j], gx, gy);
                        wide::add_float(sums[3 * j], pv[j]);
                        wide::add_float(sums[3 * j + 1], m3ih * gx);
                        wide::add_float(sums[3 * j + 2], m3ih * gy);
                    }
                } else if constexpr (kGrad) {
                    // value and gradient in q of sum w W(|q - c|), pair by pair in FP64:
                    // dW/dr / r = 2 sigma (3 A r + 2 B) for r < h/2, -6 sigma t^2/(h r) below h
                    const GT hw = GT(G.hw), ih = GT(1) / hw;
                    const GT A = GT(3) * ih * ih * ih, B = GT(-3) * ih * ih;
                    GT px[QPT], py[QPT], pv[QPT], pgx[QPT], pgy[QPT];
                    bool use[QPT];
#pragma unroll
                    for (int j = 0; j < QPT; ++j) {
                        px[j] = GT(qx[j]) + GT(pc.qdx);
                        py[j] = GT(qy[j]) + GT(pc.qdy);
                        pv[j] = pgx[j] = pgy[j] = GT(0);
                        use[j] = true;
                        if (kGrad9) {
                            const int mx = int(uint32_t(qfl >> (6 * j)) & 7u) - 2 + pc.mx;
                            const int my = int(uint32_t(qfl >> (6 * j + 3)) & 7u) - 2 + pc.my;
                            use[j] = mx >= -1 && mx <= 1 && my >= -1 && my <= 1;
                        }
                    }
                    for (int c = 0; c < cnt; ++c) {
                        const Cand cv = cs[c];
                        const GT cxd = cv.x, cyd = cv.y;
                        const GT wd = GT(double(cv.w) + double(cv.wl));
#pragma unroll
                        for (int j = 0; j < QPT; ++j) {
                            const GT dx = px[j] - cxd, dy = py[j] - cyd;   // q - c
                            const GT r2 = dx * dx + dy * dy;
                            const GT r = sqrt(r2);
                            if (r >= hw) continue;
                            const GT t = GT(1) - ih * r;
                            GT v, dr;   // W / 2 sigma and its r-derivative over r
                            if (r <= GT(0.5) * hw) {
                                v = GT(0.5) + r2 * (A * r + B);
                                dr = GT(3) * A * r + GT(2) * B;
                            } else {
                                v = t * t * t;
                                dr = GT(-3) * t * t * ih / r;
                            }
                            pv[j] += wd * v;
                            pgx[j] += wd * dr * dx;
                            pgy[j] += wd * dr * dy;
                        }
                    }
#pragma unroll
                    for (int j = 0; j < QPT; ++j) {
                        if (!use[j]) continue;
                        acc[j] += double(pv[j]);
                        accg[j][0] += double(pgx[j]);
                        accg[j][1] += double(pgy[j]);
                        part[j] = 0.0;
                    }
                } else if constexpr (kF64) {
                    float px[QPT], py[QPT];
#pragma unroll
                    for (int j = 0; j < QPT; ++j) {
                        px[j] = qx[j] + pc.qdx;
                        py[j] = qy[j] + pc.qdy;
                        part[j] = Acc(0);
                    }
                    const double hw = double(G.hw);
                    const float lim = G.hw * G.hw * 1.0001f;
#pragma unroll 2
                    for (int c = 0; c < cnt; ++c) {
                        const Cand cv = cs[c];
#pragma unroll
                        for (int j = 0; j < QPT; ++j) {
                            const float dx = cv.x - px[j], dy = cv.y - py[j];
                            if (dx * dx + dy * dy < lim) {
                                const double ddx = double(cv.x) - (double(qx[j]) + double(pc.qdx));
                                const double ddy = double(cv.y) - (double(qy[j]) + double(pc.qdy));
                                const double r = sqrt(ddx * ddx + ddy * ddy);
                                part[j] += (double(cv.w) + double(cv.wl)) * spline_w_d(r, hw);
                            }
                        }
                    }
                } else {
                    float px[QPT], py[QPT];
#pragma unroll
                    for (int j = 0; j < QPT; ++j) {
                        px[j] = qx[j] + pc.qdx;
                        py[j] = qy[j] + pc.qdy;
                        part[j] = Acc(0);
                    }
                    const float A = G.A, B = G.B, ih = G.inv_hw;
#pragma unroll 4
                    for (int c = 0; c < cnt; ++c) {
                        const float cx = cs[c].x, cy = cs[c].y, cw = cs[c].w;
#pragma unroll
                        for (int j = 0; j < QPT; ++j) {
                            const float dx = cx - px[j], dy = cy - py[j];
                            const float r2 = fmaf(dx, dx, fmaf(dy, dy, 1e-30f));
                            const float r = r2 * rsqrtf(r2);
                            const float inner = fmaf(r2, fmaf(A, r, B), 0.5f);
                            const float t = fmaf(-ih, r, 1.0f);
                            float v = fmaxf(fminf(inner, t * t * t), 0.0f);
                            if (MODE == EVAL_FIELD_EXC && r2 < 1e-12f) v = 0.f;
                            part[j] = fmaf(cw, v, part[j]);
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < QPT && !kGrad; ++j) {
                    bool use = true;
                    if (kField9) {
                        const int mx = int(uint32_t(qfl >> (6 * j)) & 7u) - 2 + pc.mx;
                        const int my = int(uint32_t(qfl >> (6 * j + 3)) & 7u) - 2 + pc.my;
                        use = mx >= -1 && mx <= 1 && my >= -1 && my <= 1;
                    }
                    if (use) {
                        if constexpr (kComp) {
                            // compensated accumulation of the per-run partial sums
                            const float y = float(part[j]) - acc_c[j];
                            const float tt = float(acc[j]) + y;
                            acc_c[j] = (tt - float(acc[j])) - y;
                            acc[j] = tt;
                        } else {
                            acc[j] += part[j];
                        }
                    }
                }
            }
            // no further batch in this item: the item's closing barrier guards the
            // staging buffer (the cursor only moves in the next planning step)
            if (s_cur_piece >= s_np) break;
            __syncthreads();   // all reads of s_cand done before the next batch overwrites it
        }
        if (s_abort) break;
#pragma unroll
        for (int j = 0; j < QPT && !kScat; ++j) {
            if (!qv[j]) continue;
            if constexpr (kGrad32) {
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    a.out_f32[3 * size_t(qid[j]) + k] = sums[3 * j + k][0] + (sums[3 * j + k][1] + sums[3 * j + k][2]);
            } else if constexpr (kGrad) {
                a.out_f64[3 * size_t(qid[j])] = acc[j];
                a.out_f64[3 * size_t(qid[j]) + 1] = accg[j][0];
                a.out_f64[3 * size_t(qid[j]) + 2] = accg[j][1];
            } else if constexpr (kField64) {
                const int k = j * 32 + (tid & 31);
                a.out_f64[qid[j]] = s_fd[k];
            } else if constexpr (kF64) a.out_f64[qid[j]] = acc[j];
            else if constexpr (kComp) a.out_f64[qid[j]] = double(acc[j]) - double(acc_c[j]);
            else a.out_f32[qid[j]] = acc[j];
        }
        if (tid == 0) s_item = next_item;
        __syncthreads();
    }
    if (s_abort) {
        if (tid == 0) {
            atomicOr(a.flags, FLAG_TIMEOUT);
            (void)mbar_wait_bounded(&s_bar, phase ^ 1u, kWaitLimit);   // let an in-flight copy land
        }
    }
}

template <int MODE, int QPT>
int launch_eval_t(vpmc_context* ctx, const EvalArgs& a) {
    const size_t smem = size_t(kCandCap) * sizeof(Cand);
    static bool configured[64] = {};
    const int dev = ctx->device;
    if (dev < 64 && !configured[dev]) {
        VPMC_CUDA(cudaFuncSetAttribute(k_eval<MODE, QPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        configured[dev] = true;
    }
    int per_sm = 0;
    VPMC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_eval<MODE, QPT>, kEvalThreads, smem));
    if (per_sm < 1) per_sm = 1;
    const int grid = ctx->sm_count * per_sm;
    VPMC_LAUNCH((k_eval<MODE, QPT>), grid, kEvalThreads, smem, ctx->stream, a);
    return VPMC_OK;
}

int blocks_for(long n, int threads = 256) {
    long b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 65535L * 16) b = 65535L * 16;
    return int(b);
}

}  // namespace

int default_k() { return 2; }

// Cells of about 2.6 particle spacings (both signs: 7 particles), as long as a bin
// still gathers 150 samples: smaller cells trim the walk closer to the disk of
// radius h_w, but each bin costs a walk, a sort key and its items.  Measured (ms a
// step, k = 2 -> the rule's k): 512^2, h_w 16 spacings, 64 + 64 samples: 27.0 -> 19.4
// (k = 6; best 18.9 at 7); 256^2, h_w 8, 32 + 32: 1.25 -> 1.18 (3, the best); 24
// ensemble members, h_w 8: 27.0 -> 25.5 (3); 256^2, h_w 4, 16 + 16: 0.52 -> 0.50 (1).
// The rule looks at one instance alone, so that a member of an ensemble sums as a
// run of its own does.  The samples of an open domain crowd its middle, so that the bins
// further out are thin: 250 are asked for there for more than two cells (1024^2, h_w 16, 16 + 16 samples: 12.3 ms
// with the 6 cells of 150, 11.3 with the 4 of 250; two cells 11.9).
int sample_k(long n, double samples, float Lx, float Ly, float hw, bool boxes, double fill) {
    if (n < 1) return default_k();
    const double spacing = std::sqrt(double(Lx) * Ly / double(n));
    int k = int(std::lround(double(hw) / (2.6 * spacing)));
    k = std::min(std::max(k, 1), kMaxK);
    for (; k > 1; --k) {
        const double cells = double(k) * Lx / hw * (double(k) * Ly / hw);
        if (samples >= (k > 2 ? fill : kBinFill) * cells && cells <= double(1L << 22)) break;
    }
    // where the pairwise choice has boxes too thin for local expansions, 7 cells may not:
    // their quadrants (h_w / 14 a side) are the largest boxes the expansions take
    // (512^2, h_w 16, 32 + 32 samples: a step takes 10.3 ms with 6 cells pair by pair, 5.8 with 7)
    if (boxes) {
        auto split = [&](int kk) {
            const double gx = std::floor(double(kk) * Lx / hw + 1e-9), gy = std::floor(double(kk) * Ly / hw + 1e-9);
            return gx >= 1.0 && gy >= 1.0 && gx * gy <= double(1L << 22) ? box_split(n, samples, Lx, Ly, hw, int(gx), int(gy)) : 0;
        };
        if (!split(k) && split(7)) return 7;
    }
    return k;
}

int query_chunk(int qpt) { return (qpt == 8 ? 8 : qpt == 6 ? 6 : 4) * kEvalThreads; }   // qpt 1 (tensor cores): 128

namespace {
// Cells of a plan: the first of k, k - 1, ..., 1 a h_w whose walk does not meet itself (no
// cells: the domain is too small for any).  Where none fits, once more with h_w 2^-22
// shorter: h_w = (Lx / Nx) hwr carries up to two FP32 roundings, and a period of 2.5 h_w
// is not refused for them (pairs in the sliver have no FP32 weight).
struct Cells {
    int k = 0, gx = 0, gy = 0;
};
Cells plan_cells(const InstDesc& d, double reach, int k) {
    for (const double r : {reach, reach * (1.0 - 0x1p-22)}) {
        Cells c;
        for (c.k = k; c.k >= 1; --c.k) {
            c.gx = int(std::floor(double(c.k) * double(d.Lx) / r + 1e-9));
            c.gy = int(std::floor(double(c.k) * double(d.Ly) / r + 1e-9));
            if (!d.periodic || (c.gx >= 2 * c.k + 1 && c.gy >= 2 * c.k + 1)) break;
        }
        if (c.k >= 1 && c.gx >= 1 && c.gy >= 1) return c;
    }
    return Cells{};
}
constexpr long kMaxCells = 1L << 24;
constexpr long kMaxBins = 1L << 31;
}  // namespace

// The library's own choice of cells decides how fast a sum is, never whether a domain is
// accepted: that is the default walk's doing, whose cells are taken wherever the chosen
// ones do not fit (a period of 2.5 to 3 h_w, or an open domain between 0.5 and 1 h_w
// wide, has room for two cells a h_w and not for one).
long grid_plan(const InstDesc* in, int n, int k, int nsets, GridInst* out) {
    if (k > kMaxK) k = kMaxK;
    std::vector<Cells> cells(static_cast<size_t>(n));
    long bins = 0;
    for (int i = 0; i < n; ++i) {
        const InstDesc& d = in[i];
        if (!(d.hw > 0.f) || !(d.Lx > 0.f) || !(d.Ly > 0.f)) return -VPMC_ERR_INVALID;
        if (!(d.cover >= 1.f)) return -VPMC_ERR_INVALID;
        const double reach = double(d.hw) * double(d.cover);   // physical support radius to cover
        cells[size_t(i)] = plan_cells(d, reach, k > 0 ? k : default_k());
        const Cells& c = cells[size_t(i)];
        if (c.k < 1) return -VPMC_ERR_GEOMETRY;
        if (long(c.gx) * c.gy > kMaxCells) return -VPMC_ERR_CAPACITY;
        bins += long(nsets) * c.gx * c.gy;
        if (bins >= kMaxBins) return -VPMC_ERR_CAPACITY;
    }
    if (k <= 0)
        for (int i = 0; i < n; ++i) {
            if (in[i].k < 1) continue;
            Cells& c = cells[size_t(i)];
            const Cells own = plan_cells(in[i], double(in[i].hw) * double(in[i].cover), std::min(in[i].k, kMaxK));
            const long more = long(nsets) * (long(own.gx) * own.gy - long(c.gx) * c.gy);
            if (own.k < 1 || long(own.gx) * own.gy > kMaxCells || bins + more >= kMaxBins) continue;
            c = own;
            bins += more;
        }
    long base = 0;
    for (int i = 0; i < n; ++i) {
        const InstDesc& d = in[i];
        const Cells& c = cells[size_t(i)];
        GridInst g{};
        g.Lx = d.Lx;
        g.Ly = d.Ly;
        g.gx = c.gx;
        g.gy = c.gy;
        g.inv_sx = float(c.gx) / d.Lx;
        g.inv_sy = float(c.gy) / d.Ly;
        g.k = c.k;
        g.bin_base = int(base);
        g.nsets = nsets;
        g.periodic = d.periodic;
        g.hw = d.hw;
        g.reach = float(double(d.hw) * double(d.cover));
        const double h = d.hw;
        g.inv_hw = float(1.0 / h);
        g.A = float(3.0 / (h * h * h));
        g.B = float(-3.0 / (h * h));
        g.two_sigma = float(2.0 * 40.0 / (7.0 * kPiD * h * h));
        g.p_begin = d.p_begin;
        g.p_end = d.p_end;
        // h^3 / 2 exactly (72 bits) as three floats: h^2 is exact in FP64, its product
        // with h as a value and an error
        const double h2 = h * h, hh = h2 * h * 0.5, he = std::fma(h2, h * 0.5, -hh);
        g.half_h3[0] = float(hh);
        g.half_h3[1] = float((hh - double(g.half_h3[0])) + he);
        g.half_h3[2] = float(((hh - double(g.half_h3[0])) - double(g.half_h3[1])) + he);
        g.inv_h3 = 1.0 / (h * h * h);
        out[i] = g;
        base += long(nsets) * c.gx * c.gy;
    }
    return base;
}

void carve_grid(Carver& c, long n, long nbins, int n_inst, GridBufs* g, bool deformed, int rows, bool records) {
    g->inst = c.take<GridInst>(size_t(n_inst));
    g->n_inst = n_inst;
    g->nbins = nbins;
    g->rows = rows < 1 ? 1 : rows;
    g->n = n;
    const long nsub = nbins * g->rows;
    g->keys = c.take<uint32_t>(size_t(n < 1 ? 1 : n));
    g->start = c.take<uint32_t>(size_t(nsub + 1));
    g->cstart = g->rows > 1 ? c.take<uint32_t>(size_t(nbins + 1)) : g->start;
    g->cand = records ? c.take<Cand>(size_t(n < 1 ? 1 : n)) : nullptr;
    g->candf = deformed ? c.take<CandF>(size_t(n < 1 ? 1 : n)) : nullptr;
    carve_radix(c, n, &g->rs);
}

int grid_sort(vpmc_context* ctx, GridBufs& g, const float2* pos, const float* omega, int set_mode) {
    cudaStream_t st = ctx->stream;
    const long nsub = g.nbins * g.rows;
    uint32_t *ks = g.keys, *vs = g.rs.vbuf[0];
    if (small_sort_fits(g.n, nsub + 1)) {
        static bool configured[64] = {};
        if (ctx->device < 64 && !configured[ctx->device]) {
            VPMC_CUDA(cudaFuncSetAttribute(k_grid_small, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmallSmem)));
            configured[ctx->device] = true;
        }
        VPMC_LAUNCH(k_grid_small, 1, kSmallThreads, small_sort_smem(g.n, nsub + 1), st, pos, omega, int(g.n), g.inst,
                    g.n_inst, set_mode, uint32_t(g.nbins), g.rows, bits_for(uint64_t(g.n)), g.start, g.cstart, vs);
    } else {
        VPMC_LAUNCH(k_grid_keys, blocks_for(g.n), 256, 0, st, pos, omega, g.n, g.inst, g.n_inst, set_mode,
                    uint32_t(g.nbins), g.rows, g.keys);
        VPMC_TRY(radix_sort(ctx, g.keys, nullptr, g.n, bits_for(uint64_t(nsub) + 1), g.rs, &ks, &vs));
        const int span = nsub < (1L << 20) ? 256 : 4096;
        VPMC_LAUNCH(k_grid_starts, blocks_for(nsub + 1, span), 256, 0, st, ks, uint32_t(g.n), nsub, g.rows, span, g.start,
                    g.cstart);
    }
    g.perm = vs;
    return VPMC_OK;
}

int grid_build(vpmc_context* ctx, GridBufs& g, const float2* pos, const float* omega, int set_mode,
               const float4* F, bool compact) {
    if (F && !g.candf) return VPMC_ERR_INVALID;
    cudaStream_t st = ctx->stream;
    VPMC_TRY(grid_sort(ctx, g, pos, omega, set_mode));
    const long nsub = g.nbins * g.rows;
    const uint32_t* vs = g.perm;
    if (F)
        VPMC_LAUNCH(k_grid_gather_f, blocks_for(g.n), 256, 0, st, vs, g.start, g.n, uint32_t(nsub), pos, omega, F,
                    g.inst, g.n_inst, set_mode, g.candf);
    else
        VPMC_LAUNCH(k_grid_gather, blocks_for(g.n), 256, 0, st, vs, g.start, g.n, uint32_t(nsub), pos, omega,
                    g.inst, g.n_inst, set_mode, g.cand, compact ? g.cand4 : nullptr);
    return VPMC_OK;
}

int grid_set_weights_sorted(vpmc_context* ctx, GridBufs& g, const double* x_sorted, double scale) {
    VPMC_LAUNCH(k_grid_weights, blocks_for(g.n), 256, 0, ctx->stream, x_sorted, g.n, scale, g.cand);
    return VPMC_OK;
}

int grid_max_sigma(vpmc_context* ctx, const float4* F, long n, unsigned* d_words, float* sigma) {
    cudaStream_t st = ctx->stream;
    VPMC_CUDA(cudaMemsetAsync(d_words, 0, 2 * sizeof(unsigned), st));
    if (n > 0)
        VPMC_LAUNCH(k_sigma, std::min(blocks_for(n), 4 * ctx->sm_count), 256, 0, st, F, n, d_words);
    unsigned h = 0u;
    VPMC_CUDA(cudaMemcpyAsync(&h, d_words, sizeof(h), cudaMemcpyDeviceToHost, st));
    VPMC_CUDA(cudaStreamSynchronize(st));
    float v;
    memcpy(&v, &h, sizeof(v));
    *sigma = n > 0 ? v : 1.f;
    return VPMC_OK;
}

void carve_items(Carver& c, long nbins, long max_queries, ItemBufs* it, long n_boxes, int chunk) {
    it->max_items = max_queries / chunk + (n_boxes < 0 ? nbins : n_boxes) + 1;
    it->items = c.take<Item>(size_t(it->max_items));
    it->n_items = c.take<uint32_t>(1);
    it->counter = c.take<uint32_t>(1);
    it->per_bin = c.take<uint32_t>(size_t(nbins + 1));
    it->item_start = c.take<uint32_t>(size_t(nbins + 1));
    it->scan_tmp = c.take<uint32_t>(scan_tmp_elems(nbins + 1) + 1);
}

namespace {
int make_items_of(vpmc_context* ctx, const GridBufs& g, const uint32_t* qstart, ItemBufs& it, int chunk, long queries,
                  int skip) {
    cudaStream_t st = ctx->stream;
    if (items_in_one(g.nbins, queries)) {
        VPMC_LAUNCH(k_items_small, 1, 1024, 0, st, static_cast<const uint32_t*>(nullptr), const_cast<uint32_t*>(qstart),
                    int(g.nbins), chunk, g.inst, g.n_inst, skip, it.items, it.n_items, it.counter, it.max_items);
        return VPMC_OK;
    }
    VPMC_LAUNCH(k_items_count, blocks_for(g.nbins), 256, 0, st, qstart, g.nbins, chunk, g.inst, g.n_inst, skip, it.per_bin);
    VPMC_TRY(exclusive_scan(ctx, it.per_bin, it.item_start, g.nbins, it.scan_tmp, true));
    VPMC_LAUNCH(k_items_fill, blocks_for(g.nbins), 256, 0, st, qstart, g.nbins, chunk, it.item_start, g.inst,
                g.n_inst, skip, it.items, it.n_items, it.counter, it.max_items);
    return VPMC_OK;
}
int make_box_items(vpmc_context* ctx, const GridBufs& g, const uint32_t* sstart, ItemBufs& it) {
    cudaStream_t st = ctx->stream;
    VPMC_LAUNCH(k_box_count, blocks_for(g.nbins), 256, 0, st, sstart, g.nbins, g.inst, g.n_inst, it.per_bin);
    VPMC_TRY(exclusive_scan(ctx, it.per_bin, it.item_start, g.nbins, it.scan_tmp, true));
    VPMC_LAUNCH(k_box_fill, blocks_for(g.nbins), 256, 0, st, sstart, g.nbins, it.item_start, g.inst, g.n_inst, it.items,
                it.n_items, it.counter, it.max_items);
    return VPMC_OK;
}
}  // namespace

int make_items(vpmc_context* ctx, const GridBufs& g, const uint32_t* qstart, ItemBufs& it, int chunk, long queries) {
    return make_items_of(ctx, g, qstart, it, chunk, queries, 0);
}

// Samples are placed directly up to this many a chunk (the records in L2), in
// three streaming passes beyond: a step of 0.26 M samples takes 105 us direct and
// 112 us staged, of 2.1 M 381 and 413 us, of 4.2 M 675 and 656 us.
constexpr long kDirectSamples = 1L << 21;
// Up to this many bins (32 MB of counters) the generator counts per (bin, sub-cell).
constexpr long kSubBins = 1L << 19;

void carve_queries(Carver& c, long nbins, long max_points, QueryBufs* q, bool samples, bool boxes) {
    const size_t m = size_t(max_points < 1 ? 1 : max_points);
    const bool sub = samples && nbins <= kSubBins, direct = sub && max_points <= kDirectSamples;
    const bool staged = samples && !direct;
    q->qbin = c.take<uint32_t>(m);
    // the counters that are zeroed for every pass lie together (clear_counts)
    const size_t n_sub = sub ? size_t(nbins) * kSubCells : 0, n_fill = staged ? size_t(nbins + 1) + kTargetSuper + 1 : 0;
    const size_t n_count = size_t(nbins + 1);
    uint32_t* counts = c.take<uint32_t>(n_sub + n_fill + n_count);
    q->qsub = sub ? counts : nullptr;
    q->super_fill = staged ? counts + n_sub : nullptr;
    q->win_fill = staged ? counts + n_sub + kTargetSuper + 1 : nullptr;
    q->qcount = counts + n_sub + n_fill;
    q->clear = counts;
    q->n_clear = n_sub + n_fill + (sub ? 0 : n_count);
    q->qstart = c.take<uint32_t>(size_t(nbins + 1));
    q->sstart = boxes ? c.take<uint32_t>(size_t(nbins) * kSubCells + 1) : nullptr;
    q->qfill = samples ? nullptr : c.take<uint32_t>(size_t(nbins + 1));
    q->qrank = direct ? c.take<uint32_t>(m) : nullptr;
    q->qrec = c.take<QRec>(m);
    q->tmp = staged ? c.take<uint4>(m) : nullptr;
    q->tmp2 = staged ? c.take<uint4>(m) : nullptr;
    q->scan_tmp = c.take<uint32_t>(scan_tmp_elems(nbins + 1) + 1);
}

int scatter_points(vpmc_context* ctx, const GridBufs& g, QueryBufs& q, const float2* pts, long M, int field9) {
    (void)field9;
    cudaStream_t st = ctx->stream;
    VPMC_TRY(exclusive_scan(ctx, q.qcount, q.qstart, g.nbins, q.scan_tmp, true));
    VPMC_CUDA(cudaMemsetAsync(q.qfill, 0, sizeof(uint32_t) * size_t(g.nbins + 1), st));
    VPMC_LAUNCH(k_scatter_points, blocks_for(M), 256, 0, st, pts, M, g.inst, g.n_inst, q.qbin, q.qstart, q.qfill,
                q.qrec);
    return VPMC_OK;
}

int clear_counts(vpmc_context* ctx, QueryBufs& q) {
    VPMC_CUDA(cudaMemsetAsync(q.clear, 0, sizeof(uint32_t) * q.n_clear, ctx->stream));
    return VPMC_OK;
}

int place_samples(vpmc_context* ctx, const GridBufs& g, QueryBufs& q, const float2* pts, long M, ItemBufs& it,
                  int chunk, ItemBufs* boxes) {
    cudaStream_t st = ctx->stream;
    const int skip = boxes ? 1 : 0;
    if (boxes && !q.sstart) return VPMC_ERR_INVALID;
    if (q.qrank && items_in_one(g.nbins, M)) {
        VPMC_LAUNCH(k_items_small, 1, 1024, 0, st, q.qsub, q.qstart, int(g.nbins), chunk, g.inst, g.n_inst, skip, it.items,
                    it.n_items, it.counter, it.max_items);
    } else {
        if (q.qsub) VPMC_LAUNCH(k_bin_totals, blocks_for(g.nbins), 256, 0, st, q.qsub, g.nbins, q.qcount);
        VPMC_TRY(exclusive_scan(ctx, q.qcount, q.qstart, g.nbins, q.scan_tmp, true));
        VPMC_TRY(make_items_of(ctx, g, q.qstart, it, chunk, M, skip));
    }
    if (q.qrank) {
        VPMC_LAUNCH(k_place_direct, blocks_for(M), 256, 0, st, pts, M, g.inst, g.n_inst, q.qbin, q.qrank, q.qstart, q.qsub,
                    q.qrec);
        if (!boxes) return VPMC_OK;
        VPMC_LAUNCH(k_sub_starts, blocks_for(g.nbins), 256, 0, st, q.qsub, q.qstart, g.nbins, q.sstart);
        return make_box_items(ctx, g, q.sstart, *boxes);
    }
    int shift = 0;
    while (((g.nbins - 1) >> shift) + 1 > kTargetSuper) ++shift;
    const int nsuper = int(((g.nbins - 1) >> shift) + 1);
    // windows of 2^W bins holding about half the assembly capacity on average, of the
    // smallest capacity that holds twice a bin and whose windows the second pass can
    // count (1.07 G samples in 1.6 M bins, windows of one bin, 3,136 a super-bin: that
    // pass reserves record by record, 18.8 ms; of two bins, 1,568: 8.8 ms)
    const double per_bin = double(M) / double(std::max<long>(g.nbins, 1));
    int asm_threads = 64, win_cap = 0, wshift = 0;
    do {
        asm_threads *= 2;
        win_cap = asm_threads * kAsmPer;
        wshift = 0;
        while ((1 << (wshift + 1)) <= kWinBinsMax && per_bin * double(2L << wshift) <= 0.5 * win_cap) ++wshift;
    } while (asm_threads < 512 && (per_bin > 0.5 * win_cap || (1L << std::max(shift - wshift, 0)) > kWinMax));
    const long nwin = ((g.nbins - 1) >> wshift) + 1;
    static bool configured[64] = {};
    const size_t tile_smem = sizeof(uint4) * size_t(kTileRecs), win_smem = sizeof(QRec) * size_t(win_cap);
    if (ctx->device < 64 && !configured[ctx->device]) {
        VPMC_CUDA(cudaFuncSetAttribute(k_scatter_coarse, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tile_smem)));
        VPMC_CUDA(cudaFuncSetAttribute(k_scatter_window, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tile_smem)));
        VPMC_CUDA(cudaFuncSetAttribute(k_scatter_assemble<256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(sizeof(QRec)) * 256 * kAsmPer));
        VPMC_CUDA(cudaFuncSetAttribute(k_scatter_assemble<512>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(sizeof(QRec)) * 512 * kAsmPer));
        configured[ctx->device] = true;
    }
    const long tiles = (M + kTileRecs - 1) / kTileRecs;
    const int tgrid = int(std::max<long>(1, std::min<long>(tiles, 2L * ctx->sm_count)));
    VPMC_LAUNCH(k_scatter_coarse, tgrid, kPlaceThreads, tile_smem, st, pts, M, q.qbin, q.qstart, shift, nsuper,
                q.super_fill, q.tmp);
    VPMC_LAUNCH(k_scatter_window, tgrid, kPlaceThreads, tile_smem, st, q.tmp, q.qstart + g.nbins, M, wshift, q.qstart,
                q.win_fill, q.tmp2);
    auto* const assemble = asm_threads == 128 ? k_scatter_assemble<128> : asm_threads == 256 ? k_scatter_assemble<256> : k_scatter_assemble<512>;
    VPMC_LAUNCH(assemble, int(std::max<long>(1, std::min<long>(nwin, (1024L / asm_threads) * ctx->sm_count))), asm_threads,
                win_smem, st, q.tmp2, g.nbins, wshift, q.qstart, g.inst, g.n_inst, q.qrec, boxes ? q.sstart : nullptr);
    return boxes ? make_box_items(ctx, g, q.sstart, *boxes) : int(VPMC_OK);
}

int bin_points(vpmc_context* ctx, const GridBufs& g, QueryBufs& q, const float2* pts, long M, int set, int field9) {
    cudaStream_t st = ctx->stream;
    VPMC_CUDA(cudaMemsetAsync(q.qcount, 0, sizeof(uint32_t) * size_t(g.nbins + 1), st));
    VPMC_LAUNCH(k_bin_points, blocks_for(M), 256, 0, st, pts, M, g.inst, set, field9, q.qbin, q.qcount);
    return scatter_points(ctx, g, q, pts, M, field9);
}

int launch_eval(vpmc_context* ctx, const GridBufs& g, const QRec* qrec, ItemBufs& it, const EvalLaunch& L) {
    if (eval_deformed(L.mode) && !g.candf) return VPMC_ERR_INVALID;
    if (eval_scat(L.mode) && (!L.qweight || !L.out_f64 || L.qpt != 4)) return VPMC_ERR_INVALID;
    if (L.qpt == 1 && (L.mode == EVAL_FIELD || L.mode == EVAL_FIELD9)) {
        const EvalTcArgs t{g.inst, g.start, L.rows > 0 ? L.rows : g.rows, g.cand, qrec, it.items, it.n_items,
                           it.counter, L.out_f32, ctx->d_flags, ctx->wait_limit};
        return launch_eval_tc(ctx, t, L.mode == EVAL_FIELD9);
    }
    EvalArgs a{g.inst, g.start, L.rows > 0 ? L.rows : g.rows, g.cand, g.candf, qrec, it.items, it.n_items, it.counter,
               L.out_f32, L.out_f64, ctx->d_flags, ctx->wait_limit, L.qweight};
    switch (L.mode) {
        case EVAL_FIELD:
            if (L.qpt == 8) return launch_eval_t<EVAL_FIELD, 8>(ctx, a);
            if (L.qpt == 6) return launch_eval_t<EVAL_FIELD, 6>(ctx, a);
            return launch_eval_t<EVAL_FIELD, 4>(ctx, a);
        case EVAL_FIELD9:
            if (L.qpt == 8) return launch_eval_t<EVAL_FIELD9, 8>(ctx, a);
            if (L.qpt == 6) return launch_eval_t<EVAL_FIELD9, 6>(ctx, a);
            return launch_eval_t<EVAL_FIELD9, 4>(ctx, a);
        case EVAL_FIELD_EXC:
            if (L.qpt != 4) return VPMC_ERR_INVALID;
            return launch_eval_t<EVAL_FIELD_EXC, 4>(ctx, a);
        case EVAL_SPMV64:
            if (L.qpt != 4) return VPMC_ERR_INVALID;
            return launch_eval_t<EVAL_SPMV64, 4>(ctx, a);
        case EVAL_SPMV32:
            if (L.qpt != 4) return VPMC_ERR_INVALID;
            return launch_eval_t<EVAL_SPMV32, 4>(ctx, a);
        case EVAL_FIELD_F:
            if (L.qpt == 8) return launch_eval_t<EVAL_FIELD_F, 8>(ctx, a);
            if (L.qpt == 6) return launch_eval_t<EVAL_FIELD_F, 6>(ctx, a);
            return launch_eval_t<EVAL_FIELD_F, 4>(ctx, a);
        case EVAL_FIELD9_F:
            if (L.qpt == 8) return launch_eval_t<EVAL_FIELD9_F, 8>(ctx, a);
            if (L.qpt == 6) return launch_eval_t<EVAL_FIELD9_F, 6>(ctx, a);
            return launch_eval_t<EVAL_FIELD9_F, 4>(ctx, a);
        case EVAL_FIELD_F_EXC:
            if (L.qpt != 4) return VPMC_ERR_INVALID;
            return launch_eval_t<EVAL_FIELD_F_EXC, 4>(ctx, a);
        case EVAL_GRAD64: return launch_eval_t<EVAL_GRAD64, 4>(ctx, a);
        case EVAL_GRAD9_64: return launch_eval_t<EVAL_GRAD9_64, 4>(ctx, a);
        case EVAL_GRAD32: return launch_eval_t<EVAL_GRAD32, 4>(ctx, a);
        case EVAL_GRAD9_32: return launch_eval_t<EVAL_GRAD9_32, 4>(ctx, a);
        case EVAL_SCAT64: return launch_eval_t<EVAL_SCAT64, 4>(ctx, a);
        case EVAL_SCAT9_64: return launch_eval_t<EVAL_SCAT9_64, 4>(ctx, a);
        case EVAL_SCAT32: return launch_eval_t<EVAL_SCAT32, 4>(ctx, a);
        case EVAL_SCAT9_32: return launch_eval_t<EVAL_SCAT9_32, 4>(ctx, a);
        case EVAL_FIELD64: return launch_eval_t<EVAL_FIELD64, 4>(ctx, a);
        case EVAL_FIELD9_64: return launch_eval_t<EVAL_FIELD9_64, 4>(ctx, a);
        default: return VPMC_ERR_INVALID;
    }
}

}  // namespace vpmc
