// sort.cu -- stable sorts of the particles' cell keys, and device-wide scans.
//
// Replaces the reference's unordered global atomics (src/mpm_solver3d.cu:
// 277-286): particles are ordered by (block, cell) key every step so that the
// P2G scatter can be done per block in a fixed order.  Every sort is stable (ties
// keep their previous order), hence bit-exact and deterministic, and all give
// the same order:
//   radixSortPairsInto   LSD radix sort with a histogram, a scan and a scatter
//                        kernel per 8-bit digit (mpm_sort_keys_device_noalloc)
//   radixSortOnesweep    one histogram kernel, then one kernel per digit whose
//                        tiles look back over one another's counts: a scene's
//                        first step, uploads, crowded blocks
//   block sort           from the last step's order: blocks put together from
//                        the particles that stayed and those that came, or by
//                        the radix passes in one launch where many moved
#include <cuda_runtime.h>
#include <stdint.h>

#include "engine_host.hpp"

#include <algorithm>

namespace mpm {

namespace {

constexpr int kScanItems = 16;                      // per thread
constexpr int kScanChunk = kThreads * kScanItems;   // 4096 per CTA
constexpr int kSortItems = kSortTileKeys / kThreads;
constexpr int kSortTile = kSortTileKeys;

template <class T>
__device__ __forceinline__ T warpInclusiveScan(T x) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// Exclusive scan across the 256 threads of a CTA; returns the CTA total in *total.
template <class T>
__device__ __forceinline__ T blockExclusiveScan(T x, T* total) {
    __shared__ T warp_tot[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T inc = warpInclusiveScan(x);
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        T t = lane < kWarps ? warp_tot[lane] : T(0);
        T ti = warpInclusiveScan(t);
        if (lane < kWarps) warp_tot[lane] = ti - t;
        // CTA total: inclusive value at the last warp
        T tl = __shfl_sync(0xffffffffu, ti, kWarps - 1);
        if (lane == 0) *total = tl;
    }
    __syncthreads();
    T r = inc - x + warp_tot[warp];
    __syncthreads();
    return r;
}

template <class T>
__global__ void __launch_bounds__(kThreads) scanReduceKernel(const T* in, size_t n, T* partials) {
    size_t base = (size_t)blockIdx.x * kScanChunk;
    T s = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        size_t i = base + (size_t)j * kThreads + threadIdx.x;
        if (i < n) s += in[i];
    }
    __shared__ T tot;
    (void)blockExclusiveScan(s, &tot);
    if (threadIdx.x == 0) partials[blockIdx.x] = tot;
}

// Single CTA exclusive scan of up to kScanChunk partials; writes the grand
// total to *total (if non-null).
template <class T>
__global__ void __launch_bounds__(kThreads) scanPartialsKernel(T* partials, int m, T* total) {
    T v[kScanItems];
    T s = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        int i = threadIdx.x * kScanItems + j;
        v[j] = i < m ? partials[i] : T(0);
        s += v[j];
    }
    __shared__ T tot;
    T run = blockExclusiveScan(s, &tot);
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        int i = threadIdx.x * kScanItems + j;
        if (i < m) partials[i] = run;
        run += v[j];
    }
    if (threadIdx.x == 0 && total) *total = tot;
}

template <class T>
__global__ void __launch_bounds__(kThreads) scanDownsweepKernel(const T* in, T* out, size_t n, const T* partials) {
    size_t base = (size_t)blockIdx.x * kScanChunk + (size_t)threadIdx.x * kScanItems;
    T v[kScanItems];
    T s = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        size_t i = base + j;
        v[j] = i < n ? in[i] : T(0);
        s += v[j];
    }
    __shared__ T tot;
    T run = blockExclusiveScan(s, &tot) + partials[blockIdx.x];
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        size_t i = base + j;
        if (i < n) out[i] = run;
        run += v[j];
    }
}

// --- radix sort -------------------------------------------------------------

__global__ void __launch_bounds__(kThreads) radixUpsweepKernel(const uint32_t* __restrict__ keys, uint32_t n,
                                                                int shift, uint32_t mask, uint32_t* __restrict__ hist,
                                                                int ntiles) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    size_t base = (size_t)blockIdx.x * kSortTile;
#pragma unroll 4
    for (int j = 0; j < kSortItems; ++j) {
        size_t i = base + (size_t)j * kThreads + threadIdx.x;
        bool valid = i < n;
        uint32_t d = valid ? (keys[i] >> shift) & mask : 0xffffffffu;
        uint32_t peers = __match_any_sync(0xffffffffu, d);
        int leader = __ffs(peers) - 1;
        if (valid && lane == leader) atomicAdd(&h[d], (uint32_t)__popc(peers));
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

template <bool kIdentVals>
__global__ void __launch_bounds__(kThreads) radixDownsweepKernel(const uint32_t* __restrict__ keys_in,
                                                                  const uint32_t* __restrict__ vals_in,
                                                                  uint32_t* __restrict__ keys_out,
                                                                  uint32_t* __restrict__ vals_out,
                                                                  const uint32_t* __restrict__ offsets, uint32_t n,
                                                                  int shift, uint32_t mask, int ntiles) {
    __shared__ uint32_t cnt[kWarps][256];
    for (int i = threadIdx.x; i < kWarps * 256; i += kThreads) (&cnt[0][0])[i] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const size_t base = (size_t)blockIdx.x * kSortTile + (size_t)warp * 32 * kSortItems;
    uint32_t k[kSortItems], v[kSortItems], r[kSortItems];
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        size_t i = base + (size_t)j * 32 + lane;
        bool valid = i < n;
        k[j] = valid ? keys_in[i] : 0u;
        v[j] = valid ? (kIdentVals ? (uint32_t)i : vals_in[i]) : 0u;
        uint32_t d = valid ? (k[j] >> shift) & mask : 256u;
        uint32_t peers = __match_any_sync(0xffffffffu, d);
        int leader = __ffs(peers) - 1;
        uint32_t before = valid ? cnt[warp][d] : 0u;
        r[j] = before + __popc(peers & lt);
        __syncwarp();
        if (valid && lane == leader) cnt[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            uint32_t c = cnt[w][threadIdx.x];
            cnt[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        size_t i = base + (size_t)j * 32 + lane;
        if (i < n) {
            uint32_t d = (k[j] >> shift) & mask;
            uint32_t pos = offsets[(size_t)d * ntiles + blockIdx.x] + cnt[warp][d] + r[j];
            keys_out[pos] = k[j];
            vals_out[pos] = v[j];
        }
    }
}

// --- single-pass ("onesweep") radix passes -----------------------------------
//
// One kernel counts the digits of every pass over all keys; then each pass is
// one kernel: a CTA takes the next tile (dynamic tile ids, so tile t only
// ever waits on tiles that started earlier), ranks its keys stably, publishes
// its per-digit count, and finds the count of every earlier tile with the
// same digit by looking back over their published words.  A word holds a
// 2-bit flag (aggregate / inclusive prefix) and a 30-bit count.  Every wait
// is bounded: after kLookbackLimit polls the kernel raises an error flag and
// goes on instead of spinning forever.

constexpr uint32_t kFlagAgg = 1u << 30, kFlagPrefix = 2u << 30, kCountMask = (1u << 30) - 1u;
constexpr int kLookbackLimit = 1 << 22;
constexpr int kLookWidth = 8;  // predecessor words read per look-back round trip

__global__ void __launch_bounds__(kThreads) onesweepHistKernel(const uint32_t* __restrict__ keys, uint32_t n,
                                                                int passes, int bits,
                                                                uint32_t* __restrict__ ghist) {
    __shared__ uint32_t h[4][256];
    for (int i = threadIdx.x; i < 4 * 256; i += kThreads) (&h[0][0])[i] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const size_t stride = (size_t)gridDim.x * kThreads;
    const size_t n_round = ((size_t)n + 31) / 32 * 32;  // whole warps iterate together
    for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < n_round; i += stride) {
        const bool valid = i < n;
        const uint32_t key = valid ? keys[i] : 0u;
        for (int p = 0; p < passes; ++p) {
            const int shift = 8 * p;
            const int pb = bits - shift < 8 ? bits - shift : 8;
            const uint32_t mask = (1u << (pb > 0 ? pb : 1)) - 1u;
            const uint32_t d = valid ? (key >> shift) & mask : 0xffffffffu;
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            if (valid && lane == __ffs(peers) - 1) atomicAdd(&h[p][d], (uint32_t)__popc(peers));
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += kThreads)
        if ((&h[0][0])[i]) atomicAdd(&ghist[i], (&h[0][0])[i]);
}

template <int NT>
struct OnesweepSmem {
    uint32_t cnt[NT / 32][256];
    uint32_t base[256];
    uint32_t wtot[8];
};

// One tile of a pass by a CTA of NT threads: (keys, vals) of the tile to their
// places by digit (key >> shift) & mask, in the order of the tiles and within
// the tile.  Every buffer is read past L1: blockSortDenseKernel runs its passes
// in one launch, where another SM may have written it.
template <int NT, bool kIdentVals>
__device__ __forceinline__ void onesweepTile(OnesweepSmem<NT>& m, const uint32_t* keys_in, const uint32_t* vals_in,
                                             uint32_t* keys_out, uint32_t* vals_out, uint32_t n, uint32_t tile,
                                             int shift, uint32_t mask, const uint32_t* ghist, uint32_t* status,
                                             uint32_t* err) {
    constexpr int W = NT / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    for (int i = threadIdx.x; i < W * 256; i += NT) (&m.cnt[0][0])[i] = 0;
    const size_t tbase = (size_t)tile * (NT * kSortItems) + (size_t)warp * 32 * kSortItems;
    uint32_t k[kSortItems], v[kSortItems], r[kSortItems];
    // all loads first, so that they are in flight together (the ranking
    // below synchronises the warp after every item)
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        const size_t i = tbase + (size_t)j * 32 + lane;
        const bool valid = i < n;
        k[j] = valid ? __ldcg(keys_in + i) : 0u;
        v[j] = valid ? (kIdentVals ? (uint32_t)i : __ldcg(vals_in + i)) : 0u;
    }
    // global start of every digit: exclusive scan of this pass's digit counts
    uint32_t start = 0;
    if (threadIdx.x < 256) {
        const uint32_t g = __ldcg(ghist + threadIdx.x), inc = warpInclusiveScan(g);
        if (lane == 31) m.wtot[warp] = inc;
        start = inc - g;
    }
    __syncthreads();
    if (threadIdx.x < 256)
        for (int w = 0; w < warp; ++w) start += m.wtot[w];
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        const size_t i = tbase + (size_t)j * 32 + lane;
        const bool valid = i < n;
        const uint32_t d = valid ? (k[j] >> shift) & mask : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const int leader = __ffs(peers) - 1;
        const uint32_t before = valid ? m.cnt[warp][d] : 0u;
        r[j] = before + __popc(peers & lt);
        __syncwarp();
        if (valid && lane == leader) m.cnt[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x < 256) {
        const int d = threadIdx.x;
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const uint32_t c = m.cnt[w][d];
            m.cnt[w][d] = run;
            run += c;
        }
        uint32_t* mine = status + (size_t)tile * 256 + d;
        uint32_t excl = 0;
        if (tile == 0) {
            atomicExch(mine, kFlagPrefix | run);
        } else {
            atomicExch(mine, kFlagAgg | run);
            // Walk back over the earlier tiles' words, kLookWidth per round
            // trip (independent loads), until an inclusive prefix is found.
            int t = (int)tile - 1;
            int polls = 0;
            bool done = false;
            while (!done && t >= 0) {
                uint32_t w[kLookWidth];
#pragma unroll
                for (int q = 0; q < kLookWidth; ++q)
                    w[q] = (t - q >= 0) ? *(volatile const uint32_t*)(status + (size_t)(t - q) * 256 + d) : kFlagPrefix;
                bool waiting = false;
#pragma unroll
                for (int q = 0; q < kLookWidth; ++q) {
                    if (done || waiting) continue;
                    const uint32_t f = w[q] & ~kCountMask;
                    if (f == 0) {  // not published yet: poll again from this tile
                        waiting = true;
                        continue;
                    }
                    excl += w[q] & kCountMask;
                    --t;
                    if (f == kFlagPrefix) done = true;
                }
                if (waiting) {
                    if (++polls > kLookbackLimit) {  // never expected: give up instead of hanging
                        atomicOr(err, 8u);
                        break;
                    }
                    __nanosleep(32);
                }
            }
            atomicExch(mine, kFlagPrefix | (excl + run));
        }
        m.base[d] = start + excl;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        const size_t i = tbase + (size_t)j * 32 + lane;
        if (i < n) {
            const uint32_t d = (k[j] >> shift) & mask;
            const uint32_t pos = m.base[d] + m.cnt[warp][d] + r[j];
            if (pos < n) {  // (past the end only after a wait that gave up)
                keys_out[pos] = k[j];
                vals_out[pos] = v[j];
            }
        }
    }
}

template <bool kIdentVals>
__global__ void __launch_bounds__(kThreads, 4) onesweepPassKernel(const uint32_t* __restrict__ keys_in,
                                                                const uint32_t* __restrict__ vals_in,
                                                                uint32_t* __restrict__ keys_out,
                                                                uint32_t* __restrict__ vals_out, uint32_t n,
                                                                int shift, uint32_t mask,
                                                                const uint32_t* __restrict__ ghist,
                                                                uint32_t* __restrict__ tile_counter,
                                                                uint32_t* __restrict__ status,
                                                                uint32_t* __restrict__ err) {
    __shared__ OnesweepSmem<kThreads> m;
    __shared__ uint32_t tile_s;
    if (threadIdx.x == 0) tile_s = atomicAdd(tile_counter, 1u);
    __syncthreads();
    onesweepTile<kThreads, kIdentVals>(m, keys_in, vals_in, keys_out, vals_out, n, tile_s, shift, mask, ghist, status,
                                       err);
}

__global__ void __launch_bounds__(kThreads) clearRangesKernel(ClearRanges r) {
    const size_t stride = (size_t)gridDim.x * kThreads;
    const size_t t = (size_t)blockIdx.x * kThreads + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        for (size_t i = t; i < r.n[k]; i += stride) r.p[k][i] = 0u;
}

}  // namespace

// A grid-stride clear: four CTAs of 256 threads per SM of a B200 cover the
// largest range (a few MB) in one or two passes.
constexpr size_t kClearMaxBlocks = 148 * 4;

void launchClear(const ClearRanges& r, cudaStream_t st) {
    size_t most = 0;
    for (int k = 0; k < 4; ++k) most = std::max(most, r.p[k] ? r.n[k] : 0);
    if (most == 0) return;
    ClearRanges q = r;
    for (int k = 0; k < 4; ++k)
        if (!q.p[k]) q.n[k] = 0;
    noteLaunches(1);
    const unsigned blocks = (unsigned)std::min<size_t>((most + kThreads - 1) / kThreads, kClearMaxBlocks);
    clearRangesKernel<<<blocks, kThreads, 0, st>>>(q);
}

// ---------------------------------------------------------------------------
// Host wrappers.
// ---------------------------------------------------------------------------
size_t onesweepScratchWords(size_t n, int bits) {
    const int passes = bits <= 8 ? 1 : (bits + 7) / 8;
    return (size_t)passes * 256 + 32 + (size_t)passes * radixTiles(n) * 256;
}

// Stable sort of (keys_a, identity values) by the low `bits` bits, one kernel
// per 8-bit pass.  `scratch` holds onesweepScratchWords(n, bits) words and is
// cleared here.  `err` receives bit 8 if a look-back wait gave up.
cudaError_t radixSortOnesweep(uint32_t* keys_a, uint32_t* vals_a, uint32_t* keys_b, uint32_t* vals_b, size_t n,
                              int bits, uint32_t* scratch, uint32_t* err, bool* result_in_b, cudaStream_t st) {
    *result_in_b = false;
    if (n == 0) return cudaSuccess;
    if (n > kCountMask) return cudaErrorInvalidValue;
    const int passes = bits <= 8 ? 1 : (bits + 7) / 8;
    const int ntiles = (int)radixTiles(n);
    uint32_t* ghist = scratch;
    uint32_t* counters = scratch + (size_t)passes * 256;
    uint32_t* status = counters + 32;
    {
        ClearRanges cr;
        cr.p[0] = scratch;
        cr.n[0] = onesweepScratchWords(n, bits);
        launchClear(cr, st);
    }
    // ~4 keys per thread: the histogram is bound by each thread's serial
    // chain of match/atomic rounds, not by the per-block flush (1M keys:
    // 16 keys per thread 0.072 ms for the whole sort, 4 keys 0.065 ms)
    const int hblocks = (int)std::min<size_t>((n + kThreads * 4 - 1) / (kThreads * 4), 148 * 8);
    noteLaunches(1 + passes);
    onesweepHistKernel<<<hblocks, kThreads, 0, st>>>(keys_a, (uint32_t)n, passes, bits, ghist);
    uint32_t *kin = keys_a, *vin = vals_a, *kout = keys_b, *vout = vals_b;
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        int pass_bits = bits - shift < 8 ? bits - shift : 8;
        if (pass_bits <= 0) pass_bits = 1;
        const uint32_t mask = (1u << pass_bits) - 1u;
        uint32_t* stat = status + (size_t)p * ntiles * 256;
        if (p == 0)
            onesweepPassKernel<true><<<ntiles, kThreads, 0, st>>>(kin, vin, kout, vout, (uint32_t)n, shift, mask,
                                                                  ghist + 256 * p, counters + p, stat, err);
        else
            onesweepPassKernel<false><<<ntiles, kThreads, 0, st>>>(kin, vin, kout, vout, (uint32_t)n, shift, mask,
                                                                   ghist + 256 * p, counters + p, stat, err);
        std::swap(kin, kout);
        std::swap(vin, vout);
        *result_in_b = !*result_in_b;
    }
    return cudaGetLastError();
}

size_t scanScratchElems(size_t n) { return (n + kScanChunk - 1) / kScanChunk; }

template <class T>
cudaError_t exclusiveScan(const T* in, T* out, size_t n, T* partials, T* total, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    size_t chunks = (n + kScanChunk - 1) / kScanChunk;
    if (chunks > (size_t)kScanChunk) return cudaErrorInvalidValue;
    noteLaunches(3);
    scanReduceKernel<T><<<(unsigned)chunks, kThreads, 0, st>>>(in, n, partials);
    scanPartialsKernel<T><<<1, kThreads, 0, st>>>(partials, (int)chunks, total);
    scanDownsweepKernel<T><<<(unsigned)chunks, kThreads, 0, st>>>(in, out, n, partials);
    return cudaGetLastError();
}

template cudaError_t exclusiveScan<uint32_t>(const uint32_t*, uint32_t*, size_t, uint32_t*, uint32_t*, cudaStream_t);
template cudaError_t exclusiveScan<unsigned long long>(const unsigned long long*, unsigned long long*, size_t,
                                                        unsigned long long*, unsigned long long*, cudaStream_t);

size_t radixTiles(size_t n) { return (n + kSortTile - 1) / kSortTile; }

// Same sort with every buffer supplied by the caller: `in_keys` is only read,
// the result always lands in (out_keys, out_vals), and (tmp_keys, tmp_vals)
// is the other ping-pong pair.  The pass count decides which pair the first
// pass writes so that the last pass writes the output pair.
cudaError_t radixSortPairsInto(const uint32_t* in_keys, uint32_t* out_keys, uint32_t* out_vals, uint32_t* tmp_keys,
                               uint32_t* tmp_vals, size_t n, int bits, uint32_t* hist, uint32_t* scan_partials,
                               cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const int ntiles = (int)radixTiles(n);
    const int passes = bits <= 8 ? 1 : (bits + 7) / 8;
    uint32_t* dk[2] = {out_keys, tmp_keys};
    uint32_t* dv[2] = {out_vals, tmp_vals};
    int dst = (passes % 2 == 1) ? 0 : 1;
    const uint32_t* kin = in_keys;
    const uint32_t* vin = nullptr;
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        int pass_bits = bits - shift < 8 ? bits - shift : 8;
        if (pass_bits <= 0) pass_bits = 1;
        const uint32_t mask = (1u << pass_bits) - 1u;
        noteLaunches(2);
        radixUpsweepKernel<<<ntiles, kThreads, 0, st>>>(kin, (uint32_t)n, shift, mask, hist, ntiles);
        cudaError_t e = exclusiveScan<uint32_t>(hist, hist, (size_t)256 * ntiles, scan_partials, nullptr, st);
        if (e != cudaSuccess) return e;
        if (p == 0)
            radixDownsweepKernel<true><<<ntiles, kThreads, 0, st>>>(kin, nullptr, dk[dst], dv[dst], hist, (uint32_t)n,
                                                                    shift, mask, ntiles);
        else
            radixDownsweepKernel<false><<<ntiles, kThreads, 0, st>>>(kin, vin, dk[dst], dv[dst], hist, (uint32_t)n,
                                                                     shift, mask, ntiles);
        kin = dk[dst];
        vin = dv[dst];
        dst ^= 1;
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Block sort: the stable sort of the step's cell keys, given that the live order
// is the previous step's sorted order.  Particles move a fraction of a cell per
// step, so nearly all of a block's particles were in it before, in order.  One
// kernel lists the particles that left their block (its emigrants, in the
// block's own range of `emig`; those that went further than a neighbouring
// block, or in or out of the grid, in `far`) beside the compaction, which gives
// every block its new range; then every occupied block is put together on its
// own: the particles that stayed in it, by a counting sort over its 64 cells,
// and the arrivals, picked from the neighbours' lists and sorted by (cell, live
// index).  Blocks are in key order, so an arrival from a lower block goes before
// the cell's own particles and one from a higher block after them: the result
// is exactly the stable sort of all keys, the same keys and permutation as
// radixSortOnesweep's.
// What bounds it is the latency of one block (list entry, ranges, keys: a few
// dependent reads from L2), paid once where a radix sort pays a launch and a
// look-back chain in every pass: blocks of at least kBigItem particles are taken
// by CTAs, first, the others by single warps (by CTAs where they are few), and
// blocks of at least kDenseBlock by CTAs of 1024 threads beside them.  Sort and
// compaction per step, against the radix sort: 65k-particle cube 0.033 -> 0.023
// ms, two-ball scene (1M) 0.064 -> 0.040 ms, 2M particles 0.090 -> 0.054 ms, and
// against a sort of the particles that changed cells and a merge: slab (8.4M)
// 0.19 -> 0.11 ms.  Crowded blocks (crowdedBlock) are left to the radix sort.
// ---------------------------------------------------------------------------
namespace {

// Passes of the radix sort in one launch (see radixOneLaunch).
__host__ __device__ inline int oddPasses(int bits) { return (bits <= 8 ? 1 : (bits + 7) / 8) | 1; }

constexpr int kBsThreads = 256, kBsWarps = kBsThreads / 32, kBsCtas = 5;  // CTAs per SM

// Small blocks are put together by single warps where there are more of them
// than the CTAs of blockSortKernel could take two each, else by CTAs as well.
__device__ __forceinline__ bool smallByCtas(const BlockSortArgs& s) {
    return s.counters[kSortBackWord] <= 2u * s.sort_grid;
}

// Whether the step's order is formed by radix passes over all keys instead of
// block by block.  The block sort is the slower one where many particles leave
// their blocks: every block reads the whole list of far movers, and an arrival
// costs more than a particle that stayed (its share of a bitonic sort).  The
// lines are where the two routes were measured to meet (ms per step, by blocks
// and by radix):
//   far movers: of 1M particles, 8 a cell, 2048: 0.394 and 0.421, 4000: 0.433
//     and 0.431; of 4M, 3 a cell, 2048: 1.384 and 1.581, 4000: 1.667 and 1.669
//     (reading the whole scene for every block instead: 3.2 and 91);
//   arrivals a block where single warps sort them: 1M, 8 a cell, 60 of them:
//     0.317 and 0.327, 115: 0.346 and 0.331, 210: 0.400 and 0.332; 4M, 3 a cell,
//     45: 1.251 and 1.362, 80: 1.372 and 1.413, 140: 1.519 and 1.441;
//   where CTAs do: 1M, 35 a cell, 250: 0.257 and 0.274, 500: 0.278 and 0.278, 920:
//     0.304 and 0.271; 65k, 8 a cell, 210: 0.104 and 0.122, 490: 0.124 and 0.120;
//   a block that more particles left than shared memory sorts: 250k particles in
//     8 blocks, one in seven leaving: 0.227 and 0.161; 1M: 0.818 and 0.276.
//   a block that became crowded after the route of its scene was chosen (see
//     crowdedBlock): one block of 65k 0.119 and 0.118, 100k 0.134 and 0.122, 250k
//     0.236 and 0.179; 8 of 62k 0.174 and 0.179, 250k 0.487 and 0.446; 1M particles,
//     100k of them in a block, 1.251 and 1.264, 250k 1.304 and 1.263; 4M, 250k: 1.647
//     and 1.733.
constexpr uint32_t kFarMax = 4096, kWarpArrivals = 112, kCtaArrivals = 512, kEmigMax = 8192, kCrowdedMax = 65536;
__device__ __forceinline__ bool sortByRadix(const BlockSortArgs& s) {
    if (s.n < kDenseBlock) return false;  // (blockSortDenseKernel is not launched)
    const uint32_t blocks = s.counters[kSortFrontWord] + s.counters[kSortBackWord] + s.counters[kSortDenseWord];
    return s.moved[0] > kFarMax || s.moved[2] || s.counters[kSortMaxWord] > kCrowdedMax + s.n / 13 ||
           s.moved[1] > (unsigned long long)blocks * (smallByCtas(s) ? kCtaArrivals : kWarpArrivals);
}

__device__ __forceinline__ int blockScene(const uint32_t* base, int nscenes, uint32_t b) {
    int lo = 0, hi = nscenes - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (base[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(kBsThreads) emigrantKernel(BlockSortArgs s) {
    const uint32_t n = s.n;
    __shared__ uint32_t moved_s;
    if (threadIdx.x == 0) moved_s = 0u;
    if (blockIdx.x == 0)  // the radix passes' digit counts
        for (int i = threadIdx.x; i < oddPasses(s.key_bits) * 256; i += kBsThreads) s.radix_scratch[i] = 0u;
    uint32_t moved = 0;
    const uint32_t stride = gridDim.x * kBsThreads * 4;
    const uint32_t n_round = (n + 127) / 128 * 128;  // whole warps iterate together
    for (uint32_t i0 = (blockIdx.x * kBsThreads + threadIdx.x) * 4; i0 < n_round; i0 += stride) {
        uint32_t key[4], old[4];
        if (i0 + 4 <= n) {  // (the buffers are 256-byte aligned)
            *reinterpret_cast<uint4*>(key) = *reinterpret_cast<const uint4*>(s.keys + i0);
            *reinterpret_cast<uint4*>(old) = *reinterpret_cast<const uint4*>(s.prev_keys + i0);
        } else {
            for (int j = 0; j < 4; ++j) {
                key[j] = i0 + j < n ? s.keys[i0 + j] : 0u;
                old[j] = i0 + j < n ? s.prev_keys[i0 + j] : 0u;
            }
        }
        // a warp's particles are neighbours in the sorted order: most of its movers
        // leave the same block, and share one atomic (all four are on their way
        // before the first is waited for)
        const int lane = threadIdx.x & 31;
        uint32_t at[4];
        unsigned peers[4] = {};  // of a mover: the lanes whose movers go to the same list
        bool near[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t home = old[j] >> 6, blk = key[j] >> 6;
            const unsigned movers = __ballot_sync(0xffffffffu, blk != home);
            moved += (uint32_t)__popc(movers);
            if (blk == home) continue;
            const SceneDev& sc = s.scenes[blockScene(s.scene_block_base, s.nscenes, home)];
            const uint32_t out = sc.nblocks, lh = home - sc.block_base, lb = blk - sc.block_base;
            near[j] = lh < out && lb < out;
            if (near[j]) {
                const int X = sc.nb[0], Y = sc.nb[1];
                const int dx = (int)(lh % X) - (int)(lb % X), dy = (int)(lh / X % Y) - (int)(lb / X % Y),
                          dz = (int)(lh / (X * Y)) - (int)(lb / (X * Y));
                near[j] = abs(dx) <= 1 && abs(dy) <= 1 && abs(dz) <= 1;
            }
            peers[j] = __match_any_sync(movers, near[j] ? home : 0xffffffffu);
            if (lane == __ffs(peers[j]) - 1)
                at[j] = atomicAdd(near[j] ? &s.emig_count[home] : &s.moved[0], (uint32_t)__popc(peers[j]));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!peers[j]) continue;
            const uint32_t home = old[j] >> 6, c = (uint32_t)__popc(peers[j]);
            const int leader = __ffs(peers[j]) - 1;
            const uint32_t first = __shfl_sync(peers[j], at[j], leader);
            if (near[j] && lane == leader && first <= kEmigMax && first + c > kEmigMax) atomicAdd(&s.moved[2], 1u);
            const uint32_t slot = first + (uint32_t)__popc(peers[j] & ((1u << lane) - 1u));
            const uint2 e = make_uint2(i0 + j, key[j]);
            if (near[j]) s.emig[s.prev_range[home].x + slot] = e;
            else s.far[slot] = e;
        }
    }
    if (!__syncthreads_or((int)moved)) return;
    if ((threadIdx.x & 31) == 0 && moved) atomicAdd(&moved_s, moved);
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(&s.moved[1], moved_s);
}

// A group of NW warps (a whole CTA, or one warp) that puts blocks together.
template <int NW>
struct BlockSorter {
    static constexpr int N = NW * 32;
    static constexpr uint32_t kCap = NW == 1 ? 192 : NW == 32 ? 8192 : 4096;  // arrivals sorted in shared memory; more in aux
    struct Smem {
        unsigned long long arr[kCap];
        uint32_t cnt[NW][64];  // own particles per warp and cell, then their first positions
        uint32_t arrLo[64], arrHi[64], own[64], ownBelow[64], cellStart[64];
        uint32_t nbStart[27], nbOff[28], narr, stayed, wsum[NW];
    };
    Smem& m;
    const BlockSortArgs& s;
    int t, lane, warp;  // thread and warp within the group
    __device__ __forceinline__ BlockSorter(Smem& m_, const BlockSortArgs& s_, int t_)
        : m(m_), s(s_), t(t_), lane(t_ & 31), warp(t_ >> 5) {}
    __device__ __forceinline__ void sync() const {
        if (NW == 1) __syncwarp();
        else __syncthreads();
    }

    // Ascending sort of a[0..n): bitonic network in the form whose comparators
    // all point the same way, so that elements past n act as infinity.
    __device__ __forceinline__ void sort(unsigned long long* a, uint32_t n) const {
        for (uint32_t k = 2; k / 2 < n; k <<= 1) {
            for (uint32_t j = k; j > 1; j >>= 1) {
                const uint32_t half = j >> 1;
                for (uint32_t p = t;; p += N) {
                    const uint32_t o = p & (half - 1), b = (p / half) * j;
                    const uint32_t l = b + o, r = j == k ? b + k - 1 - o : l + half;
                    if (l >= n) break;
                    if (r < n) {
                        const unsigned long long x = a[l], y = a[r];
                        if (x > y) {
                            a[l] = y;
                            a[r] = x;
                        }
                    }
                }
                sync();
            }
        }
    }

    // The keys of the warp's part [w0, w1) that stayed, as cells (64: not this
    // block's); f(live index, cell, key) for each 32.  One warp's chain of reads
    // bounds a crowded block (130k particles by one CTA: 107 us), so the keys of
    // the next U rows are read ahead: 94 us.
    template <class Fn>
    __device__ __forceinline__ void forOwn(uint2 prev, uint32_t w0, uint32_t w1, uint32_t blk, Fn&& f) const {
        constexpr int U = NW == 32 ? 8 : 4;
        uint32_t key[U], next[U];
        auto load = [&](uint32_t (&k)[U], uint32_t i) {
#pragma unroll
            for (int j = 0; j < U; ++j) k[j] = i + 32 * j + lane < w1 ? s.keys[prev.x + i + 32 * j + lane] : 0xffffffffu;
        };
        load(next, w0);
        for (uint32_t i = w0; i < w1; i += 32 * U) {
#pragma unroll
            for (int j = 0; j < U; ++j) key[j] = next[j];
            if (i + 32 * U < w1) load(next, i + 32 * U);
#pragma unroll
            for (int j = 0; j < U; ++j) {
                if (i + 32 * j >= w1) break;
                const bool mine = i + 32 * j + lane < w1 && (key[j] >> 6) == blk;
                f(prev.x + i + 32 * j + lane, mine ? key[j] & 63u : 64u, key[j]);
            }
        }
    }

    __device__ __forceinline__ void run(const BlockItem& it, uint2 prev, uint32_t nfar) const {
        const SceneDev& sc = s.scenes[it.scene];
        const uint32_t blk = it.block, lt = (1u << lane) - 1u;
        const bool outside = blk == sc.block_base + sc.nblocks;
        for (int q = t; q < NW * 64; q += N) (&m.cnt[0][0])[q] = 0u;
        for (int q = t; q < 64; q += N) m.arrLo[q] = m.arrHi[q] = 0u;
        if (t == 0) m.narr = 0u;
        if (warp == NW - 1) {
            // the neighbouring blocks' emigrant lists
            uint32_t c = 0, start = 0;
            if (lane < 27 && lane != 13 && !outside) {
                const uint32_t lb = blk - sc.block_base;
                const int x = (int)(lb % (uint32_t)sc.nb[0]) + lane % 3 - 1;
                const int y = (int)((lb / (uint32_t)sc.nb[0]) % (uint32_t)sc.nb[1]) + (lane / 3) % 3 - 1;
                const int z = (int)(lb / ((uint32_t)sc.nb[0] * (uint32_t)sc.nb[1])) + lane / 9 - 1;
                if (x >= 0 && y >= 0 && z >= 0 && x < sc.nb[0] && y < sc.nb[1] && z < sc.nb[2]) {
                    const uint32_t nb = sc.block_base + (uint32_t)((z * sc.nb[1] + y) * sc.nb[0] + x);
                    c = s.emig_count[nb];
                    start = s.prev_range[nb].x;
                }
            }
            uint32_t inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane < 27) {
                m.nbStart[lane] = start;
                m.nbOff[lane + 1] = inc;
            }
            if (lane == 0) m.nbOff[0] = 0u;
        }
        sync();
        // ---- own particles: each warp a part of the block's previous range ----
        const uint32_t per = ((prev.y + N - 1) / N) * 32;
        const uint32_t w0 = min(prev.y, warp * per), w1 = min(prev.y, w0 + per);
        forOwn(prev, w0, w1, blk, [&](uint32_t, uint32_t c, uint32_t) {
            const uint32_t peers = __match_any_sync(0xffffffffu, c);
            if (c < 64u && lane == __ffs(peers) - 1) m.cnt[warp][c] += (uint32_t)__popc(peers);
            __syncwarp();
        });
        sync();
        if (warp == 0) {  // cells 2 lane and 2 lane + 1
            uint32_t tot[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t run = 0;
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    const uint32_t c = m.cnt[w][2 * lane + h];
                    m.cnt[w][2 * lane + h] = run;
                    run += c;
                }
                m.own[2 * lane + h] = tot[h] = run;
            }
            uint32_t inc = tot[0] + tot[1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            m.ownBelow[2 * lane] = inc - tot[0] - tot[1];
            m.ownBelow[2 * lane + 1] = inc - tot[1];
            if (lane == 31) m.stayed = inc;
        }
        sync();
        const uint32_t stayed = m.stayed;
        const uint32_t A = it.count >= stayed ? it.count - stayed : 0u;
        uint32_t na = 0;
        unsigned long long* arr = A <= kCap ? m.arr : s.aux + it.start;
        if (A || it.count < stayed) {
            // ---- arrivals ----
            auto add = [&](uint32_t slot, uint2 e) {
                if (slot < A) arr[slot] = ((unsigned long long)(e.y & 63u) << 32) | e.x;
            };
            const uint32_t E = m.nbOff[27], F = E + nfar;
            for (uint32_t e = t; e < F; e += N) {
                uint2 v;
                if (e < E) {
                    int q = 0;
#pragma unroll
                    for (int h = 16; h > 0; h >>= 1)
                        if (q + h < 27 && m.nbOff[q + h] <= e) q += h;
                    v = s.emig[m.nbStart[q] + (e - m.nbOff[q])];
                } else {
                    v = s.far[e - E];
                }
                if ((v.y >> 6) == blk) add(atomicAdd(&m.narr, 1u), v);
            }
            sync();
            if (t == 0 && (m.narr != A || it.count < stayed)) atomicOr(s.err, ERR_INDEX);  // never expected
            na = min(m.narr, A);
            sort(arr, na);
            for (uint32_t q = t; q < na; q += N) {
                const uint32_t c = (uint32_t)(arr[q] >> 32), g = (uint32_t)arr[q];
                atomicAdd(g < prev.x ? &m.arrLo[c] : &m.arrHi[c], 1u);
            }
            sync();
        }
        if (warp == 0) {
            const uint32_t a0 = m.arrLo[2 * lane] + m.arrHi[2 * lane];
            const uint32_t a1 = m.arrLo[2 * lane + 1] + m.arrHi[2 * lane + 1];
            uint32_t inc = a0 + a1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            m.cellStart[2 * lane] = m.ownBelow[2 * lane] + inc - a0 - a1;
            m.cellStart[2 * lane + 1] = m.ownBelow[2 * lane + 1] + inc - a1;
        }
        sync();
        // ---- positions ----
        auto put = [&](uint32_t pos, uint32_t key, uint32_t g) {
            if (pos >= it.count) return;  // never expected
            s.out_keys[it.start + pos] = key;
            s.out_perm[it.start + pos] = g;
        };
        // the q-th arrival of all is the r-th of its cell
        for (uint32_t q = t; q < na; q += N) {
            const uint32_t c = (uint32_t)(arr[q] >> 32), g = (uint32_t)arr[q];
            const uint32_t r = q - (m.cellStart[c] - m.ownBelow[c]);
            put(m.cellStart[c] + r + (r < m.arrLo[c] ? 0u : m.own[c]), (blk << 6) | c, g);
        }
        forOwn(prev, w0, w1, blk, [&](uint32_t g, uint32_t c, uint32_t key) {
            const uint32_t peers = __match_any_sync(0xffffffffu, c);
            uint32_t before = 0;
            if (c < 64u) before = m.cnt[warp][c];
            __syncwarp();
            if (c < 64u) {
                put(m.cellStart[c] + m.arrLo[c] + before + __popc(peers & lt), key, g);
                if (lane == __ffs(peers) - 1) m.cnt[warp][c] = before + (uint32_t)__popc(peers);
            }
            __syncwarp();
        });
        sync();
    }
};

constexpr int kRadixThreads = 1024, kRadixTile = kRadixThreads * kSortItems;
__device__ __forceinline__ uint32_t radixMask(int bits, int width, int p) {
    return (1u << min(width, bits - p * width)) - 1u;
}

// The stable sort of all keys by radix passes in one launch.  Its phases -- count
// the digits of all passes, then the passes -- are cut into ntiles tickets
// each, handed out in order; a phase's tickets wait until those of the phase
// before are done.  A ticket is only ever waited for by later ones, and every
// earlier one is done or in the hands of a running CTA, so no number of CTAs
// need be resident; every wait is bounded all the same.  The pass count is odd,
// so that the last one writes the sorted buffers.
struct RadixSmem {
    OnesweepSmem<kRadixThreads> tile;
    uint32_t ticket;
};
__device__ __forceinline__ void radixOneLaunch(const BlockSortArgs& s, RadixSmem& m) {
    const int passes = oddPasses(s.key_bits), width = (s.key_bits + passes - 1) / passes;
    const uint32_t ntiles = (s.n + kRadixTile - 1) / kRadixTile;
    uint32_t *ghist = s.radix_scratch, *status = ghist + passes * 256;
    uint32_t* ctr = s.counters + kSortRadixWord;  // tickets handed out, tickets done per phase
    const uint32_t total = (1 + passes) * ntiles;
    for (;;) {
        __syncthreads();  // the previous ticket's shared memory is no longer read
        if (threadIdx.x == 0) {
            uint32_t ticket = atomicAdd(&ctr[0], 1u);
            if (ticket >= ntiles && ticket < total) {
                const volatile uint32_t* done = ctr + ticket / ntiles;  // of the phase before
                int polls = 0;
                while (*done < ntiles) {
                    if (++polls > kLookbackLimit) {  // never expected: give up instead of hanging
                        atomicOr(s.err, 8u);
                        ticket = total;
                        break;
                    }
                    __nanosleep(32);
                }
                __threadfence();
            }
            m.ticket = ticket;
        }
        __syncthreads();
        const uint32_t ticket = m.ticket;
        if (ticket >= total) return;
        const int phase = (int)(ticket / ntiles);
        const uint32_t tile = ticket % ntiles;
        if (phase == 0) {
            // (emigrantKernel has cleared the digit counts; a tile clears its status words)
            for (int i = threadIdx.x; i < passes * 256; i += kRadixThreads)
                status[((size_t)(i >> 8) * ntiles + tile) * 256 + (i & 255)] = 0u;
            uint32_t* h = &m.tile.cnt[0][0];  // [pass][256]
            for (int i = threadIdx.x; i < passes * 256; i += kRadixThreads) h[i] = 0u;
            uint32_t key[kSortItems];
#pragma unroll
            for (int j = 0; j < kSortItems; ++j) {
                const uint32_t i = tile * kRadixTile + j * kRadixThreads + threadIdx.x;
                key[j] = i < s.n ? __ldcg(s.keys + i) : 0u;
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kSortItems; ++j) {
                const bool valid = tile * kRadixTile + j * kRadixThreads + threadIdx.x < s.n;
                for (int p = 0; p < passes; ++p) {
                    const uint32_t d = valid ? (key[j] >> (p * width)) & radixMask(s.key_bits, width, p) : 0xffffffffu;
                    const uint32_t peers = __match_any_sync(0xffffffffu, d);
                    if (valid && (threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&h[p * 256 + d], (uint32_t)__popc(peers));
                }
            }
            __syncthreads();
            for (int i = threadIdx.x; i < passes * 256; i += kRadixThreads)
                if (h[i]) atomicAdd(&ghist[i], h[i]);
        } else {
            const int p = phase - 1;
            const uint32_t mask = radixMask(s.key_bits, width, p);
            uint32_t* st = status + (size_t)p * ntiles * 256;
            const uint32_t* gh = ghist + p * 256;
            if (p == 0) {
                onesweepTile<kRadixThreads, true>(m.tile, s.keys, nullptr, s.out_keys, s.out_perm, s.n, tile, 0, mask, gh,
                                                  st, s.err);
            } else {
                const bool back = p & 1;  // from the output to the spare buffers
                onesweepTile<kRadixThreads, false>(m.tile, back ? s.out_keys : s.keys, back ? s.out_perm : s.spare_vals,
                                                   back ? s.keys : s.out_keys, back ? s.spare_vals : s.out_perm, s.n,
                                                   tile, p * width, mask, gh, st, s.err);
            }
        }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(&ctr[1 + phase], 1u);
    }
}

constexpr size_t kBsSmem = std::max(sizeof(BlockSorter<kBsWarps>::Smem), kBsWarps * sizeof(BlockSorter<1>::Smem));
constexpr size_t kBsDenseSmem = std::max(sizeof(BlockSorter<32>::Smem), sizeof(RadixSmem));

__global__ void __launch_bounds__(kBsThreads, kBsCtas) blockSortKernel(BlockSortArgs s) {
    extern __shared__ unsigned long long bs_smem[];
    __shared__ uint32_t item_s;
    const uint32_t nfront = s.counters[kSortFrontWord], nback = s.counters[kSortBackWord];
    const uint32_t nfar = s.moved[0];
    // few small blocks: by CTAs as well, whose latency is a third of a warp's
    const bool all = smallByCtas(s);
    const uint32_t ncta = nfront + (all ? nback : 0u);
    const bool fixed = ncta <= gridDim.x;  // at most one each: no scheduler
    BlockItem it{};
    uint2 prev{};
    auto take = [&](uint32_t wi) {
        it = s.list[wi < nfront ? wi : s.list_cap - 1 - (wi - nfront)];
        prev = s.prev_range[it.block];
    };
    // the reads of the first block are in flight while the route is decided
    if (fixed && blockIdx.x < ncta) take(blockIdx.x);
    if (sortByRadix(s)) return;  // blockSortDenseKernel sorts
    {
        auto& m = *reinterpret_cast<BlockSorter<kBsWarps>::Smem*>(bs_smem);
        const BlockSorter<kBsWarps> g(m, s, threadIdx.x);
        for (uint32_t wi = blockIdx.x;;) {
            if (!fixed) wi = nextWorkItem(s.counters + kSortSchedWord, ncta, &item_s);
            if (wi >= ncta) break;
            if (!fixed) take(wi);
            g.run(it, prev, nfar);
            if (fixed) break;
        }
    }
    if (all) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    auto& m = reinterpret_cast<BlockSorter<1>::Smem*>(bs_smem)[warp];
    const BlockSorter<1> g(m, s, lane);
    uint32_t* sched = s.counters + kSortSchedWord + 2;
    for (;;) {
        uint32_t wi = 0;
        if (lane == 0) {
            wi = atomicAdd(&sched[0], 1u);
            if (wi >= nback && atomicAdd(&sched[1], 1u) == gridDim.x * kBsWarps - 1) {
                sched[0] = 0u;
                sched[1] = 0u;
            }
        }
        wi = __shfl_sync(0xffffffffu, wi, 0);
        if (wi >= nback) return;
        const BlockItem it = s.list[s.list_cap - 1 - wi];
        g.run(it, s.prev_range[it.block], nfar);
    }
}

// Blocks of at least kDenseBlock particles, by CTAs of 1024 threads; or the
// whole sort by radix passes.
__global__ void __launch_bounds__(1024, 1) blockSortDenseKernel(BlockSortArgs s) {
    extern __shared__ unsigned long long bs_smem[];
    __shared__ uint32_t item_s;
    if (sortByRadix(s)) return radixOneLaunch(s, *reinterpret_cast<RadixSmem*>(bs_smem));
    const uint32_t ndense = s.counters[kSortDenseWord];
    if (ndense == 0) return;
    const uint32_t nfar = s.moved[0];
    auto& m = *reinterpret_cast<BlockSorter<32>::Smem*>(bs_smem);
    const BlockSorter<32> g(m, s, threadIdx.x);
    for (;;) {
        const uint32_t wi = nextWorkItem(s.counters + kSortSchedWord + 4, ndense, &item_s);
        if (wi >= ndense) return;
        const BlockItem it = s.dense[wi];
        g.run(it, s.prev_range[it.block], nfar);
    }
}

}  // namespace

unsigned blockSortGrid(unsigned max_blocks, int num_sms) {
    return std::max(1u, std::min(max_blocks, (unsigned)(num_sms * kBsCtas)));
}

size_t blockSortScratchWords(size_t n, int bits) {
    return (size_t)oddPasses(bits) * 256 * ((n + kRadixTile - 1) / kRadixTile + 1);
}

cudaError_t launchEmigrants(const BlockSortArgs& a, int num_sms, cudaStream_t st) {
    noteLaunches(1);
    const unsigned grid = (unsigned)std::min<size_t>(((size_t)a.n + kBsThreads * 4 - 1) / (kBsThreads * 4), (size_t)num_sms * 8);
    emigrantKernel<<<std::max(1u, grid), kBsThreads, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launchBlockSort(const BlockSortArgs& a, cudaStream_t st) {
    static_assert(kBsSmem <= 47 * 1024, "dynamic shared memory without an attribute");
    noteLaunches(1);
    blockSortKernel<<<a.sort_grid, kBsThreads, kBsSmem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launchBlockSortDense(const BlockSortArgs& a, unsigned max_blocks, int num_sms, cudaStream_t st) {
    noteLaunches(1);
    const cudaError_t e =
        cudaFuncSetAttribute(blockSortDenseKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBsDenseSmem);
    if (e != cudaSuccess) return e;
    blockSortDenseKernel<<<std::max(1u, std::min(max_blocks, (unsigned)num_sms)), 1024, kBsDenseSmem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace mpm
