// kernels.cu -- the MPM step kernels for sm_100a.
//
//   keyKernel       cell keys of the live particle order (first step / after uploads)
//   compactOnesweepKernel   work items from per-block particle counts (P2G's,
//                   with their per-combination lists, and G2P's)
//   stressKernel    V0 * stress (tau) from Fe, Fp (first step / after uploads)
//   p2gKernel       deterministic block scatter by whole CTAs
//                   (src/mpm_solver3d.cu:237-294, src/apic_mpm_solver3d.cu:245-304)
//   p2gWarpKernel   the same scatter by single warps for small work items
//                   (bitwise p2gKernel's tiles)
//   gridKernel      tile merge + gravity + velocity update + collision in one
//                   pass (src/mpm_solver3d.cu:394-426, src/grid3d.cu:36-41)
//   g2pKernel       gather + transfer blend + Fe/Fp plasticity + SVD + next
//                   step's stress + particle collision + advection + next key
//                   (src/mpm_solver3d.cu:316-391,428-445; apic :326-388)
//   split-mode kernels for the reference's sub-step API.
#include <cuda.h>  // CUtensorMap and its enums (the encoder is fetched at run time)
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "engine_host.hpp"
#include "mpm_math.cuh"
#include "particle_common.cuh"
#include "per_device.hpp"

#include <atomic>
#include <cstdlib>
#include <type_traits>

namespace mpm {

static std::atomic<uint64_t> g_launches{0};
void noteLaunches(uint64_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
uint64_t kernelLaunches() { return g_launches.load(std::memory_order_relaxed); }

namespace {


__device__ __forceinline__ float ldg(const float* p) { return __ldg(p); }

// Asynchronous 4-byte global -> shared copies (cp.async, L1-allocating).
__device__ __forceinline__ void cpAsync4(float* smem_dst, const float* gsrc) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cpAsyncWaitAll() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// G2P's prefetch row of a thread (floats): Fe, Fp, V0, x, mass, pid, and v
// (PIC-FLIP); odd, so that rows of consecutive threads fall in different banks.
constexpr int kPreVol = 18, kPreX = 19, kPreMass = 22, kPrePid = 23, kPreV = 24, kPreStride = 27;


__device__ __forceinline__ uint32_t outsideKey(const SceneDev& sc) { return (sc.block_base + sc.nblocks) << 6; }

__device__ __forceinline__ uint32_t particleKey(const SceneDev& sc, const float* x, uint32_t* err) {
    int base[3];
    bool fin = isfinite(x[0]) && isfinite(x[1]) && isfinite(x[2]);
    if (!fin) atomicOr(err, ERR_NONFINITE);
    if (fin && stencilBase(sc, x, base)) return makeKey(sc, base);
    return outsideKey(sc);
}


// tau = V0 * (dPsi/dFe) Fe^T, symmetric (xx yy zz xy xz yz), from the SVD of Fe.
//  fixed corotated (src/material_point3d.cu:110-128):
//     2 mu (Fe - R) Fe^T + la (J-1) J I  =  2 mu U diag(s(s-1)) U^T + la (J-1) J I
//  Neo-Hookean (:131-155), with s clamped to >= FLT_EPSILON (Fe projected):
//     mu (Fe Fe^T - I) + la ln(J) I      =  mu U diag(s^2) U^T - mu I + la ln J I
__device__ __forceinline__ void tauFromSvd(int model, const float* U, const float* s, float mu, float la, float V0,
                                           float* tau) {
    float d[3], diag;
    float J = s[0] * s[1] * s[2];
    if (model == MPM_MODEL_NEO_HOOKEAN) {
#pragma unroll
        for (int k = 0; k < 3; ++k) d[k] = mu * s[k] * s[k];
        diag = la * logf(J) - mu;
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) d[k] = 2.0f * mu * s[k] * (s[k] - 1.0f);
        diag = la * (J - 1.0f) * J;
    }
    const int I[6] = {0, 1, 2, 0, 0, 1}, Jx[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
    for (int e = 0; e < 6; ++e) {
        int i = I[e], j = Jx[e];
        float v = U[3 * i] * d[0] * U[3 * j] + U[3 * i + 1] * d[1] * U[3 * j + 1] + U[3 * i + 2] * d[2] * U[3 * j + 2];
        if (e < 3) v += diag;
        tau[e] = V0 * v;
    }
}

// Stress of a particle from its current Fe (Neo-Hookean projects Fe in place).
__device__ __forceinline__ void stressFromFe(const MaterialDev& m, float* Fe, const float* Fp, float V0, float* tau) {
    float U[9], V[9], s[3];
    svd3(Fe, U, s, V);
    float mu, la;
    plasticLame(m, Fp, mu, la);
    if (m.model == MPM_MODEL_NEO_HOOKEAN) {
        bool proj = false;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            proj |= s[k] < kFltEps;
            s[k] = fmaxf(s[k], kFltEps);
        }
        if (proj) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    Fe[3 * i + j] = U[3 * i] * s[0] * V[3 * j] + U[3 * i + 1] * s[1] * V[3 * j + 1] +
                                    U[3 * i + 2] * s[2] * V[3 * j + 2];
        }
    }
    tauFromSvd(m.model, U, s, mu, la, V0, tau);
}

__device__ __forceinline__ int sceneOfBlock(const uint32_t* scene_block_base, int nscenes, uint32_t b) {
    int lo = 0, hi = nscenes - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (scene_block_base[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

}  // namespace

// ---------------------------------------------------------------------------
// Keys of the live particle order (used when keys were not produced by G2P).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) keyKernel(const SceneDev* __restrict__ scenes, int parity,
                                                       uint32_t* __restrict__ keys, uint32_t* __restrict__ block_count,
                                                       uint32_t* __restrict__ err) {
    const SceneDev& sc = scenes[blockIdx.y];
    const float* f = sc.buf[parity].f;
    const size_t cap = sc.cap;
    // whole warps iterate together, so that a warp's particles of one block
    // add to its count with one atomic (cell-sorted particles share blocks)
    const uint32_t n_round = (sc.n + 31u) & ~31u;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n_round; i += gridDim.x * kThreads) {
        const bool valid = i < sc.n;
        uint32_t blk = 0xffffffffu;
        if (valid) {
            float x[3] = {f[(F_X + 0) * cap + i], f[(F_X + 1) * cap + i], f[(F_X + 2) * cap + i]};
            const uint32_t key = particleKey(sc, x, err);
            keys[sc.key_offset + i] = key;
            blk = key >> 6;
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, blk);
        if (valid && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&block_count[blk], (uint32_t)__popc(peers));
    }
}

// Block compaction in one kernel: each CTA scans a tile of 512 block counts,
// publishes the tile's (work items, particles) sums and looks back over the
// earlier tiles' published words (single-pass scan, dynamic tile ids, every
// wait bounded), then writes the work items, slots and outside items of its
// blocks and clears their counts.  Word layout: [63:62] flag, [61:32] items,
// [31:0] particles.
// one block a thread, so that neighbouring threads write neighbouring words of
// the dense tables (two-ball step 0.268 ms; four a thread 0.271 ms, four a
// thread of 1024 0.277 ms)
constexpr int kCompactPer = 1, kCompactThreads = 512;
constexpr int kCompactTile = kCompactThreads * kCompactPer;
constexpr unsigned long long kCFlagAgg = 1ull << 62, kCFlagPrefix = 2ull << 62, kCFlagMask = 3ull << 62;

template <int W>  // warps of the CTA
__device__ __forceinline__ unsigned long long blockExclusiveScanU64(unsigned long long x, unsigned long long* total) {
    __shared__ unsigned long long wt[W];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) wt[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        unsigned long long t = lane < W ? wt[lane] : 0ull, ti = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= o) ti += y;
        }
        if (lane < W) wt[lane] = ti - t;
        const unsigned long long tl = __shfl_sync(0xffffffffu, ti, W - 1);
        if (lane == 0) *total = tl;
    }
    __syncthreads();
    const unsigned long long r = inc - x + wt[warp];
    __syncthreads();
    return r;
}

// The particles [start, start + count) of block b as `items` work items of
// nearly equal size: count / items each, the first count % items one more.
__device__ __forceinline__ void splitItems(BlockItem* out, uint32_t b, uint32_t start, uint32_t count,
                                           uint32_t items, uint32_t scene) {
    const uint32_t base = count / items, rem = count % items;
    uint32_t off = 0;
    for (uint32_t q = 0; q < items; ++q) {
        const uint32_t len = base + (q < rem ? 1u : 0u);
        out[q] = BlockItem{b, start + off, len, scene};
        off += len;
    }
}

struct CompactArgs {
    uint32_t* block_count;
    uint32_t total_blocks;
    const uint32_t* scene_block_base;
    int nscenes;
    BlockItem *active, *outside;
    uint32_t* counters;
    int2* block_slot;
    BlockItem* g2p_items;
    uint32_t g2p_cap;
    ComboSplit split;
    uint32_t* p2g_lists;
    uint32_t p2g_list_cap;
    uint2* block_range;
    uint32_t *emig_count, *moved;
    BlockItem* sort_list;
    uint32_t sort_list_cap;
    BlockItem* dense_list;
    const SceneDev* scenes;
    uint32_t* err;
};

// Block b's (work items << 32 | particles) and its scene.
__device__ __forceinline__ unsigned long long blockLoad(const CompactArgs& a, uint32_t b, int* scene) {
    *scene = 0;
    if (b >= a.total_blocks) return 0ull;
    const uint32_t c = a.block_count[b];
    if (c == 0) return 0ull;
    const int s = *scene = sceneOfBlock(a.scene_block_base, a.nscenes, b);
    const bool out = b == a.scene_block_base[s + 1] - 1;
    return ((out ? 0ull : (unsigned long long)blockItems(c, a.scenes[s].n)) << 32) | (unsigned long long)c;
}

// The work items, slots, ranges and list entries of the thread's PER blocks
// from b0 on, `run` the (items, particles) of all blocks before them.
template <int PER>
__device__ __forceinline__ void placeBlocks(const CompactArgs& a, uint32_t b0, const unsigned long long (&packed)[PER],
                                            const int (&scn)[PER], unsigned long long run) {
    // Most blocks of a scene are empty: a warp of empty ones has no items, no
    // list entries and no scene to look up (874k blocks of 64 scenes, 9.8k of
    // them occupied: 54 -> 47 us).
    unsigned long long any = 0ull;
#pragma unroll
    for (int j = 0; j < PER; ++j) any |= packed[j];
    if (!__any_sync(0xffffffffu, any != 0ull)) {
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const uint32_t b = b0 + j;
            if (b >= a.total_blocks) break;
            a.block_range[b] = make_uint2((uint32_t)(run & 0xffffffffull), 0u);
            a.emig_count[b] = 0u;
            a.block_slot[b] = make_int2(-1, 0);
        }
        return;
    }
    // Slots are aggregated per warp when every block of the warp that has
    // items belongs to one combination (the common case), else taken per block.
    uint32_t gtot = 0;
    int gcombo = -1;
    bool mixed = false;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const uint32_t b = b0 + j;
        if (b >= a.total_blocks) continue;
        if ((packed[j] >> 32) == 0) continue;
        const uint32_t count = (uint32_t)(packed[j] & 0xffffffffull);
        const int k = a.scenes[scn[j]].combo;
        gtot += (count + a.split.g2p_chunk[k] - 1) / a.split.g2p_chunk[k];
        if (gcombo < 0) gcombo = k;
        else mixed |= k != gcombo;
    }
    const int lane = threadIdx.x & 31;
    const unsigned has = __ballot_sync(0xffffffffu, gtot > 0);
    const int lead = __shfl_sync(0xffffffffu, gcombo, has ? __ffs(has) - 1 : 0);
    const bool warp_fast = __all_sync(0xffffffffu, gtot == 0 || (!mixed && gcombo == lead));
    // Slots of this thread's P2G items in their combination's lists: list 0
    // for items of at most the combination's warp threshold (P2G by warps),
    // list 1 for the others -- those of at least kBigItem particles from its
    // front, the rest from its back (class 2); the items of at most
    // kWarpAutoMax particles are counted as well (class 3).  Then of its
    // blocks in the block sort's lists (classes 5 to 7).  Totals per warp, and
    // the classes' atomics issued together, each by a lane of its own (one
    // after another, each waited for, they took a third of the kernel).
    constexpr int kClasses = 8;  // P2G 0..3, G2P 4, block sort 5, 6, 7
    uint32_t ctot[kClasses] = {};
    if (warp_fast) ctot[4] = gtot;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        if (b0 + j >= a.total_blocks) continue;
        const uint32_t items = (uint32_t)(packed[j] >> 32), count = (uint32_t)(packed[j] & 0xffffffffull);
        ctot[5] += count >= kBigItem && count < kDenseBlock ? 1u : 0u;
        ctot[6] += count && count < kBigItem ? 1u : 0u;
        ctot[7] += count >= kDenseBlock ? 1u : 0u;
        if (!a.p2g_lists || !warp_fast || !items) continue;
        const uint32_t size = (count + items - 1) / items;
        const int cls = size <= a.split.p2g_warp_max[lead] ? 0 : (size >= kBigItem ? 1 : 2);
        ctot[0] += cls == 0 ? items : 0u;
        ctot[1] += cls == 1 ? items : 0u;
        ctot[2] += cls == 2 ? items : 0u;
        if (size <= kWarpAutoMax) ctot[3] += items;
    }
    uint32_t cnext[kClasses], want = 0;
#pragma unroll
    for (int cls = 0; cls < kClasses; ++cls) {
        uint32_t inc = ctot[cls];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        cnext[cls] = inc - ctot[cls];
        const uint32_t all = __shfl_sync(0xffffffffu, inc, 31);
        if (lane == cls) want = all;
    }
    {
        const int word = lane < 2    ? kP2GListWord + 2 * lead + lane
                         : lane == 2 ? kP2GBackWord + lead
                         : lane == 3 ? kP2GSmallWord + lead
                         : lane == 4 ? kG2PCountWord + lead
                         : lane == 5 ? kSortFrontWord
                         : lane == 6 ? kSortBackWord
                                     : kSortDenseWord;
        const uint32_t base = lane < kClasses && want ? atomicAdd(&a.counters[word], want) : 0u;
#pragma unroll
        for (int cls = 0; cls < kClasses; ++cls) cnext[cls] += __shfl_sync(0xffffffffu, base, cls);
    }
    uint32_t gnext = cnext[4];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const uint32_t b = b0 + j;
        if (b >= a.total_blocks) break;
        const unsigned long long v = packed[j];
        const uint32_t count = (uint32_t)(v & 0xffffffffull);
        const uint32_t items = (uint32_t)(v >> 32);
        const uint32_t start = (uint32_t)(run & 0xffffffffull);
        const int scene = scn[j];
        a.block_range[b] = make_uint2(start, count);
        a.emig_count[b] = 0u;
        if (count) {
            const BlockItem e{b, start, count, (uint32_t)scene};
            if (count >= kDenseBlock) {
                a.dense_list[cnext[7]++] = e;
                atomicMax(&a.counters[kSortMaxWord], count);
            } else if (count >= kBigItem) a.sort_list[cnext[5]++] = e;
            else a.sort_list[a.sort_list_cap - 1 - cnext[6]++] = e;
        }
        // a block's items have count / items particles, the first
        // count % items of them one more (sizes differ by at most one)
        if (items) {
            const uint32_t slot = (uint32_t)(run >> 32);
            splitItems(a.active + slot, b, start, count, items, (uint32_t)scene);
            a.block_slot[b] = make_int2((int)slot, (int)items);
            // G2P's items of the block, in its combination's list at slots
            // taken from a counter (their order does not matter)
            const int k = a.scenes[scene].combo;
            const uint32_t parts = (count + a.split.g2p_chunk[k] - 1) / a.split.g2p_chunk[k];
            uint32_t g0;
            if (warp_fast) {
                g0 = gnext;
                gnext += parts;
            } else {
                g0 = atomicAdd(&a.counters[kG2PCountWord + k], parts);
            }
            splitItems(a.g2p_items + (size_t)k * a.g2p_cap + g0, b, start, count, parts, (uint32_t)scene);
            if (a.p2g_lists) {
                const uint32_t size = (count + items - 1) / items;
                const int cls = size <= a.split.p2g_warp_max[k] ? 0 : (size >= kBigItem ? 1 : 2);
                uint32_t p0;
                if (warp_fast) {
                    p0 = cls == 0 ? cnext[0] : cls == 1 ? cnext[1] : cnext[2];
                    cnext[0] += cls == 0 ? items : 0u;
                    cnext[1] += cls == 1 ? items : 0u;
                    cnext[2] += cls == 2 ? items : 0u;
                } else {
                    p0 = atomicAdd(&a.counters[cls == 2 ? kP2GBackWord + k : kP2GListWord + 2 * k + cls], items);
                    if (size <= kWarpAutoMax) atomicAdd(&a.counters[kP2GSmallWord + k], items);
                }
                uint32_t* lst = a.p2g_lists + (size_t)(2 * k + (cls == 0 ? 0 : 1)) * a.p2g_list_cap;
                for (uint32_t q = 0; q < items; ++q) {
                    if (cls == 2) lst[a.p2g_list_cap - 1 - (p0 + q)] = slot + q;  // from the back
                    else lst[p0 + q] = slot + q;
                }
            }
        } else {
            a.block_slot[b] = make_int2(-1, 0);
            if (count > 0) {
                const uint32_t nitems = blockItems(count, a.scenes[scene].n);
                const uint32_t o = atomicAdd(&a.counters[1], nitems);
                atomicAdd(&a.counters[3], 1u);
                splitItems(a.outside + o, b, start, count, nitems, (uint32_t)scene);
            }
        }
        a.block_count[b] = 0;
        run += v;
    }
}

__global__ void __launch_bounds__(kCompactThreads) compactOnesweepKernel(CompactArgs a, unsigned long long* __restrict__ status,
                                                                  uint32_t* __restrict__ tile_counter, uint32_t ntiles) {
    __shared__ uint32_t tile_s;
    __shared__ unsigned long long tot, excl_s;
    if (threadIdx.x == 0) tile_s = atomicAdd(tile_counter, 1u);
    __syncthreads();
    const uint32_t tile = tile_s;
    const uint32_t b0 = tile * kCompactTile + threadIdx.x * kCompactPer;
    unsigned long long packed[kCompactPer];
    int scn[kCompactPer];
    unsigned long long sum = 0;
#pragma unroll
    for (int j = 0; j < kCompactPer; ++j) sum += packed[j] = blockLoad(a, b0 + j, &scn[j]);
    unsigned long long run = blockExclusiveScanU64<kCompactThreads / 32>(sum, &tot);
    if (threadIdx.x == 0) {
        unsigned long long excl = 0;
        if (tile == 0) {
            atomicExch(&status[0], kCFlagPrefix | tot);
        } else {
            atomicExch(&status[tile], kCFlagAgg | tot);
            // 8 predecessor words per round trip (independent loads)
            int t = (int)tile - 1;
            int polls = 0;
            bool done = false;
            while (!done && t >= 0) {
                unsigned long long w[8];
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    w[q] = (t - q >= 0) ? *(volatile const unsigned long long*)(status + (t - q)) : kCFlagPrefix;
                bool waiting = false;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    if (done || waiting) continue;
                    const unsigned long long f = w[q] & kCFlagMask;
                    if (f == 0) {  // not published yet: poll again from this tile
                        waiting = true;
                        continue;
                    }
                    excl += w[q] & ~kCFlagMask;
                    --t;
                    if (f == kCFlagPrefix) done = true;
                }
                if (waiting) {
                    if (++polls > (1 << 22)) {  // never expected: give up instead of hanging
                        atomicOr(a.err, 16u);
                        break;
                    }
                    __nanosleep(32);
                }
            }
            atomicExch(&status[tile], kCFlagPrefix | (excl + tot));
        }
        excl_s = excl;
        if (tile == ntiles - 1) a.counters[0] = (uint32_t)((excl + tot) >> 32);
    }
    __syncthreads();
    run += excl_s;
    if (tile == 0 && threadIdx.x < 4) a.moved[threadIdx.x] = 0u;
    placeBlocks<kCompactPer>(a, b0, packed, scn, run);
}

// The same compaction by one cluster of eight CTAs of 1024 threads, one block a
// thread, for scenes of at most kClusterBlocks blocks: the CTAs read one
// another's totals from shared memory.  No status words to clear, no look-back
// and no clear of the counters ahead of it (the first CTA zeroes them before
// the cluster barrier).  What bounds both is the latency of a few dependent
// reads and atomics (65k-particle cube, 5,833 blocks: clear and compaction
// 13.5 us, this one 9.0).  With more blocks a thread, eight SMs write the
// dense block table more slowly than the whole GPU does in the kernel above
// (two-ball scene, 36k blocks: 0.020 ms more a step).
constexpr int kClusterCtas = 8, kClusterThreads = 1024;
constexpr uint32_t kClusterBlocks = kClusterCtas * kClusterThreads;

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads, 1)
    compactClusterKernel(CompactArgs a) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ unsigned long long tot;
    const uint32_t rank = cluster.block_rank(), b0 = rank * kClusterThreads + threadIdx.x;
    if (rank == 0) {
        const int t = threadIdx.x;
        if (t < 4) a.counters[t] = 0u;
        if (t < kMaxCombos) a.counters[kG2PCountWord + t] = 0u;
        if (t >= kP2GListWord && t < kSortSchedWord) a.counters[t] = 0u;
        if (t < 4) a.moved[t] = 0u;
    }
    unsigned long long packed[1];
    int scn[1];
    packed[0] = blockLoad(a, b0, &scn[0]);
    unsigned long long run = blockExclusiveScanU64<kClusterThreads / 32>(packed[0], &tot), total = 0;
    cluster.sync();  // every CTA's total is in its `tot`, the counters are zero
#pragma unroll
    for (int r = 0; r < kClusterCtas; ++r) {
        const unsigned long long x = *cluster.map_shared_rank(&tot, r);
        if (r < (int)rank) run += x;
        total += x;
    }
    cluster.barrier_arrive();
    if (rank == 0 && threadIdx.x == 0) a.counters[0] = (uint32_t)(total >> 32);
    placeBlocks<1>(a, b0, packed, scn, run);
    cluster.barrier_wait();  // the others have read this CTA's total
}

// ---------------------------------------------------------------------------
// tau from Fe/Fp for the live order (first step, after uploads).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) stressKernel(const SceneDev* __restrict__ scenes, int parity) {
    const SceneDev& sc = scenes[blockIdx.y];
    float* f = sc.buf[parity].f;
    const uint16_t* mat = sc.buf[parity].mat;
    const size_t cap = sc.cap;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < sc.n; i += gridDim.x * kThreads) {
        float Fe[9], Fp[9], tau[6];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            Fe[k] = f[(F_FE + k) * cap + i];
            Fp[k] = f[(F_FP + k) * cap + i];
        }
        // Fe = I (a new scene): tau = 0 exactly for both models (R = I,
        // J = 1), without the FP32 SVD's round-off in s (~1e-7), which a
        // stiff material turns into a spurious force at light surface nodes.
        bool identity = true;
#pragma unroll
        for (int k = 0; k < 9; ++k) identity = identity && Fe[k] == ((k % 4 == 0) ? 1.f : 0.f);
        if (identity) {
#pragma unroll
            for (int k = 0; k < 6; ++k) f[(F_TAU + k) * cap + i] = 0.f;
            continue;
        }
        MaterialDev m = sc.mats[sc.nmat > 1 ? mat[i] : 0];
        stressFromFe(m, Fe, Fp, f[F_VOL * cap + i], tau);
        if (m.model == MPM_MODEL_NEO_HOOKEAN)
#pragma unroll
            for (int k = 0; k < 9; ++k) f[(F_FE + k) * cap + i] = Fe[k];
#pragma unroll
        for (int k = 0; k < 6; ++k) f[(F_TAU + k) * cap + i] = tau[k];
    }
}

// ---------------------------------------------------------------------------
// P2G.  The unit of summation is a row: the (up to) four cells of a block that
// follow one another along x, so their particles follow one another in sorted
// order.  A warp takes whole rows and keeps a window of S nodes along x, for
// all S^2 columns (offsets b, c along y, z), in its lanes' registers: when the
// row's particles have passed a node, its sums leave the window.  So a row
// leaves one partial of (S+3) x S^2 nodes where one partial per cell would be
// four of S^3.  The lanes form G groups that take a cell's particles in turn;
// a lane holds kCols columns.  Every sum has a fixed order (a group's
// particles in sorted order, the groups in a fixed tree, rows in order), there
// are no floating-point atomics, and which warp takes a row does not matter:
// bitwise deterministic.
//
// What bounds it: instruction issue and, in the inner loop, what a lane reads
// per particle -- a 16-byte shared-memory load keeps the SM's load path busy
// for four cycles, broadcast or not.  Hence the staging forms everything that
// depends on the particle and one axis only.  With X, Y, Z the spline factors
// of node (a, b, c) and X', Y', Z' their derivatives, a node's share of
// (momentum + dt force)_i is
//   w XX_a^i + X_a R^i,   w = Y_b Z_c,   R^i = Z_c Y_b^i + Y_b Z_c^i
//   XX_a^i = X_a (q_i + a hC_i0) + X'_a T_i0
//   Y_b^i  = b Y_b hC_i1 + Y'_b T_i1,   Z_c^i = c Z_c hC_i2 + Z'_c T_i2
// (q = m v - m C delta, hC = h m C with C = B D^-1, T = stress term): 28 floats
// read and 16 __ffma2_rn per particle and column for cubic splines.  Against
// one partial per cell with the column factors formed in the inner loop (42
// floats): two-ball scene (1M particles, 35 a cell) 0.134 -> 0.099 ms and 77M ->
// 50M warp instructions, 8.4M-particle slab (3 a cell) 1.18 -> 0.95 ms, 2M
// particles quadratic (36 a cell) 0.198 -> 0.139 ms, 65k-particle cube 0.035 ->
// 0.021 ms.
//
// Staged payload of a particle, in 16-byte words (an odd number, so that the
// same word of eight particles lies in different banks):
//   APIC fused : (XX_a^x XX_a^y XX_a^z m X_a) [S] | X_0.. | (Y_b^x Y_b^y Y_b^z Y_b) [S] | (Z_c^i, Z_c) [S]
//   PIC-FLIP   : (m v, m) | X_0.. | X'_0.. | (T_i0, -) | (Y'_b T_i1, Y_b) [S] | (Z'_c T_i2, Z_c) [S]
//                momentum w X_a m v, force X'_a w T_i0 + X_a R^i
//   SPLIT      : the first with T = 0, then X' | T_i0 | (Y'_b T_i1, -) [S] | (Z'_c T_i2, -) [S]
//   MASS       : m X_0.. | Y_0.. | Z_0..
//   HESS       : PIC-FLIP's without the first (the force of the semi-implicit
//                solver's T = V0 dP Fe^T, not symmetric)
// ---------------------------------------------------------------------------
// One lane's sums for one stencil node, in packed FP32 pairs so that two
// components go through one __ffma2_rn (two exactly rounded FMAs):
//   pxy = (p_x, p_y), pzm = (p_z, m), fxy = (f_x, f_y), fz = f_z.
// Field f of the tile layout (m, p[3], f[3]) is get(f).
struct NodeAcc {
    float2 pxy, pzm, fxy;
    float fz;
    __device__ __forceinline__ void zero() {
        pxy = pzm = fxy = make_float2(0.f, 0.f);
        fz = 0.f;
    }
    __device__ __forceinline__ float get(int f) const {
        return f == 0 ? pzm.y : f == 1 ? pxy.x : f == 2 ? pxy.y : f == 3 ? pzm.x : f == 4 ? fxy.x : f == 5 ? fxy.y : fz;
    }
};

// A staged particle's layout (offsets in 16-byte words).
template <int S, int MODE>
struct P2GStage {
    static constexpr int F = modeFields(MODE);
    static constexpr int T = S + 3;                   // nodes of a row along x
    static constexpr int TN = tileNodes(S);
    static constexpr bool kC = MODE == MODE_APIC_FUSED || MODE == MODE_SPLIT;  // XX words
    static constexpr bool kMom = MODE != MODE_HESS;                            // mass and momentum
    static constexpr bool kSepF = MODE == MODE_FLIP || MODE == MODE_SPLIT || MODE == MODE_HESS;  // force apart from momentum
    static constexpr int WXX = 0;                     // XX (or m v, m)
    static constexpr int WX = MODE == MODE_MASS || !kMom ? 0 : (kC ? S : 1);
    static constexpr int WXD = WX + 1;                // X' (kSepF), then T_i0
    static constexpr int WT = WXD + 1;
    static constexpr int WY = MODE == MODE_MASS ? 1 : (kSepF ? WT + 1 : WX + 1);
    static constexpr int WZ = WY + (MODE == MODE_MASS ? 1 : S);
    static constexpr int WYF = MODE == MODE_SPLIT ? WZ + S : WY;  // the force's Y and Z words
    static constexpr int WZF = MODE == MODE_SPLIT ? WYF + S : WZ;
    static constexpr int kWords = WZF + (MODE == MODE_MASS ? 1 : S);
    static constexpr int P4 = kWords | 1;             // 16-byte words per staged particle
    static constexpr int kSeg = 192;                  // particles per row segment (at most)
};

// How a warp's lanes share a row: G particle groups, each lane one column:
// lane = group + G (b + S c).  (Two columns a lane and 4 groups for cubic, the
// three of a b and 8 groups for quadratic read half as much shared memory per
// particle, but double or treble the accumulators and the sums over the groups
// at every flushed node: two-ball P2G 0.102 against 0.104 ms, 2M-particle
// quadratic scene 0.143 against 0.139 ms, 8.4M-particle slab 1.12 against
// 0.95 ms.)
template <int S, int MODE>
struct P2GLanes {
    static constexpr int F = modeFields(MODE);
    static constexpr int G = S == 4 ? 2 : (S == 3 ? 3 : 8);
    // A flushed node's F values are summed over the groups; a lane then owns
    // kOut of them (see groupReduce).
    static constexpr int half(int n) { return (n + 1) / 2; }
    static constexpr int kOut = G == 3 ? F : G == 2 ? half(F) : half(half(half(F)));
    int grp, b, c;
    bool on;
    __device__ __forceinline__ explicit P2GLanes(int lane) {
        grp = lane % G;
        b = (lane / G) % S;
        c = (lane / G) / S;
        on = c < S;
    }
    // The first particle >= lo (index in its segment) that this lane's group
    // takes: a segment's particles go to the groups in turn, however it is
    // cut into passes and cells.
    __device__ __forceinline__ int first(int lo) const {
        const int r = lo % G;
        return grp >= r ? grp - r : grp - r + G;
    }
};

// Sums over the groups of the warp of the values v[0..N-1].  A power of two of
// groups: halving exchanges (each step a lane passes on half of its values and
// adds the other half), the lane's share ends up in v[0..kOut-1].  Three
// groups: added in turn, valid in group 0.
template <int N, int BIT, int G>
__device__ __forceinline__ void groupReduce(float* v, int lane) {
    if constexpr (G == 3) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float s1 = __shfl_down_sync(0xffffffffu, v[i], 1), s2 = __shfl_down_sync(0xffffffffu, v[i], 2);
            v[i] = (v[i] + s1) + s2;
        }
    } else if constexpr (BIT < G) {
        constexpr int H = (N + 1) / 2;
        const bool up = (lane & BIT) != 0;
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const float hi = i + H < N ? v[i + H] : 0.f;
            const float mine = up ? hi : v[i], other = up ? v[i] : hi;
            v[i] = mine + __shfl_xor_sync(0xffffffffu, other, BIT);
        }
        groupReduce<H, 2 * BIT, G>(v, lane);
    }
}
// The index of the value that ends up in v[i] of a lane of
// group `grp`, or -1 where the lane has none.
template <int N, int BIT, int G>
__device__ __forceinline__ int valueOf(int i, int grp) {
    if constexpr (G == 3) {
        return grp == 0 ? i : -1;
    } else if constexpr (BIT < G) {
        constexpr int H = (N + 1) / 2;
        const int k = valueOf<H, 2 * BIT, G>(i, grp);
        if (k < 0) return -1;
        const int j = (grp & BIT) ? k + H : k;
        return j < N ? j : -1;
    } else {
        return i < N ? i : -1;
    }
}

// Origin (node index) of the (S+3)^3 tile of an active block: 4 B - 4 per axis.
__device__ __forceinline__ void tileOrigin(const SceneDev& sc, uint32_t block, int* t0) {
    const uint32_t lb = block - sc.block_base;
    t0[0] = 4 * (int)(lb % (uint32_t)sc.nb[0]) - 4;
    t0[1] = 4 * (int)((lb / (uint32_t)sc.nb[0]) % (uint32_t)sc.nb[1]) - 4;
    t0[2] = 4 * (int)(lb / ((uint32_t)sc.nb[0] * (uint32_t)sc.nb[1])) - 4;
}

// num / h with one correction by the remainder (Markstein's method): as exact
// as a division of these operands, in three instructions.
__device__ __forceinline__ float quotient(float num, float h, float inv_h) {
    const float q = num * inv_h;
    return fmaf(fmaf(-q, h, num), inv_h, q);
}

// What P2G reads of a particle, in registers: loaded one staging pass ahead, so
// that the loads are in flight while the warp accumulates the pass before.
template <int S, int MODE>
struct P2GRaw {
    using R = P2GStage<S, MODE>;
    float x[3], m, v[3], t[6], B[9];
    bool bad;  // range check failed: the particle contributes nothing
    __device__ __forceinline__ void load(const StepArgs& args, const SceneDev& sc, const float* pf, size_t cap,
                                         uint32_t perm, uint32_t at) {
        if constexpr (MODE == MODE_HESS) {  // by sorted position: x holds the stencil offsets, B the matrix T
            const float4 q = args.solve_pofs[at];
            x[0] = q.x, x[1] = q.y, x[2] = q.z;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const float4 row = args.solve_T[3 * (size_t)at + r];
                B[3 * r] = row.x, B[3 * r + 1] = row.y, B[3 * r + 2] = row.z;
            }
            return;
        }
        uint32_t old = perm - sc.key_offset;
        bad = old >= sc.n;
        if (bad) {
            atomicOr(args.err, ERR_INDEX);
            old = 0;
        }
        const float* pp = pf + old;
#pragma unroll
        for (int a = 0; a < 3; ++a) x[a] = ldg(pp + (F_X + a) * cap);
        m = ldg(pp + F_MASS * cap);
        if (MODE == MODE_MASS) return;
#pragma unroll
        for (int a = 0; a < 3; ++a) v[a] = ldg(pp + (F_V + a) * cap);
#pragma unroll
        for (int k = 0; k < 6; ++k) t[k] = ldg(pp + (F_TAU + k) * cap);
        if (MODE == MODE_APIC_FUSED || (MODE == MODE_SPLIT && sc.transfer == MPM_TRANSFER_APIC)) {
#pragma unroll
            for (int k = 0; k < 9; ++k) B[k] = ldg(pp + (F_B + k) * cap);
        } else if (MODE == MODE_SPLIT) {
#pragma unroll
            for (int k = 0; k < 9; ++k) B[k] = 0.f;
        }
    }
};

// Staging of one particle (of `cell` in the block whose tile starts at t0) at
// `my`, in the layout above.  The stencil base comes from the cell, which the
// key was formed from.
template <int S, int MODE>
__device__ __forceinline__ void p2gStageParticle(const SceneDev& sc, const P2GRaw<S, MODE>& raw, float dt, float h,
                                                 float inv_h, const int* t0, uint32_t cell, float4* my) {
    using R = P2GStage<S, MODE>;
    const float (&x)[3] = raw.x;
    const float (&v)[3] = raw.v;
    const float m = MODE == MODE_HESS || raw.bad ? 0.f : raw.m;
    float t[6], mC[9];
    if (MODE != MODE_MASS && MODE != MODE_HESS) {
        const float ts = raw.bad ? 0.f : (MODE == MODE_APIC_FUSED ? -dt : -1.0f);
#pragma unroll
        for (int k = 0; k < 6; ++k) t[k] = ts * raw.t[k];
        if (R::kC) {
            const float md = m * sc.dinv;
#pragma unroll
            for (int k = 0; k < 9; ++k) mC[k] = md * raw.B[k];
        }
    }
    const int base[3] = {t0[0] + (int)(cell & 3u), t0[1] + (int)((cell >> 2) & 3u), t0[2] + (int)(cell >> 4)};
    float delta[3], wk[3][S], dwk[3][S];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float gp0 = __fadd_rn(sc.origin[a], __fmul_rn(h, (float)base[a]));
        delta[a] = x[a] - gp0;
        // Node distances.  The linear kernel's weights have relative error
        // ~ulp(d)/w near |d| = 1, so it forms each one as the reference does,
        // (x_p - (o + h i)) / h; the B-splines are smooth there and use
        // d0 - k (exact subtraction).
        float dk[S];
        if (MODE == MODE_HESS) {
#pragma unroll
            for (int k = 0; k < S; ++k) dk[k] = x[a] - (float)k;
        } else if (S == 2) {
#pragma unroll
            for (int k = 0; k < S; ++k) {
                const float gp = __fadd_rn(sc.origin[a], __fmul_rn(h, (float)(base[a] + k)));
                dk[k] = quotient(__fsub_rn(x[a], gp), h, inv_h);
            }
        } else {
            dk[0] = quotient(delta[a], h, inv_h);
#pragma unroll
            for (int k = 1; k < S; ++k) dk[k] = dk[0] - (float)k;
        }
        splineWeights<S>(dk, wk[a], dwk[a]);
#pragma unroll
        for (int k = 0; k < S; ++k) dwk[a][k] *= inv_h;
    }
    auto row4 = [](const float* w) {
        return make_float4(w[0], w[1], S > 2 ? w[S > 2 ? 2 : 0] : 0.f, S > 3 ? w[S > 3 ? 3 : 0] : 0.f);
    };
    if (MODE == MODE_MASS) {
        float mx[S];
#pragma unroll
        for (int k = 0; k < S; ++k) mx[k] = m * wk[0][k];
        my[R::WXX] = row4(mx);
        my[R::WY] = row4(wk[1]);
        my[R::WZ] = row4(wk[2]);
        return;
    }
    my[R::WX] = row4(wk[0]);
    if (R::kC) {
        float q[3], hC[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            q[i] = m * v[i] - (mC[3 * i] * delta[0] + mC[3 * i + 1] * delta[1] + mC[3 * i + 2] * delta[2]);
#pragma unroll
        for (int k = 0; k < 9; ++k) hC[k] = h * mC[k];
        const float tx[3] = {t[0], t[3], t[4]}, ty[3] = {t[3], t[1], t[5]}, tz[3] = {t[4], t[5], t[2]};
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const float wy = (float)k * wk[1][k], wz = (float)k * wk[2][k];
            float xx[3], yy[3], zz[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                xx[i] = wk[0][k] * fmaf((float)k, hC[3 * i], q[i]);
                yy[i] = wy * hC[3 * i + 1];
                zz[i] = wz * hC[3 * i + 2];
                if (MODE == MODE_APIC_FUSED) {
                    xx[i] = fmaf(dwk[0][k], tx[i], xx[i]);
                    yy[i] = fmaf(dwk[1][k], ty[i], yy[i]);
                    zz[i] = fmaf(dwk[2][k], tz[i], zz[i]);
                }
            }
            my[R::WXX + k] = make_float4(xx[0], xx[1], xx[2], m * wk[0][k]);
            my[R::WY + k] = make_float4(yy[0], yy[1], yy[2], wk[1][k]);
            my[R::WZ + k] = make_float4(zz[0], zz[1], zz[2], wk[2][k]);
        }
    } else if (R::kMom) {
        my[R::WXX] = make_float4(m * v[0], m * v[1], m * v[2], m);
    }
    if (MODE == MODE_HESS) {
        const float (&B)[9] = raw.B;
        my[R::WXD] = row4(dwk[0]);
        my[R::WT] = make_float4(B[0], B[3], B[6], 0.f);
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const float dy = dwk[1][k], dz = dwk[2][k];
            my[R::WYF + k] = make_float4(dy * B[1], dy * B[4], dy * B[7], wk[1][k]);
            my[R::WZF + k] = make_float4(dz * B[2], dz * B[5], dz * B[8], wk[2][k]);
        }
    } else if (R::kSepF) {
        my[R::WXD] = row4(dwk[0]);
        my[R::WT] = make_float4(t[0], t[3], t[4], 0.f);
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const float dy = dwk[1][k], dz = dwk[2][k];
            my[R::WYF + k] = make_float4(dy * t[3], dy * t[1], dy * t[5], wk[1][k]);
            my[R::WZF + k] = make_float4(dz * t[4], dz * t[5], dz * t[2], wk[2][k]);
        }
    }
}

__device__ __forceinline__ float pick(const float4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
__device__ __forceinline__ float2 dup2(float x) { return make_float2(x, x); }

// One lane's sums over the staged particles q0, q0 + G, ... below qhi (its
// group's share of a cell at x offset X in its row, in order) for the column
// (b, c).  The window's register of tile node n is n % S, so the cell's nodes a
// sit in acc[(X + a) % S].
template <int S, int MODE, int X>
__device__ __forceinline__ void p2gAccumulate(const float4* st, int q0, int qhi, int b, int c, NodeAcc (&acc)[S]) {
    using R = P2GStage<S, MODE>;
#pragma unroll 1
    for (int q = q0; q < qhi; q += P2GLanes<S, MODE>::G) {
        const float4* pq = st + q * R::P4;
        if (MODE == MODE_MASS) {
            const float4 xm = pq[R::WXX];
            const float w = reinterpret_cast<const float*>(pq + R::WY)[b] * reinterpret_cast<const float*>(pq + R::WZ)[c];
#pragma unroll
            for (int a = 0; a < S; ++a) acc[(X + a) % S].pzm.y = fmaf(w, pick(xm, a), acc[(X + a) % S].pzm.y);
            continue;
        }
        const float4 xw = pq[R::WX], y = pq[R::WY + b], z = pq[R::WZ + c];
        const float w = y.w * z.w;
        const float2 w2 = dup2(w);
        if (R::kC) {
            const float2 Rxy = __ffma2_rn(dup2(z.w), make_float2(y.x, y.y), __fmul2_rn(dup2(y.w), make_float2(z.x, z.y)));
            const float2 Rz0 = make_float2(fmaf(z.w, y.z, y.w * z.z), 0.f);
#pragma unroll
            for (int a = 0; a < S; ++a) {
                NodeAcc& n = acc[(X + a) % S];
                const float4 xx = pq[R::WXX + a];
                const float2 xa = dup2(pick(xw, a));
                n.pxy = __ffma2_rn(w2, make_float2(xx.x, xx.y), __ffma2_rn(xa, Rxy, n.pxy));
                n.pzm = __ffma2_rn(w2, make_float2(xx.z, xx.w), __ffma2_rn(xa, Rz0, n.pzm));
            }
        } else if (R::kMom) {
            const float4 mv = pq[R::WXX];
            const float2 Pxy = __fmul2_rn(w2, make_float2(mv.x, mv.y)), Pzm = __fmul2_rn(w2, make_float2(mv.z, mv.w));
#pragma unroll
            for (int a = 0; a < S; ++a) {
                NodeAcc& n = acc[(X + a) % S];
                const float2 xa = dup2(pick(xw, a));
                n.pxy = __ffma2_rn(xa, Pxy, n.pxy);
                n.pzm = __ffma2_rn(xa, Pzm, n.pzm);
            }
        }
        if (R::kSepF) {
            const float4 xd = pq[R::WXD], t0 = pq[R::WT];
            const float4 yf = MODE == MODE_SPLIT ? pq[R::WYF + b] : y, zf = MODE == MODE_SPLIT ? pq[R::WZF + c] : z;
            const float2 Rxy =
                __ffma2_rn(dup2(z.w), make_float2(yf.x, yf.y), __fmul2_rn(dup2(y.w), make_float2(zf.x, zf.y)));
            const float Rz = fmaf(z.w, yf.z, y.w * zf.z);
            const float2 Bxy = __fmul2_rn(w2, make_float2(t0.x, t0.y));
            const float Bz = w * t0.z;
#pragma unroll
            for (int a = 0; a < S; ++a) {
                NodeAcc& n = acc[(X + a) % S];
                const float xa = pick(xw, a), da = pick(xd, a);
                n.fxy = __ffma2_rn(dup2(da), Bxy, __ffma2_rn(dup2(xa), Rxy, n.fxy));
                n.fz = fmaf(da, Bz, fmaf(xa, Rz, n.fz));
            }
        }
    }
}

// A warp's state within a row segment, and one staging pass of it.
template <int S, int MODE>
struct RowWindow {
    using L = P2GLanes<S, MODE>;
    NodeAcc acc[S];
    int col;         // tile x of the first node still in the window
    unsigned cells;  // cells of the segment that had particles
    __device__ __forceinline__ void reset() {
        col = 0;
        cells = 0u;
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int a = 0; a < S; ++a) acc[a].zero();
        reset();
    }
    // Tile node n along x is final: its sums over the groups go to out(n, v),
    // v the lane's share; where no cell touched it, out(n, null).
    template <int N, class Out>
    __device__ __forceinline__ void flush(int lane, Out&& out) {
        constexpr unsigned touch = ((((1u << S) - 1u) << N) >> (S - 1)) & 15u;  // cells N - S + 1 .. N
        if (cells & touch) {
            float v[L::F];
#pragma unroll
            for (int f = 0; f < L::F; ++f) v[f] = acc[N % S].get(MODE == MODE_HESS ? 4 + f : f);
            acc[N % S].zero();
            groupReduce<L::F, 1, L::G>(v, lane);
            out(N, v);
        } else {
            out(N, (const float*)nullptr);
        }
    }
    // The staged particles [qlo, qhi) of a pass, which belong to one segment of
    // row `row`; cl is the lane's staged particle's cell, j0 the index in the
    // segment of particle qlo.  Nodes x < lim are final after it (lim = 4:
    // the segment ends, and all are).
    template <class Out>
    __device__ __forceinline__ void pass(const float4* st, uint32_t cl, int qlo, int qhi, int row, int j0, int lim,
                                         int lane, const L& ln, Out&& out) {
        const bool mine = lane >= qlo && lane < qhi;
        step<0>(st, cl, mine, qlo, row, j0, lim, lane, ln, out);
        step<1>(st, cl, mine, qlo, row, j0, lim, lane, ln, out);
        step<2>(st, cl, mine, qlo, row, j0, lim, lane, ln, out);
        step<3>(st, cl, mine, qlo, row, j0, lim, lane, ln, out);
        if (lim == 4) {
            flush<4>(lane, out);
            if constexpr (S > 2) flush<5>(lane, out);
            if constexpr (S > 3) flush<6>(lane, out);
            reset();
        }
    }
    template <int X, class Out>
    __device__ __forceinline__ void step(const float4* st, uint32_t cl, bool mine, int qlo, int row, int j0, int lim,
                                         int lane, const L& ln, Out&& out) {
        const unsigned m = __ballot_sync(0xffffffffu, mine && cl == (uint32_t)(4 * row + X));
        if (m) {
            const int a = __ffs(m) - 1, e = a + __popc(m);
            if (ln.on) p2gAccumulate<S, MODE, X>(st, a + ln.first(j0 + a - qlo), e, ln.b, ln.c, acc);
            cells |= 1u << X;
        }
        if (X < lim && col == X) {
            flush<X>(lane, out);
            col = X + 1;
        }
    }
};

// A block of several items (slot = first slot, items): counts this item's tile
// as written and says whether it was the last one; the count goes back to
// zero for the next launch.  The caller's writes of the tile are fenced.
__device__ __forceinline__ int lastOfBlock(const StepArgs& args, int2 slot) {
    if (atomicAdd(&args.tile_done[slot.x], 1u) != (uint32_t)slot.y - 1u) return 0;
    args.tile_done[slot.x] = 0u;
    __threadfence();
    return 1;
}
// Adds a block's tiles of N floats up in item order, into its first one
// (thread t of nt; read from L2, where the other items' writes are).
template <int N>
__device__ __forceinline__ void mergeItemTiles(const StepArgs& args, int2 slot, int t, int nt) {
    float* first = args.tiles + (size_t)slot.x * args.tile_stride;
    for (int q = t; q < N; q += nt) {
        float sum = __ldcg(first + q);
#pragma unroll 8
        for (int s = 1; s < slot.y; ++s) sum += __ldcg(first + (size_t)s * args.tile_stride + q);
        first[q] = sum;
    }
}

// Row starts of an item's `count` particles (keys sorted by cell): row r's
// particles are [beg[r], beg[r + 1]), r < 16.  Thread t of nt writes those of
// the rows that begin at its particles.
__device__ __forceinline__ void findRows(const uint32_t* keys, int count, int* beg, int t, int nt) {
#pragma unroll 4
    for (int i = t; i < count; i += nt) {
        const int r = (int)((keys[i] & 63u) >> 2), before = i ? (int)((keys[i - 1] & 63u) >> 2) : -1;
        for (int q = before + 1; q <= r; ++q) beg[q] = i;
        if (i == count - 1)
            for (int q = r + 1; q <= 16; ++q) beg[q] = count;
    }
}

template <int S, int MODE, int STAGE>
struct P2GLayout : P2GStage<S, MODE> {
    using R = P2GStage<S, MODE>;
    static constexpr int F = R::F, T = R::T;
    static constexpr int kStage = STAGE;              // particles staged per warp pass
    static constexpr int kSlots = 16;                 // segment partials per round: a block's rows, one segment each
    // Floats between a partial's x nodes: with 18 (cubic), 9 (quadratic) and
    // 4 (linear) the gather's (x, y) neighbours fall in different banks.
    static constexpr int CS = S == 4 ? 18 : S * S;
    static constexpr int kSlotFloats = F * T * CS;
    static constexpr int kMaxSeg = 32;                // >= 16 + kBlockChunk / kSeg + 1
    static constexpr int kCtlInts = 17 + 3 * kMaxSeg + 4 + 3;
    // dynamic shared memory of nw warps: stage [nw][kStage][P4] 16-byte words,
    // partials [kSlots][F][T][CS] floats, then the control ints (rowBeg[17],
    // segRow/segBeg/segEnd[kMaxSeg], ctl[4]); the kernel takes its pointers
    // from these offsets
    static constexpr size_t smemFor(int nw) {
        return (size_t)nw * kStage * R::P4 * 16 + (size_t)kSlots * kSlotFloats * 4 + (size_t)kCtlInts * 4;
    }
    static constexpr bool kThreeOf8 = (smemFor(8) + 1024) * 3 <= 228 * 1024;
    // Threads per CTA: three CTAs of 8 warps per SM where the shared memory
    // holds them (228 KB per SM, 1 KB of it reserved per CTA), else two.
    static constexpr int NT = 256;
    static constexpr int NW = NT / 32;
    static constexpr int MIN_CTAS = kThreeOf8 && S * F <= 16 ? 3 : 2;
    static constexpr int TJ = (R::TN + NT - 1) / NT;
    static constexpr size_t kPartialOff = (size_t)NW * kStage * R::P4 * 4;  // floats
    static constexpr size_t kCtlOff = kPartialOff + (size_t)kSlots * kSlotFloats;
    static constexpr size_t smemBytes = smemFor(NW);
    static_assert(smemBytes == kCtlOff * 4 + (size_t)kCtlInts * 4, "layout");
    static_assert(kMaxSeg >= 16 + (int)(kBlockChunk / R::kSeg) + 1, "segment list too small");
    static_assert(kSlots <= 32 && kStage <= 32, "a round's segments and a pass's particles: one per lane");
};

template <int S, int MODE, int STAGE>
__global__ void __launch_bounds__(P2GLayout<S, MODE, STAGE>::NT, P2GLayout<S, MODE, STAGE>::MIN_CTAS)
    p2gKernel(StepArgs args, int want_transfer) {
    using L = P2GLayout<S, MODE, STAGE>;
    constexpr int F = L::F, T = L::T, TN = L::TN, CS = L::CS;
    extern __shared__ float4 smem4[];
    float* smem = reinterpret_cast<float*>(smem4);
    float* partial = smem + L::kPartialOff;  // [slot][F][T][CS]
    int* rowBeg = (int*)(smem + L::kCtlOff); // item index of each row's first particle, then the item's count
    int* segRow = rowBeg + 17;                                  // segment list, in row order
    int* segBeg = segRow + L::kMaxSeg;
    int* segEnd = segBeg + L::kMaxSeg;
    int* ctl = segEnd + L::kMaxSeg;                             // [0] segments, [1] next window

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4* st = smem4 + (size_t)warp * L::kStage * L::P4;
    // the combination's list of items for whole CTAs, or every active item
    const uint32_t* list = args.p2g_lists ? args.p2g_lists + (size_t)(2 * args.combo + 1) * args.p2g_list_cap : nullptr;
    // the long items from the list's front first, then the others from its
    // back, then -- unless the warp kernel takes them -- the small items
    const uint32_t nfront = list ? args.counters[kP2GListWord + 2 * args.combo + 1] : 0u;
    const uint32_t nlist1 = list ? nfront + args.counters[kP2GBackWord + args.combo] : 0u;
    const uint32_t nsmall = list ? args.counters[kP2GListWord + 2 * args.combo] : 0u;
    const uint32_t nwork = !list ? args.counters[0]
                                 : nlist1 + (p2gWarpTakesSmall(args.p2g_warp, nsmall) ? 0u : nsmall);
    const uint32_t* small = list ? args.p2g_lists + (size_t)(2 * args.combo) * args.p2g_list_cap : nullptr;
    const int solve_k = MODE == MODE_HESS && args.solve_iter ? args.solve_iter[0] : -1;
    if (MODE == MODE_HESS && args.solve_iter && args.solve_iter[1]) return;  // every scene has converged
    spanBegin(args.spans, SPAN_P2G);
    __shared__ uint32_t item_s;
    __shared__ SceneDev sc_s;
    for (;;) {
        const uint32_t wi = nextWorkItem(args.sched, nwork, &item_s);
        if (wi >= nwork) break;
        const uint32_t w = !list ? wi
                           : wi < nfront ? list[wi]
                           : wi < nlist1 ? list[args.p2g_list_cap - 1 - (wi - nfront)]
                                         : small[wi - nlist1];
        const BlockItem it = args.active[w];
        {
            const SceneDev& scg = args.scenes[it.scene];
            if (scg.S != S || (want_transfer >= 0 && scg.transfer != want_transfer)) continue;
            if (MODE == MODE_MASS && !scg.init_pass) continue;
            if (MODE == MODE_HESS && !(scg.beta > 0.f && scg.solve.status->done_at > solve_k)) continue;
        }
        const uint32_t i0 = it.start;
        const int icount = (int)it.count;
        const uint32_t* keys = args.sorted_keys + i0;
        const uint32_t* perm = args.perm + i0;
        // the scene's entry into shared memory (the staging reads its fields
        // per particle)
        if (warp == 0) {
            const int4* src = reinterpret_cast<const int4*>(args.scenes + it.scene);
            int4* dst = reinterpret_cast<int4*>(&sc_s);
            for (int q = lane; q < (int)(sizeof(SceneDev) / 16); q += 32) dst[q] = src[q];
        }
        findRows(keys, icount, rowBeg, (int)threadIdx.x, L::NT);
        __syncthreads();
        if (warp == 0) {
            // Segment list: every non-empty row cut into equal runs of at most
            // kSeg particles, in row order (lane r < 16 owns row r).
            const int lo = lane < 16 ? rowBeg[lane] : 0, end = lane < 16 ? rowBeg[lane + 1] : 0;
            const int len = end - lo, n = (len + L::kSeg - 1) / L::kSeg;
            int x = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            int o = x - n;
            for (int j = 0; j < n; ++j, ++o) {
                segRow[o] = lane;
                segBeg[o] = lo + len * j / n;
                segEnd[o] = lo + len * (j + 1) / n;
            }
            if (lane == 31) {
                ctl[0] = x;
                ctl[1] = 0;
            }
        }
        __syncthreads();
        const SceneDev& sc = sc_s;
        const float* pf = sc.buf[args.parity].f;
        const size_t cap = sc.cap;
        const int nseg = ctl[0];
        float* tile = args.tiles + (size_t)w * args.tile_stride;

        const float dt = sc.dt, h = sc.h, inv_h = sc.inv_h;
        int t0[3];
        tileOrigin(sc, it.block, t0);
        // ---- particle phase of a round: warps take its segments dynamically ----
        // The round's particles [rb, re) are cut into windows (of kStage,
        // fewer where that leaves warps without one); a warp takes a window
        // and handles the segments that start in it: several sparse rows
        // share one staging pass, a long segment takes several.  Each segment
        // is summed by one warp, in order.
        auto particles = [&](int r0, int rend) {
            using LN = P2GLanes<S, MODE>;
            const LN ln(lane);
            // where the lane's share of a flushed node goes in a partial (-1: nowhere)
            int off[LN::kOut];
#pragma unroll
            for (int i = 0; i < LN::kOut; ++i) {
                const int k = valueOf<F, 1, LN::G>(i, ln.grp);
                off[i] = k < 0 || !ln.on ? -1 : k * T * CS + ln.b + S * ln.c;
            }
            const int rb = segBeg[r0], re = segEnd[rend - 1];
            const int win = min(L::kStage, (re - rb + L::NW - 1) / L::NW);
            const int nwin = (re - rb + win - 1) / win;
            RowWindow<S, MODE> rw;
            rw.clear();
            while (true) {
                int wi = 0;
                if (lane == 0) wi = atomicAdd(&ctl[1], 1);
                wi = __shfl_sync(0xffffffffu, wi, 0);
                if (wi >= nwin) break;
                const int sl = r0 + lane;  // one segment of the round per lane
                const bool starts = sl < rend && (segBeg[sl] - rb) / win == wi;
                const unsigned own = __ballot_sync(0xffffffffu, starts);
                if (!own) continue;
                const int s_last = r0 + 31 - __clz(own);
                int cur = r0 + __ffs(own) - 1;  // segment being summed
                const int ce0 = segEnd[s_last];
                // the loads of a pass are issued one pass ahead (the permutation
                // entries and keys two)
                const int gb = segBeg[cur];
                P2GRaw<S, MODE> raw;
                uint32_t cl = 0, ncl = 0, nperm = 0;
                const bool stages = lane < L::kStage;
                if (stages && gb + lane < ce0) {
                    cl = keys[gb + lane] & 63u;
                    raw.load(args, sc, pf, cap, perm[gb + lane], i0 + (uint32_t)(gb + lane));
                }
                if (stages && gb + L::kStage + lane < ce0) {
                    ncl = keys[gb + L::kStage + lane] & 63u;
                    nperm = perm[gb + L::kStage + lane];
                }
                for (int g0 = gb; g0 < ce0; g0 += L::kStage) {
                    const int np = min(L::kStage, ce0 - g0);
                    if (lane < np) p2gStageParticle<S, MODE>(sc, raw, dt, h, inv_h, t0, cl, st + lane * L::P4);
                    const uint32_t pcl = cl;  // this pass's cells
                    const int next_x = (int)(__shfl_sync(0xffffffffu, ncl, 0) & 3u);  // only read where the segment goes on
                    if (stages && g0 + L::kStage + lane < ce0)
                        raw.load(args, sc, pf, cap, nperm, i0 + (uint32_t)(g0 + L::kStage + lane));
                    cl = ncl;
                    if (stages && g0 + 2 * L::kStage + lane < ce0) {
                        ncl = keys[g0 + 2 * L::kStage + lane] & 63u;
                        nperm = perm[g0 + 2 * L::kStage + lane];
                    }
                    __syncwarp();
                    // the segments overlapping this pass, in order
                    while (cur <= s_last) {
                        const int sb = segBeg[cur], se = segEnd[cur];
                        const int qlo = max(sb, g0) - g0, qhi = min(se, g0 + np) - g0;
                        const bool ends = se <= g0 + np;
                        float* slot = partial + (size_t)(cur - r0) * L::kSlotFloats;
                        rw.pass(st, pcl, qlo, qhi, segRow[cur], g0 + qlo - sb, ends ? 4 : next_x, lane, ln,
                                [&](int n, const float* v) {
#pragma unroll
                                    for (int i = 0; i < LN::kOut; ++i)
                                        if (off[i] >= 0) slot[off[i] + n * CS] = v ? v[i] : 0.f;
                                });
                        if (!ends) break;  // the segment continues in the next pass
                        ++cur;
                    }
                    __syncwarp();
                }
            }
        };
        for (int r0 = 0; r0 < nseg; r0 += L::kSlots) {
            const int rend = min(nseg, r0 + L::kSlots);
            particles(r0, rend);
            __syncthreads();
            if (threadIdx.x == 0) ctl[1] = 0;  // next round's dynamic counter (no warp reads it until the barrier below)
            // ---- gather phase: fixed-order merge of this round's segments ----
            // (a later round adds to the tile that the same thread wrote before)
#pragma unroll 1
            for (int j = 0; j < L::TJ; ++j) {
                const int tn = threadIdx.x + j * L::NT;
                if (tn >= TN) break;
                const int tx = tn % T, ty = (tn / T) % T, tz = tn / (T * T);
                float sum[F];
#pragma unroll
                for (int f = 0; f < F; ++f) sum[f] = r0 ? tile[f * TN + tn] : 0.f;
                for (int sg = r0; sg < rend; ++sg) {
                    const int row = segRow[sg];
                    const int dy = ty - (row & 3), dz = tz - (row >> 2);
                    if ((unsigned)dy >= (unsigned)S || (unsigned)dz >= (unsigned)S) continue;
                    const float* pc = partial + (size_t)(sg - r0) * L::kSlotFloats + tx * CS + dy + S * dz;
#pragma unroll
                    for (int f = 0; f < F; ++f) sum[f] += pc[f * T * CS];
                }
#pragma unroll
                for (int f = 0; f < F; ++f) tile[f * TN + tn] = sum[f];
            }
            __syncthreads();
        }
        // the last of a block's items adds up their tiles
        const int2 slot = args.block_slot[it.block];
        if (slot.y > 1) {
            __shared__ int last_s;
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) last_s = lastOfBlock(args, slot);
            __syncthreads();
            if (last_s) mergeItemTiles<F * TN>(args, slot, (int)threadIdx.x, L::NT);
        }
    }
    spanEnd(args.spans, SPAN_P2G);
}


// ---------------------------------------------------------------------------
// P2G by whole warps for the small items (the combination's warp list).  Each
// warp takes an item and sums its particles row by row as p2gKernel does (the
// same segments, RowWindow) and adds the nodes that leave its window into its
// own shared-memory tile, segment after segment, the order of p2gKernel's
// merge: the tile is bitwise p2gKernel's, so which kernel takes an item
// changes no result.  No CTA barrier: an item of a few particles per cell
// spends most of p2gKernel's time in its per-item set-up, barriers and merge.
// ---------------------------------------------------------------------------
template <int S, int MODE>
struct P2GWarpLayout : P2GStage<S, MODE> {
    using R = P2GStage<S, MODE>;
    static constexpr int kStage = 32;  // particles staged per pass (8.4M-particle slab P2G 1.02, 1.00 and 0.95 ms at 16, 24, 32)
    // per warp: its item's scene entry, its tile [F][TN], its staging words
    // (field-major: neighbouring columns add to neighbouring banks; a
    // node-major tile of 16-byte words had bank conflicts and was slower)
    static constexpr int kSceneFloats = (int)((sizeof(SceneDev) + 15) / 16 * 4);
    static constexpr int kTileFloats = (R::F * R::TN + 3) / 4 * 4;
    static constexpr int kRowInts = 20;
    static constexpr int kWarpFloats = kSceneFloats + kTileFloats + kStage * R::P4 * 4 + kRowInts;
    // Two CTAs per SM of as many warps as its shared memory holds, at most 20 in
    // all: 96 registers a thread.  24 leave 80, where quadratic APIC spills 148
    // bytes a thread (24 at 96; step of 4M particles, 1 a cell: 2.452 and 2.171 ms,
    // 4 a cell 1.117 and 1.049; linear 2.260 and 2.235; quadratic PIC-FLIP and
    // cubic, bound by the shared memory, unchanged); 16 without spills: 2.207, 1.047
    // and 2.315.
    static constexpr int kWarpsPerSm = (int)(226u * 1024 / (kWarpFloats * 4));
    static constexpr int NW = (kWarpsPerSm < 20 ? kWarpsPerSm : 20) / 2, NT = 32 * NW;
    static constexpr size_t smemBytes = (size_t)NW * kWarpFloats * 4;
    static constexpr int MIN_CTAS = 2;
};

template <int S, int MODE>
__global__ void __launch_bounds__(P2GWarpLayout<S, MODE>::NT, P2GWarpLayout<S, MODE>::MIN_CTAS)
    p2gWarpKernel(StepArgs args) {
    using W = P2GWarpLayout<S, MODE>;
    constexpr int F = W::F, T = S + 3, TN = W::TN;
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* wbase = reinterpret_cast<float*>(smem4) + (size_t)warp * W::kWarpFloats;
    SceneDev& sc = *reinterpret_cast<SceneDev*>(wbase);
    float* tile = wbase + W::kSceneFloats;
    float4* st = reinterpret_cast<float4*>(tile + W::kTileFloats);
    int* rowBeg = reinterpret_cast<int*>(st + W::kStage * W::P4);
    using LN = P2GLanes<S, MODE>;
    const LN ln(lane);
    int off[LN::kOut];  // where the lane's share of a flushed node goes in the tile (-1: nowhere)
#pragma unroll
    for (int i = 0; i < LN::kOut; ++i) {
        const int k = valueOf<F, 1, LN::G>(i, ln.grp);
        off[i] = k < 0 || !ln.on ? -1 : k * TN + T * (ln.b + T * ln.c);
    }
    const uint32_t* list = args.p2g_lists + (size_t)(2 * args.combo) * args.p2g_list_cap;
    const uint32_t nwork = args.counters[kP2GListWord + 2 * args.combo];
    // the warps' item scheduler: [0] hands out list indices, [1] counts the
    // warps that have run out; the last of them clears both
    uint32_t* sched = args.sched + 2;
    const uint32_t warps = gridDim.x * (uint32_t)W::NW;
    // nothing for warps (the scheduler is untouched): p2gKernel takes the
    // small items when the list is too short to fill the GPU with warps
    if (nwork == 0 || !p2gWarpTakesSmall(args.p2g_warp, nwork)) return;
    RowWindow<S, MODE> win;
    spanBegin(args.spans, SPAN_P2G);
    for (;;) {
        uint32_t wi = 0;
        if (lane == 0) {
            wi = atomicAdd(&sched[0], 1u);
            if (wi >= nwork && atomicAdd(&sched[1], 1u) == warps - 1) {
                sched[0] = 0u;
                sched[1] = 0u;
            }
        }
        wi = __shfl_sync(0xffffffffu, wi, 0);
        if (wi >= nwork) break;
        const uint32_t w = list[wi];  // the item's slot: its tile
        const BlockItem it = args.active[w];
        if (args.scenes[it.scene].S != S) {  // never expected: lists are per combination
            if (lane == 0) atomicOr(args.err, ERR_INDEX);
            continue;
        }
        {
            const int4* src = reinterpret_cast<const int4*>(args.scenes + it.scene);
            int4* dst = reinterpret_cast<int4*>(&sc);
            for (int q = lane; q < (int)(sizeof(SceneDev) / 16); q += 32) dst[q] = src[q];
            for (int q = lane; q < W::kTileFloats; q += 32) tile[q] = 0.f;
        }
        __syncwarp();
        const float* pf = sc.buf[args.parity].f;
        const size_t cap = sc.cap;
        const float dt = sc.dt, h = sc.h, inv_h = sc.inv_h;
        const uint32_t i0 = it.start;
        const int count = (int)it.count;
        const uint32_t* keys = args.sorted_keys + i0;
        const uint32_t* perm = args.perm + i0;
        int t0[3];
        tileOrigin(sc, it.block, t0);
        win.clear();
        findRows(keys, count, rowBeg, lane, 32);
        __syncwarp();
        // the open row [rb, re) and its open segment [sb, se), the j-th of n
        int row = 0, rb = 0, re = 0, sb = 0, se = 0, j = 0, n = 0;
        // the loads of a pass are issued one pass ahead (the permutation
        // entries and keys two)
        P2GRaw<S, MODE> raw;
        uint32_t cl = 0, ncl = 0, nperm = 0;
        const bool stages = lane < W::kStage;
        if (stages && lane < count) {
            cl = keys[lane] & 63u;
            raw.load(args, sc, pf, cap, perm[lane], i0 + (uint32_t)lane);
        }
        if (stages && W::kStage + lane < count) {
            ncl = keys[W::kStage + lane] & 63u;
            nperm = perm[W::kStage + lane];
        }
        for (int g0 = 0; g0 < count; g0 += W::kStage) {
            const int np = min(W::kStage, count - g0);
            if (lane < np) p2gStageParticle<S, MODE>(sc, raw, dt, h, inv_h, t0, cl, st + lane * W::P4);
            const uint32_t pcl = cl;  // this pass's cells
            const int next_x = (int)(__shfl_sync(0xffffffffu, ncl, 0) & 3u);  // only read where the segment goes on
            if (stages && g0 + W::kStage + lane < count)
                raw.load(args, sc, pf, cap, nperm, i0 + (uint32_t)(g0 + W::kStage + lane));
            cl = ncl;
            if (stages && g0 + 2 * W::kStage + lane < count) {
                ncl = keys[g0 + 2 * W::kStage + lane] & 63u;
                nperm = perm[g0 + 2 * W::kStage + lane];
            }
            __syncwarp();  // the staged particles are visible to the warp
            for (int q = 0; q < np;) {
                if (g0 + q == se) {  // the next segment, as p2gKernel cuts them
                    if (se == re) {
                        row = (int)(__shfl_sync(0xffffffffu, pcl, q) >> 2);
                        rb = rowBeg[row];
                        re = rowBeg[row + 1];
                        n = (re - rb + W::kSeg - 1) / W::kSeg;
                        j = 0;
                    }
                    sb = se;
                    se = rb + (re - rb) * ++j / n;
                }
                const int qhi = min(se - g0, np);
                const bool ends = se <= g0 + np;
                const int base = T * ((row & 3) + T * (row >> 2));
                win.pass(st, pcl, q, qhi, row, g0 + q - sb, ends ? 4 : next_x, lane, ln,
                         [&](int n, const float* v) {
                             if (v)
#pragma unroll
                                 for (int i = 0; i < LN::kOut; ++i)
                                     if (off[i] >= 0) tile[off[i] + base + n] += v[i];
                         });
                if (ends) __syncwarp();  // the next segment's sums may land on the same nodes from other lanes
                q = qhi;
            }
            __syncwarp();  // the staged particles are read before the next pass overwrites them
        }
        float* out = args.tiles + (size_t)w * args.tile_stride;
        for (int q = lane; q < F * TN; q += 32) out[q] = tile[q];
        const int2 slot = args.block_slot[it.block];
        if (slot.y > 1) {
            __threadfence();
            __syncwarp();
            int last = 0;
            if (lane == 0) last = lastOfBlock(args, slot);
            if (__shfl_sync(0xffffffffu, last, 0)) mergeItemTiles<F * TN>(args, slot, lane, 32);
        }
        __syncwarp();  // the tile is read before the next item clears it
    }
    __syncthreads();  // every warp done: the CTA's span ends here
    spanEnd(args.spans, SPAN_P2G, false);
}

// ---------------------------------------------------------------------------
// Grid pass: merge the <= 8 overlapping tiles of every node in fixed order,
// then gravity, v = p/m, v* = v + dt f/m (m > FLT_EPSILON), boundary.
// Node-block N (4^3 nodes starting at 4N-4) is processed by the active block
// B = N - d with the smallest d in {0,1}^3 (x + 2y + 4z order).
// ---------------------------------------------------------------------------
// Barrier of the 64 threads (two warps) of group g of a 256-thread CTA:
// named barrier 1 + g (immediate ids, so the kernel reserves only those).
__device__ __forceinline__ void groupBarrier(int g) {
    switch (g) {
        case 0: asm volatile("bar.sync 1, 64;\n" ::: "memory"); break;
        case 1: asm volatile("bar.sync 2, 64;\n" ::: "memory"); break;
        case 2: asm volatile("bar.sync 3, 64;\n" ::: "memory"); break;
        default: asm volatile("bar.sync 4, 64;\n" ::: "memory"); break;
    }
}

__device__ __forceinline__ int blockSlotAt(const StepArgs& args, const SceneDev& sc, int x, int y, int z) {
    if (x < 0 || y < 0 || z < 0 || x >= sc.nb[0] || y >= sc.nb[1] || z >= sc.nb[2]) return -1;
    return args.block_slot[sc.block_base + (uint32_t)((z * sc.nb[1] + y) * sc.nb[0] + x)].x;
}

// CTAs per SM: 4 (64 registers) where that costs at most a few bytes of
// spills, else 3 (80 registers): the 8.4M-particle slab's grid pass took
// 0.15 ms at 4 against 0.26 at 3; quadratic APIC and PIC-FLIP spill 36-44
// bytes at 64 registers.
template <int S, int MODE>
struct GridBounds {
    static constexpr int MIN_CTAS = (MODE == MODE_FLIP || (MODE == MODE_APIC_FUSED && S != 4)) ? 3 : 4;
};

template <int S, int MODE>
__global__ void __launch_bounds__(kThreads, GridBounds<S, MODE>::MIN_CTAS) gridKernel(StepArgs args, int want_transfer) {
    constexpr int F = modeFields(MODE);
    constexpr int T = S + 3;
    constexpr int TN = tileNodes(S);
    // A block's merge is a chain of dependent loads.  With at least two work
    // items per CTA, each group of 64 threads merges its own blocks (four in
    // flight per CTA), group g taking items g, g + 4, ... of the CTA's share
    // and synchronising on its own named barrier; with fewer, the whole CTA
    // merges one block, four node blocks at a time.  Per group, the tile slots
    // of the 3^3 blocks around the current one, index (ox + 1) + 3 (oy + 1) +
    // 9 (oz + 1).
    constexpr int kGroups = kThreads / 64;
    __shared__ int nbSlotAll[kGroups][27];
    const uint32_t nact = args.counters[0];
    const bool grouped = nact >= 2u * gridDim.x;  // uniform over the CTA
    const int ngroups = grouped ? kGroups : 1;
    const int grp = grouped ? (int)(threadIdx.x >> 6) : 0;
    const int gt = grouped ? (int)(threadIdx.x & 63) : (int)threadIdx.x;  // thread within the group
    const int dstep = grouped ? 1 : kGroups;  // node blocks per round
    int* nbSlot = nbSlotAll[grp];
    spanBegin(args.spans, SPAN_GRID);
    for (uint32_t w = blockIdx.x * ngroups + grp; w < nact; w += gridDim.x * ngroups) {
        const BlockItem it = args.active[w];
        const SceneDev& sc = args.scenes[it.scene];
        if (sc.S != S || (want_transfer >= 0 && sc.transfer != want_transfer)) continue;
        if (MODE == MODE_MASS && !sc.init_pass) continue;
        if (args.block_slot[it.block].x != (int32_t)w) continue;  // a block's first work item does its nodes
        const uint32_t lb = it.block - sc.block_base;
        const int B[3] = {(int)(lb % (uint32_t)sc.nb[0]), (int)((lb / (uint32_t)sc.nb[0]) % (uint32_t)sc.nb[1]),
                          (int)(lb / ((uint32_t)sc.nb[0] * (uint32_t)sc.nb[1]))};
        if (gt < 27) {
            const int o[3] = {gt % 3 - 1, (gt / 3) % 3 - 1, gt / 9 - 1};
            nbSlot[gt] = blockSlotAt(args, sc, B[0] + o[0], B[1] + o[1], B[2] + o[2]);
        }
        if (grouped) groupBarrier(grp);
        else __syncthreads();
#pragma unroll 1
        for (int d0 = 0; d0 < 8; d0 += dstep) {  // the 8 node blocks this block may own
            const int d = d0 + (gt >> 6);
            const int dd[3] = {d & 1, (d >> 1) & 1, (d >> 2) & 1};
            const int N[3] = {B[0] + dd[0], B[1] + dd[1], B[2] + dd[2]};
            if (N[0] >= sc.nb[0] || N[1] >= sc.nb[1] || N[2] >= sc.nb[2]) continue;
            bool owner = true;
            for (int e = 0; e < d && owner; ++e)
                if (nbSlot[(dd[0] - (e & 1) + 1) + 3 * (dd[1] - ((e >> 1) & 1) + 1) + 9 * (dd[2] - ((e >> 2) & 1) + 1)] >= 0)
                    owner = false;
            if (!owner) continue;
            const int l = gt & 63;
            const int L[3] = {l & 3, (l >> 2) & 3, l >> 4};
            const int n[3] = {4 * N[0] - 4 + L[0], 4 * N[1] - 4 + L[1], 4 * N[2] - 4 + L[2]};
            if (n[0] < 0 || n[1] < 0 || n[2] < 0 || n[0] >= sc.res[0] || n[1] >= sc.res[1] || n[2] >= sc.res[2])
                continue;
            float acc[F];
#pragma unroll
            for (int f = 0; f < F; ++f) acc[f] = 0.f;
            // The 8 tiles that overlap the node, summed in order e; the loads of
            // Q of them are in flight at once.
            constexpr int Q = F <= 4 ? 8 : 4;
#pragma unroll
            for (int hq = 0; hq < 8 / Q; ++hq) {
                float v[Q][F];
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const int e = Q * hq + q;
                    const int de[3] = {e & 1, (e >> 1) & 1, (e >> 2) & 1};
                    const int ix = L[0] + 4 * de[0], iy = L[1] + 4 * de[1], iz = L[2] + 4 * de[2];
                    const int nbi = (dd[0] - de[0] + 1) + 3 * (dd[1] - de[1] + 1) + 9 * (dd[2] - de[2] + 1);
                    const int slot = (ix < T && iy < T && iz < T) ? nbSlot[nbi] : -1;
                    const float* tp = args.tiles + (size_t)(slot >= 0 ? slot : 0) * args.tile_stride + ix + T * (iy + T * iz);
#pragma unroll
                    for (int f = 0; f < F; ++f) v[q][f] = slot >= 0 ? tp[f * TN] : 0.f;
                }
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int f = 0; f < F; ++f) acc[f] += v[q][f];
            }
            const size_t node = (size_t)n[0] + (size_t)sc.res[0] * ((size_t)n[1] + (size_t)sc.res[1] * n[2]);
            const size_t nodes = (size_t)sc.res[0] * sc.res[1] * sc.res[2];
            if (MODE == MODE_SPLIT) {
                float* dbg = sc.dbg;
                dbg[node] += acc[0];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    dbg[(1 + a) * nodes + node] += acc[1 + a];
                    dbg[(4 + a) * nodes + node] += acc[4 + a];
                }
                continue;
            }
            if (MODE == MODE_MASS) {
                sc.vstar[node] = make_float4(0.f, 0.f, 0.f, acc[0]);
                continue;
            }
            const float m = acc[0], dt = sc.dt;
            if (m > 0.f) atomicAdd(&args.stats[2], 1u);
            float vs[3] = {0.f, 0.f, 0.f}, vo[3] = {0.f, 0.f, 0.f};
            if (MODE == MODE_APIC_FUSED) {
                if (m > kFltEps) {
#pragma unroll
                    for (int a = 0; a < 3; ++a) vs[a] = __fdiv_rn(acc[1 + a], m);
                    vs[1] -= dt * sc.gravity;
                }
            } else {  // MODE_FLIP
                if (m > kFltEps) {
                    float fy = acc[5] - sc.gravity * m;
                    const float fo[3] = {acc[4], fy, acc[6]};
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        vo[a] = __fdiv_rn(acc[1 + a], m);
                        vs[a] = vo[a] + __fdiv_rn(dt * fo[a], m);
                    }
                } else {
#pragma unroll
                    for (int a = 0; a < 3; ++a) vo[a] = acc[1 + a];
                }
            }
            if (sc.boundary == MPM_BOUNDARY_STICKY) {
                bool wall = false;
#pragma unroll
                for (int a = 0; a < 3; ++a) wall |= (n[a] < sc.sticky) || (n[a] >= sc.res[a] - sc.sticky);
                if (wall) vs[0] = vs[1] = vs[2] = 0.f;
            } else {
                float pos[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) pos[a] = (sc.origin[a] + sc.h * (float)n[a]) + dt * vs[a];
                boundaryCollision(pos, vs, sc.origin, sc.target, sc.friction);
            }
            if (sc.phi) {
                float pos[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) pos[a] = (sc.origin[a] + sc.h * (float)n[a]) + dt * vs[a];
                levelSetCollision(sc, pos, vs);
            }
            sc.vstar[node] = make_float4(vs[0], vs[1], vs[2], m);
            if (MODE == MODE_FLIP) sc.vold[node] = make_float4(vo[0], vo[1], vo[2], 0.f);
        }
        if (grouped) groupBarrier(grp);  // the neighbour table is rewritten for the next item
        else __syncthreads();
    }
    __syncthreads();  // every group done: the CTA's span ends here
    spanEnd(args.spans, SPAN_GRID);
}

// ---------------------------------------------------------------------------
// G2P, fused with the particle update.  An item of a block's particles at a time:
// the block's (S+3)^3 node tile of v* (and v) is staged in shared memory, then one
// thread per particle.  Writes the particle to its sorted slot of the other buffer.
// ---------------------------------------------------------------------------
// The loads of a particle's update, issued one particle ahead into the thread's
// shared-memory row by cp.async (one commit group per particle, possibly
// empty), so that their latency overlaps the previous particle's update; its
// permutation entry and key, which they wait for, two ahead.  (Holding x and v
// in registers instead, and reading mass and pid where they are stored, left
// the loads of a permutation entry, of mass and of pid exposed in every
// update.)
struct G2PIn {
    uint32_t old, cell;
    bool ok;
};
template <bool APIC>
__device__ __forceinline__ G2PIn g2pFetch(const StepArgs& args, const SceneDev& sc, uint32_t gs, uint32_t perm,
                                          uint32_t key, float* pre) {
    G2PIn p;
    const size_t cap = sc.cap;
    const uint32_t old = perm - sc.key_offset;
    const uint32_t dst = gs - sc.key_offset;
    p.ok = old < sc.n && dst < sc.n;  // range check: never expected, skip instead of faulting
    p.old = p.ok ? old : 0u;
    p.cell = key & 63u;
    if (p.ok) {
        const float* pf = sc.buf[args.parity].f + old;
#pragma unroll
        for (int a = 0; a < 3; ++a) cpAsync4(pre + kPreX + a, pf + (F_X + a) * cap);
        if (!APIC)
#pragma unroll
            for (int a = 0; a < 3; ++a) cpAsync4(pre + kPreV + a, pf + (F_V + a) * cap);
#pragma unroll
        for (int k = 0; k < 18; ++k) cpAsync4(pre + k, pf + (F_FE + k) * cap);  // Fe, Fp
        cpAsync4(pre + kPreVol, pf + F_VOL * cap);
        cpAsync4(pre + kPreMass, pf + F_MASS * cap);
        cpAsync4(pre + kPrePid, reinterpret_cast<const float*>(sc.buf[args.parity].pid + old));
    } else {
        atomicOr(args.err, ERR_INDEX);
    }
    cpAsyncCommit();
    return p;
}
__device__ __forceinline__ void cpAsyncWaitPrevious() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

template <int S, bool APIC>
__device__ __forceinline__ void particleUpdate(const StepArgs& args, const SceneDev& sc, uint32_t gs, const G2PIn& in,
                                               bool next_pending, const float4* tvs, const float4* tvo, const int* t0,
                                               bool fused, float* pre, const MaterialDev& mat0) {
    constexpr int T = S + 3;
    float* nf = sc.buf[args.parity ^ 1].f;
    const size_t cap = sc.cap;
    if (next_pending) cpAsyncWaitPrevious();  // this particle's group; the next one's may still run
    else cpAsyncWaitAll();
    if (!in.ok) return;
    const uint32_t old = in.old;
    const uint32_t dst = gs - sc.key_offset;
    const float h = sc.h, dt = sc.dt;
    float vpic[3] = {0.f, 0.f, 0.f}, dflip[3] = {0.f, 0.f, 0.f};
    float gv[9], K[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) gv[k] = K[k] = 0.f;
    if (tvs) {
        // the stencil base comes from the cell, which the key was formed from
        const int lo[3] = {(int)(in.cell & 3u), (int)((in.cell >> 2) & 3u), (int)(in.cell >> 4)};
        float w[3][S], dw[3][S];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            float gp0 = __fadd_rn(sc.origin[a], __fmul_rn(h, (float)(t0[a] + lo[a])));
            float dk[S];
            dk[0] = quotient(pre[kPreX + a] - gp0, h, sc.inv_h);
#pragma unroll
            for (int k = 1; k < S; ++k) dk[k] = dk[0] - (float)k;  // exact subtraction
            splineWeights<S>(dk, w[a], dw[a]);
#pragma unroll
            for (int k = 0; k < S; ++k) {
                dw[a][k] *= sc.inv_h;
            }
        }
        // Separable gather, one axis after another: along x for every row (b,
        // c) of the stencil, along y for every plane c, then along z.  In
        // packed FP32 pairs: the x and y components of every sum go through
        // one __ffma2_rn (two exactly rounded FMAs, the same results as
        // fmaf), z through fmaf.  Sums of v* with the weights N_x N_y N_z (the
        // velocity), N'_x N_y N_z and so on (the columns of grad v), a N_x N_y
        // N_z and so on (those of the APIC moment K); PIC-FLIP's of v* - v.
        // Instruction issue and load latency bound the kernel: summing the rows
        // straight into the results took seven scaled additions a row (with
        // the loads of g2pFetch and the base from the cell: two-ball
        // G2P 0.118 -> 0.106 ms and 62M -> 56M warp instructions, slab 1.14 ->
        // 0.98 ms).
        struct V3 {
            float2 xy;
            float z;
        };
        auto fma3 = [](float k, const V3& v, V3& sum) {
            sum.xy = __ffma2_rn(make_float2(k, k), v.xy, sum.xy);
            sum.z = fmaf(k, v.z, sum.z);
        };
        const V3 zero{make_float2(0.f, 0.f), 0.f};
        V3 sv = zero, sg[3] = {zero, zero, zero}, sk[3] = {zero, zero, zero}, sf = zero;
#pragma unroll
        for (int c = 0; c < S; ++c) {
            // plane sums: y weight N_y of the rows' N_x, N'_x and a N_x (or
            // v* - v) sums, and N'_y and b N_y of the first
            V3 p0 = zero, pd = zero, p1 = zero, py = zero, pb = zero;
#pragma unroll
            for (int b = 0; b < S; ++b) {
                V3 r0 = zero, rd = zero, r1 = zero;
                const int rowbase = lo[0] + T * ((lo[1] + b) + T * (lo[2] + c));
#pragma unroll
                for (int a = 0; a < S; ++a) {
                    const float4 g = tvs[rowbase + a];
                    const V3 gv3{make_float2(g.x, g.y), g.z};
                    fma3(w[0][a], gv3, r0);
                    fma3(dw[0][a], gv3, rd);
                    if (APIC) {
                        if (a) fma3(w[0][a] * (float)a, gv3, r1);
                    } else {
                        const float4 o = tvo[rowbase + a];
                        const V3 d{__fadd2_rn(gv3.xy, make_float2(-o.x, -o.y)), g.z - o.z};  // g - o, exactly
                        fma3(w[0][a], d, r1);
                    }
                }
                fma3(w[1][b], r0, p0);
                fma3(w[1][b], rd, pd);
                fma3(w[1][b], r1, p1);
                fma3(dw[1][b], r0, py);
                if (APIC && b) fma3(w[1][b] * (float)b, r0, pb);
            }
            fma3(w[2][c], p0, sv);
            fma3(w[2][c], pd, sg[0]);
            fma3(w[2][c], py, sg[1]);
            fma3(dw[2][c], p0, sg[2]);
            if (APIC) {
                fma3(w[2][c], p1, sk[0]);
                fma3(w[2][c], pb, sk[1]);
                if (c) fma3(w[2][c] * (float)c, p0, sk[2]);
            } else {
                fma3(w[2][c], p1, sf);
            }
        }
        vpic[0] = sv.xy.x;
        vpic[1] = sv.xy.y;
        vpic[2] = sv.z;
        dflip[0] = sf.xy.x;
        dflip[1] = sf.xy.y;
        dflip[2] = sf.z;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            gv[0 * 3 + j] = sg[j].xy.x;
            gv[1 * 3 + j] = sg[j].xy.y;
            gv[2 * 3 + j] = sg[j].z;
            K[0 * 3 + j] = sk[j].xy.x;
            K[1 * 3 + j] = sk[j].xy.y;
            K[2 * 3 + j] = sk[j].z;
        }
    }
    // New velocity (src/mpm_solver3d.cu:362-363; apic :366-374).
    float vn[3];
    if (APIC) {
#pragma unroll
        for (int i = 0; i < 3; ++i) vn[i] = vpic[i];
    } else {
        const float al = sc.blend, om = 1.0f - sc.blend;
#pragma unroll
        for (int i = 0; i < 3; ++i) vn[i] = al * (pre[kPreV + i] + dflip[i]) + om * vpic[i];
    }
    // Fe <- (I + dt grad v) Fe ; F = Fe Fp ; SVD clamp (src/material_point3d.cu:53-70).
    float Fe[9], Fp[9], A[9], Fn[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        Fe[k] = pre[k];
        Fp[k] = pre[9 + k];
        A[k] = dt * gv[k] + ((k % 4 == 0) ? 1.0f : 0.0f);
    }
    matmul3(A, Fe, Fn);
    const uint16_t mid = sc.nmat > 1 ? sc.buf[args.parity].mat[old] : (uint16_t)0;
    const MaterialDev m = sc.nmat > 1 ? sc.mats[mid] : mat0;
    const float hi = 1.0f + m.theta_s, lo = 1.0f - m.theta_c;
    const float V0 = pre[kPreVol];
    float mu, la, tau[6];
    // Elastic fast path: no singular value can be clamped, so Fe = Fn and Fp
    // stay as they are, and the stress comes from the polar rotation of Fn
    // (no SVD).  Material bounds beyond 25 % always take the SVD path.
    const float theta = fmaxf(m.theta_s, m.theta_c);
    if (theta <= 0.25f && singularValuesInside(Fn, lo, hi)) {
#pragma unroll
        for (int k = 0; k < 9; ++k) Fe[k] = Fn[k];
        plasticLame(m, Fp, mu, la);
        const float J = det3(Fn);
        float P[9];  // 2 mu (F - R) for fixed corotated, mu F for Neo-Hookean
        float diag;
        if (m.model == MPM_MODEL_NEO_HOOKEAN) {
#pragma unroll
            for (int k = 0; k < 9; ++k) P[k] = mu * Fn[k];
            diag = la * logf(J) - mu;
        } else {
            float R[9];
            polarRotation(Fn, R, theta <= 0.1f ? 3 : 4);
#pragma unroll
            for (int k = 0; k < 9; ++k) P[k] = 2.0f * mu * (Fn[k] - R[k]);
            diag = la * (J - 1.0f) * J;
        }
        const int I[6] = {0, 1, 2, 0, 0, 1}, Jx[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
        for (int e = 0; e < 6; ++e) {
            const int i = I[e], j = Jx[e];
            float v = fmaf(P[3 * i + 2], Fn[3 * j + 2], fmaf(P[3 * i + 1], Fn[3 * j + 1], P[3 * i] * Fn[3 * j]));
            if (e < 3) v += diag;
            tau[e] = V0 * v;
        }
    } else {
    float U[9], V[9], s[3];
    svd3(Fn, U, s, V);
    bool clamped = false;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float c = fmaxf(fminf(s[k], hi), lo);
        clamped |= c != s[k];
        s[k] = c;
    }
    if (clamped) {
        // Fe = U S V^T ; Fp = V S^-1 U^T (Fe Fp)
        float Ff[9];
        matmul3(Fn, Fp, Ff);
        float US[9], VSi[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                US[3 * i + k] = U[3 * i + k] * s[k];
                VSi[3 * i + k] = V[3 * i + k] / s[k];
            }
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                Fe[3 * i + j] = US[3 * i] * V[3 * j] + US[3 * i + 1] * V[3 * j + 1] + US[3 * i + 2] * V[3 * j + 2];
                A[3 * i + j] = VSi[3 * i] * U[3 * j] + VSi[3 * i + 1] * U[3 * j + 1] + VSi[3 * i + 2] * U[3 * j + 2];
            }
        matmul3(A, Ff, Fp);
    } else {
        // No singular value clamped: U S V^T = Fn and V S^-1 U^T Fn Fp = Fp in
        // exact arithmetic; keeping Fn and Fp avoids the FP32 SVD round-off.
#pragma unroll
        for (int k = 0; k < 9; ++k) Fe[k] = Fn[k];
    }
    // Next step's stress from the clamped SVD (Fe = U S V^T exactly).
    plasticLame(m, Fp, mu, la);
    if (m.model == MPM_MODEL_NEO_HOOKEAN) {
        bool proj = false;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            proj |= s[k] < kFltEps;
            s[k] = fmaxf(s[k], kFltEps);
        }
        if (proj)
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    Fe[3 * i + j] = U[3 * i] * s[0] * V[3 * j] + U[3 * i + 1] * s[1] * V[3 * j + 1] +
                                    U[3 * i + 2] * s[2] * V[3 * j + 2];
    }
    tauFromSvd(m.model, U, s, mu, la, V0, tau);
    }
    // the position, read again (held in registers across the update it would
    // spill others)
    float x[3], delta[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        x[a] = *(volatile const float*)(pre + kPreX + a);
        const int lo = (int)((in.cell >> (2 * a)) & 3u);
        delta[a] = tvs ? x[a] - __fadd_rn(sc.origin[a], __fmul_rn(h, (float)(t0[a] + lo))) : 0.f;
    }
    if (fused) {
        if (sc.pcoll) {  // particlesCollision (src/mpm_solver3d.cu:428-445)
            float pos[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) pos[a] = x[a] + dt * vn[a];
            boundaryCollision(pos, vn, sc.origin, sc.target, sc.friction);
            if (sc.phi) {
#pragma unroll
                for (int a = 0; a < 3; ++a) pos[a] = x[a] + dt * vn[a];
                levelSetCollision(sc, pos, vn);
            }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) x[a] += dt * vn[a];  // advectParticles (:381-391)
        const uint32_t key = particleKey(sc, x, args.err);
        args.next_keys[gs] = key;
        // one atomic per distinct block among the converged lanes (sorted
        // particles: a warp's lanes nearly always share their next block)
        const uint32_t blk = key >> 6;
        const uint32_t peers = __match_any_sync(__activemask(), blk);
        if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&args.block_count[blk], (uint32_t)__popc(peers));
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        nf[(F_X + a) * cap + dst] = x[a];
        nf[(F_V + a) * cap + dst] = vn[a];
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        nf[(F_FE + k) * cap + dst] = Fe[k];
        nf[(F_FP + k) * cap + dst] = Fp[k];
    }
    if (APIC) {
        // B = sum w v* (x_i - x_p)^T = h K - vpic delta^T
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) nf[(F_B + 3 * i + j) * cap + dst] = h * K[3 * i + j] - vpic[i] * delta[j];
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) nf[(F_TAU + k) * cap + dst] = tau[k];
    nf[F_MASS * cap + dst] = pre[kPreMass];
    nf[F_VOL * cap + dst] = V0;
    sc.buf[args.parity ^ 1].pid[dst] = __float_as_uint(pre[kPrePid]);
    if (sc.nmat > 1) sc.buf[args.parity ^ 1].mat[dst] = mid;
}

// ---------------------------------------------------------------------------
// TMA (cp.async.bulk.tensor) and mbarrier helpers for G2P's grid tile.  The
// tensor map of a scene's dense float4 grid is 4-D FP32: (component, x, y, z),
// so the innermost box extent is one node's 16 bytes and every tile origin is
// aligned whatever its x; nodes outside the grid read as zeros (OOB fill).
// The maps cover this GPU's own grid memory; there is no multicast.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smemAddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbarInit(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smemAddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbarInitFence() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
__device__ __forceinline__ void mbarExpectTx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smemAddr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbarTryWait(uint64_t* bar, unsigned parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smemAddr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Orders this CTA's earlier generic-proxy accesses of shared memory before
// later async-proxy (TMA) writes to it.
__device__ __forceinline__ void fenceProxyAsyncShared() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void tensorMapAcquire(const void* map) {
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" ::"l"(map) : "memory");
}
// Box of the 4-D map at (0, x, y, z) into dst, completing on bar.
__device__ __forceinline__ void tmaLoadTile(void* dst, const void* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];\n" ::"r"(smemAddr(dst)),
        "l"(map), "r"(0), "r"(x), "r"(y), "r"(z), "r"(smemAddr(bar))
        : "memory");
}

// Bounded wait on an mbarrier phase: gives up after ~2^22 polls (seconds),
// raising ERR_WAIT_TIMEOUT and setting *abort (when given) so that the CTA's
// other waiters give up too (they look at it every 256 polls).  Returns false
// when it gave up.
__device__ __forceinline__ bool waitTile(uint64_t* bar, unsigned parity, uint32_t* err, volatile int* abort) {
    for (uint32_t i = 0; !mbarTryWait(bar, parity); ++i) {
        if (i > (1u << 22)) {
            atomicOr(err, ERR_WAIT_TIMEOUT);
            if (abort) *abort = 1;
            return false;
        }
        if (abort && (i & 255u) == 255u && *abort) return false;
        if (i > 64) __nanosleep(64);
    }
    return true;
}

// Bulk copy (cp.async.bulk) of bytes from global to shared memory, completing
// on bar; both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulkLoad(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smemAddr(dst)),
                 "l"(src), "r"(bytes), "r"(smemAddr(bar))
                 : "memory");
}
__device__ __forceinline__ void mbarArrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smemAddr(bar)) : "memory");
}

// G2P: persistent CTAs take work items from this combination's list (then the
// outside items).  One elected thread produces: it fetches the next item and
// copies, by TMA, the item's tile of v* (and v), its scene entry and the
// scene's first material into one of two shared-memory slots, completing on
// the slot's "full" mbarrier.  Every warp consumes: it waits on "full",
// updates its particles of the item and arrives on the slot's "empty"
// mbarrier; the producer refills a slot only when all warps have released it.
// So warps run up to one item apart instead of meeting at a CTA barrier after
// every item, and the particle update reads the scene and material from
// shared memory.
// Resident G2P CTAs per SM the register budget is fitted to: 2 gives 128
// registers a thread and no spills but for cubic PIC-FLIP's 16 bytes (two-ball
// G2P 0.132 -> 0.117 ms against 3 CTAs at 80 registers, which spill ~150 bytes a
// thread).
#ifndef MPM_G2P_THREADS
#define MPM_G2P_THREADS 256
#endif
constexpr int kG2PThreads = MPM_G2P_THREADS;
constexpr int kG2PWarps = kG2PThreads / 32;
#ifndef MPM_G2P_MIN_CTAS
#define MPM_G2P_MIN_CTAS (2 * 256 / MPM_G2P_THREADS)
#endif
template <int S, bool APIC>
__global__ void __launch_bounds__(kG2PThreads, MPM_G2P_MIN_CTAS) g2pKernel(StepArgs args, int fused) {
    constexpr int TN = tileNodes(S);
    constexpr int TNP = (TN + 7) & ~7;  // buffers 128-byte aligned
    constexpr unsigned kTileBytes = (unsigned)TN * 16u;
    static_assert(sizeof(SceneDev) % 16 == 0 && sizeof(MaterialDev) % 16 == 0, "bulk copies need 16-byte sizes");
    __shared__ __align__(128) float4 tvs[2][TNP];
    __shared__ __align__(128) float4 tvo[APIC ? 1 : 2][APIC ? 8 : TNP];
    // two per-thread prefetch rows of Fe, Fp, V0 (dynamic shared memory: with
    // the tiles they exceed the 48 KB of static shared memory)
    extern __shared__ float4 g2p_dyn[];
    float (*pre)[kG2PThreads * kPreStride] = reinterpret_cast<float (*)[kG2PThreads * kPreStride]>(g2p_dyn);
    __shared__ SceneDev scs[2];
    __shared__ MaterialDev mat0[2];
    __shared__ BlockItem its[2];
    __shared__ uint32_t item_s[2];
    __shared__ __align__(8) uint64_t full[2], empty[2];
    const int want = APIC ? MPM_TRANSFER_APIC : MPM_TRANSFER_PIC_FLIP;
    // this combination's own (finer) items of the active blocks, then the
    // outside items of all scenes (the others' are skipped)
    const uint32_t nact = args.counters[kG2PCountWord + args.combo];
    const BlockItem* items = args.g2p_items + (size_t)args.combo * args.g2p_cap;
    const uint32_t nout = args.counters[1];
    const uint32_t total = nact + nout;
    uint32_t* sched = args.sched + 4;
    const int lane = threadIdx.x & 31;

    // Producer (thread 0): the next item (the last CTA to run out clears the
    // scheduler, so every launch starts from zero) into slot b -- its scene
    // entry, the scene's first material and, for an active block, the tile
    // of v* (and v) -- completing on full[b].  After the first index past the
    // end it only hands out the end marker.
    bool ran_out = false;
    auto produce = [&](int b) {
        uint32_t w = total;
        if (!ran_out) {
            w = atomicAdd(&sched[0], 1u);
            if (w >= total) {
                ran_out = true;
                if (atomicAdd(&sched[1], 1u) == gridDim.x - 1) {
                    sched[0] = 0u;
                    sched[1] = 0u;
                }
            }
        }
        item_s[b] = w;
        if (w >= total) {
            mbarArrive(&full[b]);
            return;
        }
        const BlockItem it = w < nact ? items[w] : args.outside[w - nact];
        its[b] = it;
        const SceneDev* sg = args.scenes + it.scene;
        const bool tile = w < nact;
        fenceProxyAsyncShared();  // the slot's earlier generic reads come first
        mbarExpectTx(&full[b], (unsigned)(sizeof(SceneDev) + sizeof(MaterialDev)) +
                                   (tile ? (APIC ? kTileBytes : 2u * kTileBytes) : 0u));
        bulkLoad(&scs[b], sg, (unsigned)sizeof(SceneDev), &full[b]);
        bulkLoad(&mat0[b], sg->mats, (unsigned)sizeof(MaterialDev), &full[b]);
        if (tile) {
            int t0[3];
            tileOrigin(*sg, it.block, t0);
            const unsigned char* maps = args.tmaps + (size_t)it.scene * 2 * kTensorMapBytes;
            tensorMapAcquire(maps);
            tmaLoadTile(&tvs[b][0], maps, t0[0], t0[1], t0[2], &full[b]);
            if (!APIC) {
                tensorMapAcquire(maps + kTensorMapBytes);
                tmaLoadTile(&tvo[b][0], maps + kTensorMapBytes, t0[0], t0[1], t0[2], &full[b]);
            }
        }
    };
    // A wait that gives up (never expected) sets abort_s: the producer stops
    // issuing copies, every warp leaves the loop at its next slot wait (as a
    // whole warp), and thread 0 waits for the copies still in flight before
    // the CTA exits, so that none lands in shared memory it no longer owns.
    __shared__ int abort_s;
    spanBegin(args.spans, SPAN_G2P);
    if (threadIdx.x == 0) {
        abort_s = 0;
        mbarInit(&full[0], 1);
        mbarInit(&full[1], 1);
        mbarInit(&empty[0], kG2PWarps);
        mbarInit(&empty[1], kG2PWarps);
        mbarInitFence();
        produce(0);
    }
    __syncthreads();
    unsigned full_ph = 0u, empty_ph = 0u;  // bit b: parity of slot b's next wait
    unsigned issued = 1u;                  // thread 0: slots whose copies it has not yet seen land
    for (int k = 0, b = 0;; ++k, b ^= 1) {
        if (threadIdx.x == 0 && !abort_s) {
            // slot b ^ 1 gets item k + 1; it held item k - 1
            bool free_slot = true;
            if (k >= 1) {
                free_slot = waitTile(&empty[b ^ 1], (empty_ph >> (b ^ 1)) & 1u, args.err, &abort_s);
                if (free_slot) empty_ph ^= 1u << (b ^ 1);
            }
            if (free_slot) {
                produce(b ^ 1);
                issued |= 1u << (b ^ 1);
            }
        }
        const bool landed = waitTile(&full[b], (full_ph >> b) & 1u, args.err, &abort_s);
        if (__any_sync(0xffffffffu, !landed)) break;  // gave up (never expected): the whole warp leaves
        if (threadIdx.x == 0) issued &= ~(1u << b);
        full_ph ^= 1u << b;
        const uint32_t w = item_s[b];
        if (w >= total) break;
        const bool inside = w < nact;
        const BlockItem it = its[b];
        const SceneDev& sc = scs[b];
        int t0[3] = {0, 0, 0};
        if (inside) tileOrigin(sc, it.block, t0);
        if ((inside || (sc.S == S && sc.transfer == want)) && threadIdx.x < it.count) {
            // each thread's particles of the item, the next one's loads in
            // flight during the current one's update (rows alternate)
            int row = 0;
            const uint32_t* perm = args.perm + it.start;
            const uint32_t* keys = args.sorted_keys + it.start;
            uint32_t i = threadIdx.x;
            uint32_t np = 0, nk = 0;  // permutation entry and key of the particle to fetch next
            if (i + kG2PThreads < it.count) {
                np = perm[i + kG2PThreads];
                nk = keys[i + kG2PThreads];
            }
            G2PIn cur = g2pFetch<APIC>(args, sc, it.start + i, perm[i], keys[i], &pre[0][threadIdx.x * kPreStride]);
            for (; i < it.count; i += kG2PThreads) {
                const bool more = i + kG2PThreads < it.count;
                G2PIn nxt;
                if (more) {
                    nxt = g2pFetch<APIC>(args, sc, it.start + i + kG2PThreads, np, nk,
                                         &pre[row ^ 1][threadIdx.x * kPreStride]);
                    if (i + 2 * kG2PThreads < it.count) {
                        np = perm[i + 2 * kG2PThreads];
                        nk = keys[i + 2 * kG2PThreads];
                    }
                }
                particleUpdate<S, APIC>(args, sc, it.start + i, cur, more, inside ? &tvs[b][0] : nullptr,
                                        APIC ? nullptr : &tvo[b][0], t0, fused != 0,
                                        &pre[row][threadIdx.x * kPreStride], mat0[b]);
                if (more) cur = nxt;
                row ^= 1;
            }
        }
        __syncwarp();
        if (lane == 0) mbarArrive(&empty[b]);
    }
    if (threadIdx.x == 0 && abort_s) {
        // copies issued and not seen landing: wait for them, bounded again
        for (int s = 0; s < 2; ++s)
            if ((issued >> s) & 1u) waitTile(&full[s], (full_ph >> s) & 1u, args.err, nullptr);
    }
    __syncthreads();  // every warp done: the CTA's span ends here
    spanEnd(args.spans, SPAN_G2P);
}

// ---------------------------------------------------------------------------
// Split-mode dense grid kernels on sc.dbg planes: mass, vel[3], force[3], vstar[3].
// ---------------------------------------------------------------------------
__global__ void denseGravityKernel(const SceneDev* __restrict__ scenes) {
    const SceneDev& sc = scenes[blockIdx.y];
    const size_t nodes = (size_t)sc.res[0] * sc.res[1] * sc.res[2];
    for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < nodes; i += (size_t)gridDim.x * kThreads) {
        float m = sc.dbg[i];
        if (m > kFltEps) sc.dbg[5 * nodes + i] -= sc.gravity * m;  // force.y
    }
}

__global__ void denseUpdateVelocityKernel(const SceneDev* __restrict__ scenes, float dt) {
    const SceneDev& sc = scenes[blockIdx.y];
    const size_t nodes = (size_t)sc.res[0] * sc.res[1] * sc.res[2];
    for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < nodes; i += (size_t)gridDim.x * kThreads) {
        float m = sc.dbg[i];
        if (m > kFltEps) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                float v = __fdiv_rn(sc.dbg[(1 + a) * nodes + i], m);
                sc.dbg[(1 + a) * nodes + i] = v;
                sc.dbg[(7 + a) * nodes + i] = v + __fdiv_rn(dt * sc.dbg[(4 + a) * nodes + i], m);
            }
        }
    }
}

__global__ void denseCollisionKernel(const SceneDev* __restrict__ scenes, float dt) {
    const SceneDev& sc = scenes[blockIdx.y];
    const size_t nodes = (size_t)sc.res[0] * sc.res[1] * sc.res[2];
    for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < nodes; i += (size_t)gridDim.x * kThreads) {
        const int n[3] = {(int)(i % sc.res[0]), (int)((i / sc.res[0]) % sc.res[1]),
                          (int)(i / ((size_t)sc.res[0] * sc.res[1]))};
        float vs[3] = {sc.dbg[7 * nodes + i], sc.dbg[8 * nodes + i], sc.dbg[9 * nodes + i]};
        if (sc.boundary == MPM_BOUNDARY_STICKY) {
            bool wall = false;
#pragma unroll
            for (int a = 0; a < 3; ++a) wall |= (n[a] < sc.sticky) || (n[a] >= sc.res[a] - sc.sticky);
            if (wall) vs[0] = vs[1] = vs[2] = 0.f;
        } else {
            float pos[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) pos[a] = (sc.origin[a] + sc.h * (float)n[a]) + dt * vs[a];
            boundaryCollision(pos, vs, sc.origin, sc.target, sc.friction);
        }
        if (sc.phi) {
            float pos[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) pos[a] = (sc.origin[a] + sc.h * (float)n[a]) + dt * vs[a];
            levelSetCollision(sc, pos, vs);
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) sc.dbg[(7 + a) * nodes + i] = vs[a];
    }
}

// dbg planes -> float4 v*, v for the G2P kernel.
__global__ void densePackKernel(const SceneDev* __restrict__ scenes) {
    const SceneDev& sc = scenes[blockIdx.y];
    const size_t nodes = (size_t)sc.res[0] * sc.res[1] * sc.res[2];
    for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < nodes; i += (size_t)gridDim.x * kThreads) {
        sc.vstar[i] = make_float4(sc.dbg[7 * nodes + i], sc.dbg[8 * nodes + i], sc.dbg[9 * nodes + i], sc.dbg[i]);
        if (sc.vold)
            sc.vold[i] = make_float4(sc.dbg[nodes + i], sc.dbg[2 * nodes + i], sc.dbg[3 * nodes + i], 0.f);
    }
}

__global__ void particlesCollisionKernel(const SceneDev* __restrict__ scenes, int parity, float dt) {
    const SceneDev& sc = scenes[blockIdx.y];
    float* f = sc.buf[parity].f;
    const size_t cap = sc.cap;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < sc.n; i += gridDim.x * kThreads) {
        float x[3], v[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            v[a] = f[(F_V + a) * cap + i];
            x[a] = f[(F_X + a) * cap + i] + dt * v[a];
        }
        boundaryCollision(x, v, sc.origin, sc.target, sc.friction);
        if (sc.phi) {
#pragma unroll
            for (int a = 0; a < 3; ++a) x[a] = f[(F_X + a) * cap + i] + dt * v[a];
            levelSetCollision(sc, x, v);
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) f[(F_V + a) * cap + i] = v[a];
    }
}

__global__ void advectKernel(const SceneDev* __restrict__ scenes, int parity, float dt) {
    const SceneDev& sc = scenes[blockIdx.y];
    float* f = sc.buf[parity].f;
    const size_t cap = sc.cap;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < sc.n; i += gridDim.x * kThreads)
#pragma unroll
        for (int a = 0; a < 3; ++a) f[(F_X + a) * cap + i] += dt * f[(F_V + a) * cap + i];
}

// Particle state of a new scene from the caller's arrays staged on the device
// as [x: 3n interleaved][v: 3n interleaved][m: n][V0: n, prescribed only]:
// SoA planes with Fe = Fp = I, B = tau = 0 and V0 = 0 unless prescribed
// (the reference's MaterialPoint3D constructor, src/material_point3d.cu:10-30).
// With `perm` slot i takes the caller's particle perm[i] (the cell-sorted
// order), else particle i; pid records it.  mat_in: the caller's material ids
// (staged), else none.
__global__ void initStateKernel(float* __restrict__ f, uint32_t* __restrict__ pid, uint16_t* __restrict__ mat,
                                size_t cap, const float* __restrict__ staged, size_t n, int has_volume,
                                const uint32_t* __restrict__ perm, const uint16_t* __restrict__ mat_in) {
    for (size_t i = blockIdx.x * (size_t)kThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kThreads) {
        const size_t o = perm ? (size_t)perm[i] : i;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            f[(F_X + a) * cap + i] = staged[3 * o + a];
            f[(F_V + a) * cap + i] = staged[3 * n + 3 * o + a];
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            f[(F_FE + k) * cap + i] = (k % 4 == 0) ? 1.f : 0.f;
            f[(F_FP + k) * cap + i] = (k % 4 == 0) ? 1.f : 0.f;
            f[(F_B + k) * cap + i] = 0.f;
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) f[(F_TAU + k) * cap + i] = 0.f;
        f[F_MASS * cap + i] = staged[6 * n + o];
        f[F_VOL * cap + i] = has_volume ? staged[7 * n + o] : 0.f;
        pid[i] = (uint32_t)o;
        if (mat_in) mat[i] = mat_in[o];
    }
}

// Cell keys of a new scene's staged positions (caller order, x y z
// interleaved), for the cell-sorted initial order.
__global__ void __launch_bounds__(kThreads) stagedKeyKernel(const SceneDev sc, const float* __restrict__ xyz,
                                                             uint32_t n, uint32_t* __restrict__ keys,
                                                             uint32_t* __restrict__ err) {
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
        const float x[3] = {xyz[3 * (size_t)i], xyz[3 * (size_t)i + 1], xyz[3 * (size_t)i + 2]};
        keys[i] = particleKey(sc, x, err);
    }
}

// initialize(): V0 = m / (sum_i m_i w_ip / h^3) with node masses in vstar.w
// (src/mpm_solver3d.cu:173-214).  Live order, dense node reads.
template <int S>
__global__ void volumeKernel(const SceneDev* __restrict__ scenes, int parity) {
    const SceneDev& sc = scenes[blockIdx.y];
    float* f = sc.buf[parity].f;
    const size_t cap = sc.cap;
    const float h = sc.h;
    const float inv_cell_vol = (float)(1.0 / (double)(h * h * h));
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < sc.n; i += gridDim.x * kThreads) {
        float x[3] = {f[F_X * cap + i], f[(F_X + 1) * cap + i], f[(F_X + 2) * cap + i]};
        int base[3];
        float dens = 0.f;
        if (stencilBase(sc, x, base)) {
            float w[3][S];
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int k = 0; k < S; ++k) {
                    float gp = __fadd_rn(sc.origin[a], __fmul_rn(h, (float)(base[a] + k)));
                    w[a][k] = splineN<S>(__fdiv_rn(__fsub_rn(x[a], gp), h));
                }
            // nodes in the grid per axis (all of them but at the edges); the
            // sum runs over the stencil in the same order either way
            bool in[3][S];
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int k = 0; k < S; ++k) in[a][k] = base[a] + k >= 0 && base[a] + k < sc.res[a];
            const size_t X = (size_t)sc.res[0], XY = X * (size_t)sc.res[1];
            const float* mass = reinterpret_cast<const float*>(sc.vstar) + 3;  // vstar[node].w
            const long long n0 = (long long)base[0] + (long long)X * base[1] + (long long)XY * base[2];
#pragma unroll
            for (int c = 0; c < S; ++c)
#pragma unroll
                for (int b = 0; b < S; ++b)
#pragma unroll
                    for (int a = 0; a < S; ++a) {
                        if (!(in[0][a] && in[1][b] && in[2][c])) continue;
                        const size_t node = (size_t)(n0 + a + (long long)X * b + (long long)XY * c);
                        const float wgt = w[0][a] * w[1][b] * w[2][c];
                        dens += (__ldg(mass + 4 * node) * wgt) * inv_cell_vol;
                    }
        }
        f[F_VOL * cap + i] = f[F_MASS * cap + i] / dens;
    }
}

// Scatter a live-order particle field back to the original order.
__global__ void gatherFieldKernel(const SceneDev* __restrict__ scenes, int scene, int parity, int field, int comps,
                                  int mode, float* __restrict__ out) {
    const SceneDev& sc = scenes[scene];
    const float* f = sc.buf[parity].f;
    const uint32_t* pid = sc.buf[parity].pid;
    const size_t cap = sc.cap;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < sc.n; i += gridDim.x * kThreads) {
        const uint32_t o = pid[i];
        if (mode == 1) {  // position4: one 16-byte store per particle
            reinterpret_cast<float4*>(out)[o] =
                make_float4(f[F_X * cap + i], f[(F_X + 1) * cap + i], f[(F_X + 2) * cap + i], 1.0f);
        } else if (mode == 2) {  // det of a 3x3 field
            float M[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) M[k] = f[(field + k) * cap + i];
            out[o] = det3(M);
        } else {
            for (int c = 0; c < comps; ++c) out[(size_t)comps * o + c] = f[(field + c) * cap + i];
        }
    }
}

// Overwrite a live-order particle field from original-order data.
__global__ void scatterFieldKernel(const SceneDev* __restrict__ scenes, int scene, int parity, int field, int comps,
                                   const float* __restrict__ in) {
    const SceneDev& sc = scenes[scene];
    float* f = sc.buf[parity].f;
    const uint32_t* pid = sc.buf[parity].pid;
    const size_t cap = sc.cap;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < sc.n; i += gridDim.x * kThreads) {
        const uint32_t o = pid[i];
        for (int c = 0; c < comps; ++c) f[(field + c) * cap + i] = in[(size_t)comps * o + c];
    }
}

// ---------------------------------------------------------------------------
// Launch wrappers (host).
// ---------------------------------------------------------------------------
void launchKeys(const LaunchCtx& c, int parity, uint32_t* keys, uint32_t* block_count, uint32_t* err) {
    noteLaunches(1);
    keyKernel<<<dim3(c.particle_blocks, c.nscenes), kThreads, 0, c.stream>>>(c.scenes, parity, keys, block_count, err);
}

size_t compactScratchWords64(uint32_t total_blocks) {
    return (size_t)(total_blocks + kCompactTile - 1) / kCompactTile + 1;  // + the tile counter
}

void launchCompact(const LaunchCtx& c, const BlockBuffers& bb, uint32_t total_blocks, unsigned long long* scratch,
                   const ComboSplit& split, uint32_t* err) {
    const CompactArgs a{bb.block_count, total_blocks,     bb.scene_block_base, c.nscenes,        bb.active,
                        bb.outside,     bb.counters,      bb.block_slot,       bb.g2p_items,     bb.g2p_cap,
                        split,          bb.p2g_lists,     bb.p2g_list_cap,     bb.block_range,   bb.emig_count,
                        bb.moved,       bb.sort_list,     bb.sort_list_cap,    bb.dense_list,    c.scenes,
                        err};
    if (total_blocks <= kClusterBlocks) {
        noteLaunches(1);
        compactClusterKernel<<<kClusterCtas, kClusterThreads, 0, c.stream>>>(a);
        return;
    }
    const uint32_t ntiles = (uint32_t)((total_blocks + kCompactTile - 1) / kCompactTile);
    ClearRanges cr;
    cr.p[0] = reinterpret_cast<uint32_t*>(scratch);
    cr.n[0] = 2 * compactScratchWords64(total_blocks);
    cr.p[1] = bb.counters;
    cr.n[1] = 4;
    cr.p[2] = bb.counters + kG2PCountWord;
    cr.n[2] = kMaxCombos;
    cr.p[3] = bb.counters + kP2GListWord;  // lists, small, back, the block sort's lists
    cr.n[3] = kSortSchedWord - kP2GListWord;
    launchClear(cr, c.stream);
    noteLaunches(1);
    compactOnesweepKernel<<<ntiles, kCompactThreads, 0, c.stream>>>(a, scratch + 1, reinterpret_cast<uint32_t*>(scratch), ntiles);
}

void launchStress(const LaunchCtx& c, int parity) {
    noteLaunches(1);
    stressKernel<<<dim3(c.particle_blocks, c.nscenes), kThreads, 0, c.stream>>>(c.scenes, parity);
}

// Raises a kernel's limit of dynamic shared memory on the current device.  A
// failure stays the last error, which the caller's check after the launch reports.
template <auto Kernel>
static void allowSharedMemory(size_t bytes) {
    static OncePerDevice once;
    int device = 0;
    cudaGetDevice(&device);
    once(device, [&] { return cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); });
}

// Particles staged per warp pass in P2G: in the fused step the engine's setting
// (16, 24 or 32: mpm_tuning.p2g_stage, else kDefaultP2GStage), elsewhere
// kDefaultP2GStage.  Every size gives bitwise the same sums.
template <int S, int MODE, int STAGE>
static void p2gLaunch(const LaunchCtx& c, const StepArgs& a, int want) {
    allowSharedMemory<p2gKernel<S, MODE, STAGE>>(P2GLayout<S, MODE, STAGE>::smemBytes);
    p2gKernel<S, MODE, STAGE><<<c.persistent_blocks, P2GLayout<S, MODE, STAGE>::NT, P2GLayout<S, MODE, STAGE>::smemBytes,
                                c.stream>>>(a, want);
}

template <int S, int MODE>
static void p2gOne(const LaunchCtx& c, const StepArgs& a, int want) {
    switch (c.p2g_stage) {
        case 16: p2gLaunch<S, MODE, 16>(c, a, want); break;
        case 24: p2gLaunch<S, MODE, 24>(c, a, want); break;
        default: p2gLaunch<S, MODE, 32>(c, a, want); break;
    }
}

template <int S, int MODE>
static void p2gWarpLaunch(const LaunchCtx& c, const StepArgs& a) {
    using W = P2GWarpLayout<S, MODE>;
    allowSharedMemory<p2gWarpKernel<S, MODE>>(W::smemBytes);
    const unsigned grid = std::min<unsigned>(c.persistent_blocks, (unsigned)std::max(1, c.num_sms) * W::MIN_CTAS);
    p2gWarpKernel<S, MODE><<<grid, W::NT, W::smemBytes, c.stream>>>(a);
}

void launchP2GWarp(const LaunchCtx& c, const StepArgs& a, int S, int mode) {
    noteLaunches(1);
    const bool apic = mode == MODE_APIC_FUSED;
    if (S == 4) apic ? p2gWarpLaunch<4, MODE_APIC_FUSED>(c, a) : p2gWarpLaunch<4, MODE_FLIP>(c, a);
    else if (S == 3) apic ? p2gWarpLaunch<3, MODE_APIC_FUSED>(c, a) : p2gWarpLaunch<3, MODE_FLIP>(c, a);
    else apic ? p2gWarpLaunch<2, MODE_APIC_FUSED>(c, a) : p2gWarpLaunch<2, MODE_FLIP>(c, a);
}

void launchP2G(const LaunchCtx& c, const StepArgs& a, int S, int mode, int want_transfer) {
    noteLaunches(1);
#define P2G_CASE(SS)                                                                   \
    if (S == SS) {                                                                     \
        switch (mode) {                                                                \
            case MODE_APIC_FUSED: p2gOne<SS, MODE_APIC_FUSED>(c, a, want_transfer); break; \
            case MODE_FLIP: p2gOne<SS, MODE_FLIP>(c, a, want_transfer); break;         \
            case MODE_SPLIT: p2gLaunch<SS, MODE_SPLIT, kDefaultP2GStage>(c, a, want_transfer); break; \
            case MODE_HESS: p2gLaunch<SS, MODE_HESS, kDefaultP2GStage>(c, a, want_transfer); break;   \
            default: p2gLaunch<SS, MODE_MASS, kDefaultP2GStage>(c, a, want_transfer); break;          \
        }                                                                              \
    }
    P2G_CASE(2) P2G_CASE(3) P2G_CASE(4)
#undef P2G_CASE
}

void launchGrid(const LaunchCtx& c, const StepArgs& a, int S, int mode, int want_transfer) {
    noteLaunches(1);
#define GRID_CASE(SS)                                                                                         \
    if (S == SS) {                                                                                            \
        switch (mode) {                                                                                       \
            case MODE_APIC_FUSED: gridKernel<SS, MODE_APIC_FUSED><<<c.persistent_blocks, kThreads, 0, c.stream>>>(a, want_transfer); break; \
            case MODE_FLIP: gridKernel<SS, MODE_FLIP><<<c.persistent_blocks, kThreads, 0, c.stream>>>(a, want_transfer); break; \
            case MODE_SPLIT: gridKernel<SS, MODE_SPLIT><<<c.persistent_blocks, kThreads, 0, c.stream>>>(a, want_transfer); break; \
            default: gridKernel<SS, MODE_MASS><<<c.persistent_blocks, kThreads, 0, c.stream>>>(a, want_transfer); break; \
        }                                                                                                     \
    }
    GRID_CASE(2) GRID_CASE(3) GRID_CASE(4)
#undef GRID_CASE
}

constexpr size_t kG2PDynSmem = sizeof(float) * 2 * kG2PThreads * kPreStride;
template <int S, bool APIC>
static void g2pLaunch(const LaunchCtx& c, const StepArgs& a, int fused) {
    allowSharedMemory<g2pKernel<S, APIC>>(kG2PDynSmem);
    g2pKernel<S, APIC><<<(c.persistent_blocks * 256 + kG2PThreads - 1) / kG2PThreads, kG2PThreads, kG2PDynSmem, c.stream>>>(a, fused);
}

void launchG2P(const LaunchCtx& c, const StepArgs& args, int S, bool apic, bool fused, int combo) {
    noteLaunches(1);
    StepArgs a = args;
    a.combo = combo;
#define G2P_CASE(SS)                                  \
    if (S == SS) {                                    \
        if (apic) g2pLaunch<SS, true>(c, a, fused ? 1 : 0); \
        else g2pLaunch<SS, false>(c, a, fused ? 1 : 0);     \
    }
    G2P_CASE(2) G2P_CASE(3) G2P_CASE(4)
#undef G2P_CASE
}

void launchDenseGravity(const LaunchCtx& c) {
    noteLaunches(1);
    denseGravityKernel<<<dim3(c.node_blocks, c.nscenes), kThreads, 0, c.stream>>>(c.scenes);
}
void launchDenseUpdate(const LaunchCtx& c, float dt) {
    noteLaunches(1);
    denseUpdateVelocityKernel<<<dim3(c.node_blocks, c.nscenes), kThreads, 0, c.stream>>>(c.scenes, dt);
}
void launchDenseCollision(const LaunchCtx& c, float dt) {
    noteLaunches(1);
    denseCollisionKernel<<<dim3(c.node_blocks, c.nscenes), kThreads, 0, c.stream>>>(c.scenes, dt);
}
void launchDensePack(const LaunchCtx& c) {
    noteLaunches(1);
    densePackKernel<<<dim3(c.node_blocks, c.nscenes), kThreads, 0, c.stream>>>(c.scenes);
}
void launchParticlesCollision(const LaunchCtx& c, int parity, float dt) {
    noteLaunches(1);
    particlesCollisionKernel<<<dim3(c.particle_blocks, c.nscenes), kThreads, 0, c.stream>>>(c.scenes, parity, dt);
}
void launchAdvect(const LaunchCtx& c, int parity, float dt) {
    noteLaunches(1);
    advectKernel<<<dim3(c.particle_blocks, c.nscenes), kThreads, 0, c.stream>>>(c.scenes, parity, dt);
}
void launchInitState(cudaStream_t st, int num_sms, float* f, uint32_t* pid, uint16_t* mat, size_t cap,
                     const float* staged, size_t n, bool has_volume, const uint32_t* perm, const uint16_t* mat_in) {
    if (n == 0) return;
    noteLaunches(1);
    const unsigned blocks = (unsigned)std::min<size_t>((n + kThreads - 1) / kThreads, (size_t)num_sms * 8);
    initStateKernel<<<blocks, kThreads, 0, st>>>(f, pid, mat, cap, staged, n, has_volume ? 1 : 0, perm, mat_in);
}
void launchStagedKeys(cudaStream_t st, int num_sms, const SceneDev& sc, const float* xyz, uint32_t n, uint32_t* keys,
                      uint32_t* err) {
    if (n == 0) return;
    noteLaunches(1);
    const unsigned blocks = (unsigned)std::min<size_t>((n + kThreads - 1) / kThreads, (size_t)num_sms * 8);
    stagedKeyKernel<<<blocks, kThreads, 0, st>>>(sc, xyz, n, keys, err);
}
void launchVolume(const LaunchCtx& c, int parity, int S) {
    noteLaunches(1);
    dim3 g(c.particle_blocks, c.nscenes);
    if (S == 2) volumeKernel<2><<<g, kThreads, 0, c.stream>>>(c.scenes, parity);
    else if (S == 3) volumeKernel<3><<<g, kThreads, 0, c.stream>>>(c.scenes, parity);
    else volumeKernel<4><<<g, kThreads, 0, c.stream>>>(c.scenes, parity);
}
// Density rasterisation (writeToOpenVDB, src/mpm_solver3d.cu:509-572): node
// density = sum_p m_p w_ip / h^3, from the node masses of a mass pass.
__global__ void densityKernel(const float4* __restrict__ vstar, size_t nodes, float inv_cell_vol,
                              float* __restrict__ out) {
    for (size_t i = blockIdx.x * (size_t)kThreads + threadIdx.x; i < nodes; i += (size_t)gridDim.x * kThreads)
        out[i] = vstar[i].w * inv_cell_vol;
}
// CFL time step (listed as unimplemented in the reference, README.md:60-67).
// A non-finite speed (NaN or Inf velocity, or |v|^2 overflowing) would leave
// dt without a bound (fmaxf drops NaN) or make it 0 (Inf): it raises
// ERR_NONFINITE, which the next synchronize reports as MPM_ERR_NUMERIC, and is
// left out of the maximum.
__global__ void __launch_bounds__(kThreads) cflMaxKernel(const SceneDev* __restrict__ scenes, int parity,
                                                         uint32_t* __restrict__ err) {
    const SceneDev& sc = scenes[blockIdx.y];
    if (!(sc.cfl > 0.f)) return;
    const float* f = sc.buf[parity].f;
    const size_t cap = sc.cap;
    float m = 0.f;
    bool bad = false;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < sc.n; i += gridDim.x * kThreads) {
        const float vx = f[(F_V + 0) * cap + i], vy = f[(F_V + 1) * cap + i], vz = f[(F_V + 2) * cap + i];
        const float v2 = __fadd_rn(__fadd_rn(__fmul_rn(vx, vx), __fmul_rn(vy, vy)), __fmul_rn(vz, vz));
        if (isfinite(v2)) m = fmaxf(m, v2);
        else bad = true;
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(err, ERR_NONFINITE);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float wm[kThreads / 32];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kThreads / 32; ++w) m = fmaxf(m, wm[w]);
        if (m > 0.f) atomicMax(&sc.cfl_state->vmax2_bits, __float_as_uint(m));
    }
}
// One thread per scene: dt from the maximum, written into the (device) scene
// table that the step's kernels read, then the maximum is cleared.
__global__ void cflFinalizeKernel(SceneDev* __restrict__ scenes, int nscenes) {
    for (int i = threadIdx.x; i < nscenes; i += blockDim.x) {
        SceneDev& sc = scenes[i];
        if (!(sc.cfl > 0.f)) continue;
        CflState* st = sc.cfl_state;
        const float vmax = sqrtf(__uint_as_float(st->vmax2_bits));
        float dt = sc.dt_max;
        if (vmax > 0.f) dt = fminf(dt, __fdiv_rn(__fmul_rn(sc.cfl, sc.h), vmax));
        sc.dt = dt;
        st->vmax2_bits = 0u;
        st->last_dt = dt;
        st->time += (double)dt;
    }
}
void launchCfl(const LaunchCtx& c, int parity, size_t max_n, uint32_t* err) {
    noteLaunches(2);
    const unsigned bx = (unsigned)std::max<size_t>(
        1, std::min<size_t>((max_n + kThreads - 1) / kThreads, (size_t)c.num_sms * 4));
    cflMaxKernel<<<dim3(bx, (unsigned)c.nscenes), kThreads, 0, c.stream>>>(c.scenes, parity, err);
    cflFinalizeKernel<<<1, 128, 0, c.stream>>>(const_cast<SceneDev*>(c.scenes), c.nscenes);
}
void launchDensity(const LaunchCtx& c, const float4* vstar, size_t nodes, float inv_cell_vol, float* out) {
    noteLaunches(1);
    const unsigned blocks = (unsigned)std::max<size_t>(1, std::min<size_t>((nodes + kThreads - 1) / kThreads,
                                                                          (size_t)c.num_sms * 16));
    densityKernel<<<blocks, kThreads, 0, c.stream>>>(vstar, nodes, inv_cell_vol, out);
}
// Loads the kernels of the host transfers (gather for downloads, scatter
// for uploads) on the current device: with CUDA's lazy loading a kernel is
// loaded at its first launch, which would otherwise stall a user's first
// download after the steps (about 2 ms).  Called once per device.
void preloadTransferKernels() {
    cudaFuncAttributes attr;
    cudaFuncGetAttributes(&attr, gatherFieldKernel);
    cudaFuncGetAttributes(&attr, scatterFieldKernel);
    cudaGetLastError();
}

void launchGatherField(const LaunchCtx& c, int scene, int parity, int field, int comps, int mode, float* out) {
    noteLaunches(1);
    gatherFieldKernel<<<c.particle_blocks, kThreads, 0, c.stream>>>(c.scenes, scene, parity, field, comps, mode, out);
}
void launchScatterField(const LaunchCtx& c, int scene, int parity, int field, int comps, const float* in) {
    noteLaunches(1);
    scatterFieldKernel<<<c.particle_blocks, kThreads, 0, c.stream>>>(c.scenes, scene, parity, field, comps, in);
}

// TMA tensor map of a dense float4 grid of res[0] x res[1] x res[2] nodes
// (node index x + X (y + Y z)) as a 4-D FP32 tensor (component, x, y, z),
// box (4, T, T, T), zero fill outside the grid.  The encoder is the driver's
// cuTensorMapEncodeTiled, fetched once through the runtime.
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encodeTiledFn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return (EncodeTiledFn) nullptr;
        }
        return (EncodeTiledFn)p;
    }();
    return fn;
}
const char* encodeGridTensorMap(void* map, const void* grid, const int* res, int T) {
    static_assert(sizeof(CUtensorMap) == kTensorMapBytes, "tensor map size");
    EncodeTiledFn fn = encodeTiledFn();
    if (!fn) return "cuTensorMapEncodeTiled is not available from the driver";
    if (((uintptr_t)grid & 15u) != 0) return "grid buffer not 16-byte aligned";
    const cuuint64_t dims[4] = {4, (cuuint64_t)res[0], (cuuint64_t)res[1], (cuuint64_t)res[2]};
    const cuuint64_t strides[3] = {16, 16ull * (cuuint64_t)res[0], 16ull * (cuuint64_t)res[0] * (cuuint64_t)res[1]};
    const cuuint32_t box[4] = {4, (cuuint32_t)T, (cuuint32_t)T, (cuuint32_t)T};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = fn(reinterpret_cast<CUtensorMap*>(map), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                          const_cast<void*>(grid), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? nullptr : "cuTensorMapEncodeTiled rejected the grid tensor map";
}

}  // namespace mpm
