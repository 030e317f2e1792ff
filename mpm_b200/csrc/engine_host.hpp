// engine_host.hpp -- host-side launch interface between the engine and the kernels.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/mpm_b200.h"
#include "engine.cuh"

namespace mpm {

struct LaunchCtx {
    const SceneDev* scenes;   // device scene table
    int nscenes;
    cudaStream_t stream;
    unsigned particle_blocks;   // grid.x of per-particle kernels (grid.y = scene)
    unsigned node_blocks;       // grid.x of dense per-node kernels
    unsigned persistent_blocks; // grid of the persistent block kernels
    int num_sms;
    int p2g_stage;              // particles staged per warp pass in the fused step's P2G (16, 24 or 32)
};

struct BlockBuffers {
    uint32_t* block_count;            // total_blocks
    uint32_t* scene_block_base;       // nscenes + 1
    BlockItem* active;                // max_active
    BlockItem* outside;               // nscenes
    BlockItem* g2p_items;             // G2P work items, g2p_cap per combination
    uint32_t g2p_cap;
    uint32_t* counters;               // see kG2PCountWord, kP2GListWord
    int2* block_slot;                 // total_blocks
    uint32_t* p2g_lists;              // P2G item slots, 2 lists of p2g_list_cap per combination
    uint32_t p2g_list_cap;
    uint2* block_range;               // total_blocks: (first sorted particle, count)
    uint32_t* emig_count;             // total_blocks: cleared for the next step
    uint32_t* moved;                  // likewise
    BlockItem* sort_list;             // see BlockSortArgs
    uint32_t sort_list_cap;
    BlockItem* dense_list;
};

// Host-side count of kernel launches issued by the library (kernels.cu).
void noteLaunches(uint64_t n);
uint64_t kernelLaunches();

// sort.cu
// Up to four word ranges zeroed by one kernel launch (launchClear): the
// step's scratch clears are kernels rather than memset nodes, which a
// device-to-host copy running beside the step (an asynchronous download on
// another stream) held back by 8-20 us each.
struct ClearRanges {
    uint32_t* p[4] = {};
    size_t n[4] = {};
};
void launchClear(const ClearRanges& r, cudaStream_t st);
size_t scanScratchElems(size_t n);
template <class T>
cudaError_t exclusiveScan(const T* in, T* out, size_t n, T* partials, T* total, cudaStream_t st);
size_t radixTiles(size_t n);
size_t onesweepScratchWords(size_t n, int bits);
cudaError_t radixSortOnesweep(uint32_t* keys_a, uint32_t* vals_a, uint32_t* keys_b, uint32_t* vals_b, size_t n,
                              int bits, uint32_t* scratch, uint32_t* err, bool* result_in_b, cudaStream_t st);
// Block sort (sort.cu): the stable sort of `keys` (live order) given that the
// live order is the order of the previous sort: launchEmigrants lists the
// particles that left their blocks (counts zero before), the compaction the
// occupied blocks with their new ranges, then launchBlockSort sorts, block by
// block or, where many particles left their blocks, by radix passes over all
// keys.  Output equals radixSortOnesweep's (keys, perm).
struct BlockSortArgs {
    const SceneDev* scenes;
    int nscenes;
    const uint32_t* scene_block_base;
    uint32_t n;                  // particles
    unsigned sort_grid;          // blockSortGrid: CTAs of the block sort
    int key_bits;
    uint32_t* keys;              // live order (overwritten by the radix passes)
    const uint32_t* prev_keys;   // live order: the previous step's sorted keys
    const uint2* prev_range;     // per block: (first, count) in the live order
    uint32_t* emig_count;        // per block: particles that left it for a neighbouring block
    uint2* emig;                 // (live index, key) of those of block b from prev_range[b].x on
    uint2* far;                  // (live index, key) of the other particles that left their block
    uint32_t* moved;             // [0] entries of far, [1] all particles that left their block,
                                 // [2] blocks that more than kEmigMax left
    const BlockItem* list;       // occupied blocks and their new ranges, full ones from the front,
    uint32_t list_cap;           // the others from the back (kSortFrontWord, kSortBackWord)
    const BlockItem* dense;      // the blocks of at least kDenseBlock particles (kSortDenseWord)
    uint32_t* counters;
    unsigned long long* aux;     // one word per particle: arrivals that exceed shared memory
    uint32_t *out_keys, *out_perm;
    uint32_t *spare_vals, *radix_scratch;  // of the radix passes: n words, blockSortScratchWords
    uint32_t* err;
};
size_t blockSortScratchWords(size_t n, int bits);
unsigned blockSortGrid(unsigned max_blocks, int num_sms);
cudaError_t launchEmigrants(const BlockSortArgs& a, int num_sms, cudaStream_t st);
cudaError_t launchBlockSort(const BlockSortArgs& a, cudaStream_t st);
// The blocks of at least kDenseBlock particles, at most max_blocks of them, or
// the radix passes (it may run beside launchBlockSort, on another stream).
cudaError_t launchBlockSortDense(const BlockSortArgs& a, unsigned max_blocks, int num_sms, cudaStream_t st);
cudaError_t radixSortPairsInto(const uint32_t* in_keys, uint32_t* out_keys, uint32_t* out_vals, uint32_t* tmp_keys,
                               uint32_t* tmp_vals, size_t n, int bits, uint32_t* hist, uint32_t* scan_partials,
                               cudaStream_t st);

// kernels.cu
void launchKeys(const LaunchCtx& c, int parity, uint32_t* keys, uint32_t* block_count, uint32_t* err);
size_t compactScratchWords64(uint32_t total_blocks);
// How the compaction splits each (stencil, transfer) combination's work:
// particles per G2P work item, and the largest P2G item taken by a single
// warp (0: none).
struct ComboSplit {
    uint32_t g2p_chunk[kMaxCombos];
    uint32_t p2g_warp_max[kMaxCombos];
};
void launchCompact(const LaunchCtx& c, const BlockBuffers& bb, uint32_t total_blocks,
                           unsigned long long* scratch, const ComboSplit& split, uint32_t* err);
void launchStress(const LaunchCtx& c, int parity);
void launchP2G(const LaunchCtx& c, const StepArgs& a, int S, int mode, int want_transfer);
// P2G of the combination a.combo's warp list (a.p2g_lists set): one warp per
// item, tiles bitwise those of launchP2G.
void launchP2GWarp(const LaunchCtx& c, const StepArgs& a, int S, int mode);
void launchGrid(const LaunchCtx& c, const StepArgs& a, int S, int mode, int want_transfer);
void launchG2P(const LaunchCtx& c, const StepArgs& a, int S, bool apic, bool fused, int combo);
void launchDenseGravity(const LaunchCtx& c);
void launchDenseUpdate(const LaunchCtx& c, float dt);
void launchDenseCollision(const LaunchCtx& c, float dt);
void launchDensePack(const LaunchCtx& c);
void launchParticlesCollision(const LaunchCtx& c, int parity, float dt);
void launchAdvect(const LaunchCtx& c, int parity, float dt);
void launchVolume(const LaunchCtx& c, int parity, int S);
// A new scene's particle planes from its staged arrays, slot i from the
// caller's particle perm[i] (perm null: i); mat_in null: no material ids.
void launchInitState(cudaStream_t st, int num_sms, float* f, uint32_t* pid, uint16_t* mat, size_t cap,
                     const float* staged, size_t n, bool has_volume, const uint32_t* perm, const uint16_t* mat_in);
// Cell keys (sc's block numbering) of n staged interleaved positions.
void launchStagedKeys(cudaStream_t st, int num_sms, const SceneDev& sc, const float* xyz, uint32_t n, uint32_t* keys,
                      uint32_t* err);
void launchDensity(const LaunchCtx& c, const float4* vstar, size_t nodes, float inv_cell_vol, float* out);
// Semi-implicit solve (implicit.cu) of the scenes with beta > 0.  Global
// buffers over the sorted particles of the batch and its cell keys.
struct SolveBuffers {
    const uint32_t* sorted_keys;  // ntot
    const uint32_t* perm;         // ntot
    float4* pofs;                 // ntot: stencil offsets (x - (o + h base)) / h (sorted order)
    float* prep;                  // kSolvePrepPlanes x ntot
    float4* T;                    // 3 x ntot: V0 dP Fe^T rows
    uint32_t ntot;
    int* iter;                    // device iteration counter
};
constexpr int kSolvePrepPlanes = 44;
constexpr int kSolveVectors = 6;
constexpr int kSolveBlocks = 512;  // node-kernel blocks per scene = partial sums per dot product
inline size_t solvePartialDoubles(int max_iter) { return (size_t)4 * (size_t)(max_iter + 2) * kSolveBlocks; }
// split: v* from and to the split-mode dense planes (no collision after);
// else from and to the fused step's v* grid, with the grid collision after.
// aux: an idle stream on which, inside a stream capture, the iteration body
// is captured as the body of a conditional while node.
// step: the arguments of the step's P2G (work items, tiles, schedulers).
cudaError_t launchSolve(const LaunchCtx& c, const StepArgs& step, const SolveBuffers& b, int parity, const int* stencils, int nstencils,
                        int max_iter, bool split, cudaStream_t aux);

// CFL time step of the scenes with cfl > 0: max |v|^2 over their live
// particles, then dt = min(dt_max, cfl h / max|v|) into the scene table.
// A non-finite particle speed sets ERR_NONFINITE in err.
void launchCfl(const LaunchCtx& c, int parity, size_t max_n, uint32_t* err);
void launchGatherField(const LaunchCtx& c, int scene, int parity, int field, int comps, int mode, float* out);
void preloadTransferKernels();
void launchScatterField(const LaunchCtx& c, int scene, int parity, int field, int comps, const float* in);
// Writes the kTensorMapBytes TMA tensor map of a dense float4 grid (res[3]
// nodes) with tile box T^3 to map (host memory); returns null or a message.
const char* encodeGridTensorMap(void* map, const void* grid, const int* res, int T);

}  // namespace mpm
