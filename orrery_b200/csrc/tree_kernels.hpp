// Launch interface of the Barnes-Hut pipeline's kernels (sort.cu, tree.cu,
// walk.cu). Raw device pointers; every launcher enqueues on `stream` only.
#pragma once

#include <atomic>
#include <cstdint>

#include <cuda_runtime.h>

#include "tree.hpp"

namespace ob {

// ---------------------------------------------------------------- ordering

// Radix sort geometry: 8-bit digits, 8 passes over the 63-bit codes.
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kRadixPasses = 8;
constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr uint32_t kSortTile = kSortThreads * kSortItems;

// Bounding-cube reduction: blocks of the min/max pass (4 per SM); the
// partials buffer holds 6 doubles per block.
constexpr uint32_t kCubeThreads = 256;
constexpr uint32_t kCubeBlocks = 592;

// Largest particle count the onesweep status words can carry (30-bit counts).
constexpr uint32_t kMaxTreeParticles = (1u << 30) - 1;

uint32_t sort_tiles(uint32_t n);
size_t cube_partials_needed(uint32_t n);

// Bounding cube (src/solvers/morton.cpp:60-104) into meta->origin/size and
// meta->root_centre; `partials` holds cube_partials_needed() doubles and
// meta->cube_blocks_done starts at zero (the last block to finish folds the
// partials).
cudaError_t launch_bounding_cube(const double *x, const double *y, const double *z, uint32_t n,
                                 double *partials, TreeMeta *meta, cudaStream_t stream);

// Morton codes (morton.cpp:128-164) with index payload, and the eight digit
// histograms of the codes (hist: kRadixPasses x kRadix, zeroed beforehand).
cudaError_t launch_encode(const double *x, const double *y, const double *z, uint32_t n,
                          const TreeMeta *meta, unsigned long long *codes, uint32_t *indices,
                          uint32_t *hist, cudaStream_t stream);

// Exclusive scan of each pass's histogram, in place.
cudaError_t launch_scan_histograms(uint32_t *hist, cudaStream_t stream);

// One onesweep pass (stable) over digit `pass`. `lookback` holds
// sort_tiles(n) * kRadix status words for this pass and `ticket` one counter,
// both zeroed beforehand. A tile polls a predecessor's look-back word at most
// `poll_limit` times (the default is far above any legitimate wait); when the
// polls run out it sets the timeout bit in `status` and returns unscattered.
constexpr uint32_t kLookbackPollLimit = 1u << 24;
cudaError_t launch_onesweep(const unsigned long long *keys_in, const uint32_t *vals_in,
                            unsigned long long *keys_out, uint32_t *vals_out, uint32_t n,
                            int pass, const uint32_t *offsets, uint32_t *lookback,
                            uint32_t *ticket, unsigned *status, cudaStream_t stream,
                            uint32_t poll_limit = kLookbackPollLimit);

// CTAs of a cooperative launch: as many as are resident at once, at most
// `wanted`. `configured` and `resident` are the caller's per-kernel caches.
constexpr uint32_t kMaxCooperativeBlocks = 592; // 4 per SM
cudaError_t cooperative_grid(const void *kernel, int threads, size_t smem,
                             std::atomic<uint64_t> &configured, std::atomic<int> &resident,
                             uint32_t wanted, uint32_t &grid);

// The whole ordering in one cooperative launch: the bounding cube into meta,
// codes (ending in keys[0]) and the permutation (perm[0]), and sorted[k * n + i]
// = source_k[perm[0][i]] for x, y, z, m; *meta's other scalars and the
// `zeroed_words` words at `zeroed` are zeroed on the way. `barrier` (one word)
// is zero at the start; hist, lookback (of all passes) and `partials`
// (order_partials_needed() doubles) are scratch. A bounded wait that ran out sets
// kStatusTimeout and leaves no nodes (kNodesUnset, tree.hpp). With a
// `silent` stage (tests) the waits end after `poll_limit` polls.
size_t order_partials_needed();
cudaError_t launch_order(const double *x, const double *y, const double *z, const double *m,
                         uint32_t n, unsigned long long *const *keys, uint32_t *const *perm,
                         uint32_t *hist, uint32_t *lookback, double *partials, double *sorted,
                         uint32_t *zeroed, size_t zeroed_words, TreeMeta *meta,
                         unsigned *barrier, unsigned *status, cudaStream_t stream,
                         SilentStage silent = SilentStage::none, uint32_t poll_limit = 0);

// ------------------------------------------------------------------ octree

// The octree's layout in one cooperative launch: offsets[b] = nodes whose first
// particle comes before b (n + 1 words), the node records (escape, first, count,
// level, parent, octant), and each internal node's children by octant, marked
// in child_mask (zeroed beforehand) and listed in its kMaxChildren child_slots.
// `totals` holds kMaxCooperativeBlocks words; `barrier` is zero at the start.
// After an abandoned ordering it lays out nothing and makes `perm` a permutation,
// so that the walks read and write nothing out of range.
constexpr uint32_t kMaxChildren = 8;
cudaError_t launch_layout(const unsigned long long *codes, uint32_t n, uint32_t leaf_cap,
                          uint32_t *offsets, uint32_t *totals, uint32_t node_capacity,
                          DeviceNode *nodes, uint32_t *child_mask, uint32_t *child_slots,
                          uint32_t *perm, TreeMeta *meta, unsigned *barrier, unsigned *status,
                          cudaStream_t stream, SilentStage silent = SilentStage::none,
                          uint32_t poll_limit = 0);

// Moments bottom-up (mass, centre of mass, quadrupole, acceptance radius) and
// the leaf-relative FP32 source positions the walk reads.
cudaError_t launch_moments(const double *sorted, const unsigned long long *codes, uint32_t n,
                           DeviceNode *nodes, DeviceQuadrupole *quads, const WalkNodes &walk,
                           const uint32_t *child_mask, const uint32_t *child_slots,
                           uint32_t *arrived, float4 *leaf_rel,
                           TreeMeta *meta, double opening_angle, uint32_t node_capacity,
                           cudaStream_t stream);

// ------------------------------------------------------------------- walk

// Accelerations written in the caller's (unsorted) order through perm; pair
// and cell counts added to counters[0] and counters[1]. `quads` NULL: monopoles
// only. stack_cap (0 = the walk's full stack) bounds the group traversal's
// stack; a group whose stack fills finishes with the per-target union walk.
uint32_t walk_stack_capacity();
cudaError_t launch_walk(const DeviceNode *nodes, const DeviceQuadrupole *quads,
                        const WalkNodes &walk, const float4 *leaf_rel, const double *sorted,
                        const uint32_t *perm, uint32_t n, double eps2, double *ax, double *ay,
                        double *az, TreeMeta *meta,
                        unsigned long long *counters, unsigned *status, cudaStream_t stream,
                        uint32_t stack_cap = 0);

// The FP64 walk of the parity mode (walk_f64.cu); `quads` NULL without
// quadrupoles; `sorted` = x, y, z, m in Morton order.
cudaError_t launch_walk_f64(const DeviceNode *nodes, const DeviceQuadrupole *quads,
                            const double *sorted, const uint32_t *perm, uint32_t n, double eps2,
                            double *ax, double *ay, double *az, const TreeMeta *meta,
                            unsigned long long *counters, unsigned *status, cudaStream_t stream);

} // namespace ob
