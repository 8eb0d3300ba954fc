// Morton ordering on the device: bounding cube, 63-bit codes, and a stable
// least-significant-digit radix sort of (code, index) in onesweep form.
//
// Parity with MortonOrdering::build (src/solvers/morton.cpp:180-197) is exact:
//   * the cube is the reference's (morton.cpp:60-104) with every FP64
//     operation explicitly rounded and min/max exact in any order;
//   * codes use the reference's grid mapping (morton.cpp:128-164), truncation
//     and clamps; x, y, z interleaved with x the high bit of each triple;
//   * a stable sort of codes whose payload starts as the identity orders ties
//     by ascending index, which is exactly std::sort on MortonKey's
//     (code, index) ordering (include/orrery/solvers/morton.hpp:155-175).
//
// The sort: one histogram pass (fused into encoding) computes all eight digit
// histograms; in each of the eight passes a CTA takes a tile, ranks its keys
// stably with warp match operations, publishes its per-digit counts, resolves
// its global offsets by decoupled look-back over earlier tiles (every wait
// bounded) and scatters through shared memory so the global writes are
// contiguous runs.
//
// Two routes launch these pieces. The tree's (order_kernel) is one cooperative
// launch for all of it, with a grid barrier between phases and tiles given to
// the CTAs in ascending order. ob_morton_order_noalloc launches each phase by
// itself; there a CTA takes the next tile in launch order from a ticket counter.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "runtime.hpp"
#include "tree_kernels.hpp"

namespace ob {
namespace {

constexpr uint32_t kReduceThreads = kCubeThreads;
constexpr uint32_t kReduceBlocks = kCubeBlocks;

__device__ __forceinline__ void min_max(double v, double &lo, double &hi) {
    lo = v < lo ? v : lo;
    hi = hi < v ? v : hi;
}

// Block-wide min (k < 3) / max (k >= 3) of the six values each thread holds
// in v[]; thread k < 6 receives component k in `out`.
__device__ __forceinline__ void block_min_max(double (&v)[6], double &out) {
    __shared__ double s[6][kReduceThreads / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        for (int off = 16; off > 0; off >>= 1) {
            const double o = __shfl_down_sync(0xffffffffu, v[k], off);
            v[k] = k < 3 ? (o < v[k] ? o : v[k]) : (v[k] < o ? o : v[k]);
        }
        if (lane == 0) {
            s[k][warp] = v[k];
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int k = threadIdx.x;
        double r = s[k][0];
        for (uint32_t w = 1; w < kReduceThreads / 32; ++w) {
            r = k < 3 ? (s[k][w] < r ? s[k][w] : r) : (r < s[k][w] ? s[k][w] : r);
        }
        out = r;
    }
}

// The cube from the extremes (morton.cpp:60-104): edge = the largest extent
// (1 when it is not positive), centred on the box.
__device__ void write_cube(const double *ext, uint32_t n, TreeMeta *meta) {
    if (n == 0) {
        for (int a = 0; a < 3; ++a) {
            meta->origin[a] = 0.0;
            meta->root_centre[a] = 0.0;
        }
        meta->size = 0.0;
        return;
    }
    const double ex = __dsub_rn(ext[3], ext[0]);
    const double ey = __dsub_rn(ext[4], ext[1]);
    const double ez = __dsub_rn(ext[5], ext[2]);
    double size = ex;
    size = size < ey ? ey : size;
    size = size < ez ? ez : size;
    if (!(size > 0.0)) {
        size = 1.0;
    }
    const double half = __ddiv_rn(size, 2.0);
    for (int a = 0; a < 3; ++a) {
        const double centre = __ddiv_rn(__dadd_rn(ext[a], ext[3 + a]), 2.0);
        const double origin = __dsub_rn(centre, half);
        meta->origin[a] = origin;
        // BoundingCube::centre (morton.hpp:93-95): origin + size/2.
        meta->root_centre[a] = __dadd_rn(origin, half);
    }
    meta->size = size;
}

// One pass over the positions: each block writes its six extremes, and the
// last block to finish (an atomic count in meta) folds all blocks' partials
// with the whole block and writes the cube. Min and max are exact, so the
// order of the fold does not change the result.
__global__ void __launch_bounds__(kReduceThreads)
    cube_kernel(const double *__restrict__ x, const double *__restrict__ y,
                const double *__restrict__ z, uint32_t n, double *partials, TreeMeta *meta) {
    double v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        min_max(x[i], v[0], v[3]);
        min_max(y[i], v[1], v[4]);
        min_max(z[i], v[2], v[5]);
    }
    double mine = 0.0;
    block_min_max(v, mine);
    __shared__ bool last;
    if (threadIdx.x < 6) {
        partials[blockIdx.x * 6 + threadIdx.x] = mine;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(&meta->cube_blocks_done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) {
        return;
    }
    __threadfence();
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        v[k] = k < 3 ? INFINITY : -INFINITY;
    }
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            // Empty blocks hold (+inf, -inf): lows only lower, highs only raise.
            const double p = __ldcg(partials + b * 6 + k);
            v[k] = k < 3 ? (p < v[k] ? p : v[k]) : (v[k] < p ? p : v[k]);
        }
    }
    __syncthreads(); // block_min_max's shared array is reused
    __shared__ double ext[6];
    double folded = 0.0;
    block_min_max(v, folded);
    if (threadIdx.x < 6) {
        ext[threadIdx.x] = folded;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        write_cube(ext, n, meta);
    }
}

// Dilation by table: each 7-bit chunk of a grid coordinate maps to 21 bits
// with its bits three apart; three chunks make the 63-bit interleave slot.
__device__ __forceinline__ unsigned long long dilate(const unsigned long long *table,
                                                     uint32_t v) {
    return table[v & 127u] | (table[(v >> 7) & 127u] << 21) | (table[(v >> 14) & 127u] << 42);
}

__device__ __forceinline__ uint32_t to_grid(double coordinate, double origin, double scale) {
    const double cell = __dmul_rn(__dsub_rn(coordinate, origin), scale);
    if (!(cell > 0.0)) {
        return 0u;
    }
    if (cell >= 2097152.0) {
        return 2097151u;
    }
    return __double2uint_rz(cell);
}

// The dilation table and zeroed local histograms (then a barrier).
__device__ __forceinline__ void encode_prepare(unsigned long long *table, uint32_t *local) {
    for (uint32_t k = threadIdx.x; k < 128; k += blockDim.x) {
        unsigned long long d = 0;
        for (int b = 0; b < 7; ++b) {
            d |= static_cast<unsigned long long>((k >> b) & 1u) << (3 * b);
        }
        table[k] = d;
    }
    for (uint32_t k = threadIdx.x; k < kRadixPasses * kRadix; k += blockDim.x) {
        local[k] = 0;
    }
}

// This CTA's share of the codes, and its digit counts added to `hist`.
__device__ __forceinline__ void encode_particles(const double *__restrict__ x,
                                                 const double *__restrict__ y,
                                                 const double *__restrict__ z, uint32_t n,
                                                 const TreeMeta &meta,
                                                 const unsigned long long *table, uint32_t *local,
                                                 unsigned long long *codes, uint32_t *indices,
                                                 uint32_t *hist) {
    const double size = meta.size;
    const bool degenerate = !(size > 0.0);
    const double scale = degenerate ? 0.0 : __ddiv_rn(2097152.0, size);
    const double ox = meta.origin[0], oy = meta.origin[1], oz = meta.origin[2];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        unsigned long long code = 0;
        if (!degenerate) {
            code = (dilate(table, to_grid(x[i], ox, scale)) << 2) |
                   (dilate(table, to_grid(y[i], oy, scale)) << 1) |
                   dilate(table, to_grid(z[i], oz, scale));
        }
        codes[i] = code;
        indices[i] = i;
#pragma unroll
        for (int p = 0; p < kRadixPasses; ++p) {
            atomicAdd(&local[p * kRadix + ((code >> (kRadixBits * p)) & (kRadix - 1))], 1u);
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kRadixPasses * kRadix; k += blockDim.x) {
        if (local[k] != 0) {
            atomicAdd(&hist[k], local[k]);
        }
    }
}

__global__ void __launch_bounds__(kReduceThreads)
    encode_kernel(const double *__restrict__ x, const double *__restrict__ y,
                  const double *__restrict__ z, uint32_t n, const TreeMeta *meta,
                  unsigned long long *codes, uint32_t *indices, uint32_t *hist) {
    __shared__ unsigned long long table[128];
    __shared__ uint32_t local[kRadixPasses * kRadix];
    encode_prepare(table, local);
    __syncthreads();
    encode_particles(x, y, z, n, *meta, table, local, codes, indices, hist);
}

__global__ void scan_histograms_kernel(uint32_t *hist) {
    __shared__ uint32_t s[kRadix];
    uint32_t *h = hist + blockIdx.x * kRadix;
    const uint32_t t = threadIdx.x;
    s[t] = h[t];
    __syncthreads();
    for (uint32_t off = 1; off < kRadix; off <<= 1) {
        const uint32_t v = t >= off ? s[t - off] : 0u;
        __syncthreads();
        s[t] += v;
        __syncthreads();
    }
    h[t] = t == 0 ? 0u : s[t - 1];
}

// Status words of the look-back: 2-bit flag over a 30-bit count.
constexpr uint32_t kFlagAggregate = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kCountMask = (1u << 30) - 1;

__device__ __forceinline__ uint32_t load_volatile(const uint32_t *p) {
    return *reinterpret_cast<const volatile uint32_t *>(p);
}

__device__ __forceinline__ void store_volatile(uint32_t *p, uint32_t v) {
    *reinterpret_cast<volatile uint32_t *>(p) = v;
}

constexpr uint32_t kWarps = kSortThreads / 32;

// Shared memory of a tile's ranking and scatter.
struct SortSpace {
    unsigned long long keys[kSortTile];
    uint32_t vals[kSortTile];
    uint32_t warp[kWarps * kRadix]; // counts per warp and digit, then prefixes
    uint32_t start[kRadix];         // tile-local digit start
    uint32_t base[kRadix];          // global output base per digit
    uint32_t sums[kWarps];          // digit counts of each warp's 32 digits
    uint32_t tile;
};

// One tile of a pass: ranks its keys stably by digit, publishes its counts,
// resolves its output bases by looking back over earlier tiles (bounded polls)
// and scatters. `offset`: where digit threadIdx.x starts in the output.
// space.warp is zeroed by the caller (and a barrier passed); the caller passes
// a barrier before it reuses the space. False, in every thread, when a wait ran
// out.
__device__ __forceinline__ bool sort_one_tile(SortSpace &space, uint32_t tile,
                                              const unsigned long long *keys_in,
                                              const uint32_t *vals_in,
                                              unsigned long long *keys_out, uint32_t *vals_out,
                                              uint32_t n, uint32_t shift, uint32_t offset,
                                              uint32_t *lookback, unsigned *status,
                                              uint32_t poll_limit) {
    static_assert(kSortThreads == kRadix, "thread t owns digit t");
    unsigned long long *s_keys = space.keys;
    uint32_t *s_vals = space.vals, *s_warp = space.warp, *s_start = space.start;
    uint32_t *s_base = space.base, *s_sums = space.sums;
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t *hist = s_warp + warp * kRadix;
    const uint32_t base = tile * kSortTile;

    // Warp-striped load: the tile order of (warp, item, lane) is this order.
    // All of a thread's loads are issued before the ranking's barriers.
    unsigned long long key[kSortItems];
    uint32_t val[kSortItems], digit[kSortItems], rank[kSortItems];
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        const uint32_t i = base + warp * (kSortItems * 32) + it * 32 + lane;
        const bool valid = i < n;
        key[it] = valid ? __ldcg(keys_in + i) : 0ull;
        val[it] = valid ? __ldcg(vals_in + i) : 0u;
    }
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        const bool valid = base + warp * (kSortItems * 32) + it * 32 + lane < n;
        digit[it] = valid ? static_cast<uint32_t>((key[it] >> shift) & (kRadix - 1)) : kRadix;
        // Stable warp-local rank: earlier items first, then lower lanes.
        const uint32_t peers = __match_any_sync(0xffffffffu, digit[it]);
        const uint32_t before = __popc(peers & lt_mask);
        const uint32_t running = valid ? hist[digit[it]] : 0u;
        __syncwarp();
        if (valid && before == 0) {
            hist[digit[it]] = running + __popc(peers);
        }
        __syncwarp();
        rank[it] = running + before;
    }
    __syncthreads();

    // Thread t owns digit t: tile count, warp prefixes, publish, look back.
    const uint32_t d = tid;
    uint32_t count = 0;
    for (uint32_t w = 0; w < kWarps; ++w) {
        const uint32_t c = s_warp[w * kRadix + d];
        s_warp[w * kRadix + d] = count;
        count += c;
    }
    uint32_t *mine = lookback + static_cast<size_t>(tile) * kRadix + d;
    if (tile == 0) {
        store_volatile(mine, kFlagPrefix | count);
    } else {
        store_volatile(mine, kFlagAggregate | count);
    }
    uint32_t exclusive = 0;
    bool ok = true;
    if (tile > 0) {
        int64_t j = static_cast<int64_t>(tile) - 1;
        uint32_t polls = 0;
        while (j >= 0) {
            const uint32_t s = load_volatile(lookback + static_cast<size_t>(j) * kRadix + d);
            const uint32_t flag = s & ~kCountMask;
            if (flag == 0u) {
                if (++polls > poll_limit) {
                    atomicOr(status, kStatusTimeout);
                    ok = false;
                    break;
                }
                continue;
            }
            exclusive += s & kCountMask;
            if (flag == kFlagPrefix) {
                break;
            }
            --j;
        }
        __threadfence();
        store_volatile(mine, kFlagPrefix | ((exclusive + count) & kCountMask));
    }
    s_base[d] = offset + exclusive;

    // Exclusive scan of the tile's digit counts gives each digit's run start:
    // within each warp's 32 digits, then over the warps.
    uint32_t inclusive = count;
#pragma unroll
    for (uint32_t off = 1; off < 32; off <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inclusive, off);
        inclusive += lane >= off ? v : 0u;
    }
    if (lane == 31) {
        s_sums[warp] = inclusive;
    }
    __syncthreads();
    uint32_t earlier = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) {
        earlier += w < warp ? s_sums[w] : 0u;
    }
    s_start[d] = earlier + inclusive - count;
    if (!__syncthreads_and(ok ? 1 : 0)) {
        return false; // a timed-out tile stays unscattered
    }

    // Place keys in shared memory in digit order, then write contiguous runs.
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        if (digit[it] < kRadix) {
            const uint32_t pos =
                s_start[digit[it]] + s_warp[warp * kRadix + digit[it]] + rank[it];
            s_keys[pos] = key[it];
            s_vals[pos] = val[it];
        }
    }
    __syncthreads();
    const uint32_t valid_in_tile = n > base ? min(kSortTile, n - base) : 0u;
    for (uint32_t k = tid; k < valid_in_tile; k += kSortThreads) {
        const unsigned long long kk = s_keys[k];
        const uint32_t dd = static_cast<uint32_t>((kk >> shift) & (kRadix - 1));
        const uint32_t dst = s_base[dd] + (k - s_start[dd]);
        keys_out[dst] = kk;
        vals_out[dst] = s_vals[k];
    }
    return true;
}

// One onesweep pass. CTAs are persistent: each takes tiles by atomic ticket
// (so every tile's predecessors were taken by CTAs that are running or done,
// which publish without waiting on later tiles) until the tiles run out.
__global__ void __launch_bounds__(kSortThreads, 5)
    onesweep_kernel(const unsigned long long *keys_in, const uint32_t *vals_in,
                    unsigned long long *keys_out, uint32_t *vals_out, uint32_t n, uint32_t tiles,
                    uint32_t shift, const uint32_t *__restrict__ offsets, uint32_t *lookback,
                    uint32_t *ticket, unsigned *status, uint32_t poll_limit) {
    extern __shared__ __align__(16) unsigned char smem[];
    SortSpace &space = *reinterpret_cast<SortSpace *>(smem);
    const uint32_t tid = threadIdx.x;
    while (true) {
        if (tid == 0) {
            space.tile = atomicAdd(ticket, 1u);
        }
        for (uint32_t k = tid; k < kWarps * kRadix; k += kSortThreads) {
            space.warp[k] = 0;
        }
        __syncthreads();
        const uint32_t tile = space.tile;
        if (tile >= tiles) {
            return; // uniform: every thread read the same ticket
        }
        if (!sort_one_tile(space, tile, keys_in, vals_in, keys_out, vals_out, n, shift,
                           offsets[tid], lookback, status, poll_limit)) {
            return; // the CTA takes no more tiles
        }
        __syncthreads(); // the next tile reuses the shared arrays
    }
}

// The whole ordering in one cooperative launch: cube, codes and digit
// histograms, eight sort passes and the gather, with a grid barrier between
// phases. An evaluation made of one launch per phase spent 90 us of host time
// on the ordering's launches and clears whatever the size (a 10,000-particle
// evaluation 309 us, of which the walk 117).
struct OrderArgs {
    const double *x, *y, *z, *m;
    uint32_t n, tiles;
    unsigned long long *keys[2];
    uint32_t *perm[2];
    uint32_t *hist;
    uint32_t *lookback; // of all passes
    double *partials;   // 6 per CTA
    double *sorted;
    uint32_t *zeroed;   // words of the construction to zero on the way
    size_t zeroed_words;
    TreeMeta *meta;
    unsigned *barrier;
    unsigned *status;
    SilentStage silent;
    uint32_t poll_limit;
};

struct OrderSpace {
    union {
        SortSpace sort;
        struct {
            unsigned long long table[128];
            uint32_t local[kRadixPasses * kRadix];
        } encode;
    };
};

// TEST: a CTA stays silent at a.silent, and waits end after a.poll_limit polls.
template <bool TEST>
__global__ void __launch_bounds__(kSortThreads, 4) order_kernel(const OrderArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    OrderSpace &space = *reinterpret_cast<OrderSpace *>(smem);
    __shared__ TreeMeta cube;
    __shared__ double ext[6];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t first = blockIdx.x * kSortThreads + tid, stride = gridDim.x * kSortThreads;
    unsigned barriers = 0;
    const uint32_t poll_limit = TEST ? a.poll_limit : kLookbackPollLimit;
    if (TEST && a.silent == SilentStage::ordering_barrier && blockIdx.x == 0 && gridDim.x > 1) {
        return;
    }
    // All CTAs' barrier; false when this CTA is to return, the ordering abandoned.
    auto meet = [&] {
        const bool met = grid_barrier(a.barrier, ++barriers, a.status, poll_limit);
        if (!met && tid == 0) {
            atomicExch(&a.meta->node_count, 0u);
        }
        return met;
    };

    // Nothing reads these words before the first barrier.
    for (size_t k = first; k < static_cast<size_t>(kRadixPasses) * kRadix; k += stride) {
        a.hist[k] = 0u;
    }
    for (size_t k = first; k < static_cast<size_t>(kRadixPasses) * a.tiles * kRadix; k += stride) {
        a.lookback[k] = 0u;
    }
    for (size_t k = first; k < a.zeroed_words; k += stride) {
        a.zeroed[k] = 0u;
    }

    // The extremes: each CTA's, then (after the barrier) all CTAs' folded by
    // every CTA alike (min and max are exact in any order).
    double v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    for (uint32_t i = first; i < a.n; i += stride) {
        min_max(a.x[i], v[0], v[3]);
        min_max(a.y[i], v[1], v[4]);
        min_max(a.z[i], v[2], v[5]);
    }
    double mine = 0.0;
    block_min_max(v, mine);
    if (tid < 6) {
        a.partials[blockIdx.x * 6 + tid] = mine;
    }
    if (!meet()) {
        return;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        v[k] = k < 3 ? INFINITY : -INFINITY;
    }
    for (uint32_t b = tid; b < gridDim.x; b += kSortThreads) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            // Empty CTAs hold (+inf, -inf): lows only lower, highs only raise.
            const double p = __ldcg(a.partials + b * 6 + k);
            v[k] = k < 3 ? (p < v[k] ? p : v[k]) : (v[k] < p ? p : v[k]);
        }
    }
    double folded = 0.0;
    block_min_max(v, folded);
    if (tid < 6) {
        ext[tid] = folded;
    }
    __syncthreads();
    if (tid == 0) {
        cube = TreeMeta{};
        cube.node_count = kNodesUnset;
        write_cube(ext, a.n, &cube);
        if (blockIdx.x == 0) {
            *a.meta = cube; // the other scalars start at zero
        }
    }
    encode_prepare(space.encode.table, space.encode.local);
    __syncthreads();
    encode_particles(a.x, a.y, a.z, a.n, cube, space.encode.table, space.encode.local, a.keys[0],
                     a.perm[0], a.hist);
    if (!meet()) {
        return;
    }

    if (TEST && a.silent == SilentStage::ordering_lookback && blockIdx.x == 0 && gridDim.x > 1) {
        return;
    }
    for (int pass = 0; pass < kRadixPasses; ++pass) {
        const bool odd = (pass & 1) != 0;
        const unsigned long long *keys_in = odd ? a.keys[1] : a.keys[0];
        unsigned long long *keys_out = odd ? a.keys[0] : a.keys[1];
        const uint32_t *perm_in = odd ? a.perm[1] : a.perm[0];
        uint32_t *perm_out = odd ? a.perm[0] : a.perm[1];
        if (blockIdx.x < a.tiles) {
            // Where digit `tid` starts in the output: the exclusive scan of the
            // pass's histogram.
            const uint32_t count = __ldcg(a.hist + pass * kRadix + tid);
            uint32_t inclusive = count;
#pragma unroll
            for (uint32_t off = 1; off < 32; off <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, inclusive, off);
                inclusive += lane >= off ? u : 0u;
            }
            if (lane == 31) {
                space.sort.sums[warp] = inclusive;
            }
            __syncthreads();
            uint32_t offset = inclusive - count;
#pragma unroll
            for (uint32_t w = 0; w < kWarps; ++w) {
                offset += w < warp ? space.sort.sums[w] : 0u;
            }
            // Ascending tiles per CTA: the lowest unfinished tile waits for none.
            for (uint32_t tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
                __syncthreads(); // the previous tile's (or the sums') last readers
                for (uint32_t k = tid; k < kWarps * kRadix; k += kSortThreads) {
                    space.sort.warp[k] = 0;
                }
                __syncthreads();
                if (!sort_one_tile(space.sort, tile, keys_in, perm_in, keys_out, perm_out, a.n,
                                   static_cast<uint32_t>(kRadixBits * pass), offset,
                                   a.lookback + static_cast<size_t>(pass) * a.tiles * kRadix,
                                   a.status, poll_limit)) {
                    if (tid == 0) {
                        atomicExch(&a.meta->node_count, 0u);
                    }
                    return; // the other CTAs' waits run out too
                }
            }
        }
        if (!meet()) {
            return;
        }
    }

    // Eight passes end in buffer 0.
    for (uint32_t i = first; i < a.n; i += stride) {
        const uint32_t j = __ldcg(a.perm[0] + i);
        a.sorted[i] = a.x[j];
        a.sorted[static_cast<size_t>(a.n) + i] = a.y[j];
        a.sorted[2ull * a.n + i] = a.z[j];
        a.sorted[3ull * a.n + i] = a.m[j];
    }
}

size_t onesweep_smem() { return sizeof(SortSpace); }

} // namespace

uint32_t sort_tiles(uint32_t n) { return ceil_div(n == 0 ? 1 : n, kSortTile); }

size_t cube_partials_needed(uint32_t) { return 6ull * kCubeBlocks; }

cudaError_t launch_bounding_cube(const double *x, const double *y, const double *z, uint32_t n,
                                 double *partials, TreeMeta *meta, cudaStream_t stream) {
    cube_kernel<<<kCubeBlocks, kCubeThreads, 0, stream>>>(x, y, z, n, partials, meta);
    return cudaGetLastError();
}

cudaError_t launch_encode(const double *x, const double *y, const double *z, uint32_t n,
                          const TreeMeta *meta, unsigned long long *codes, uint32_t *indices,
                          uint32_t *hist, cudaStream_t stream) {
    const uint32_t blocks = max(1u, min(ceil_div(n, kReduceThreads), kReduceBlocks));
    encode_kernel<<<blocks, kReduceThreads, 0, stream>>>(x, y, z, n, meta, codes, indices, hist);
    return cudaGetLastError();
}

cudaError_t launch_scan_histograms(uint32_t *hist, cudaStream_t stream) {
    scan_histograms_kernel<<<kRadixPasses, kRadix, 0, stream>>>(hist);
    return cudaGetLastError();
}

cudaError_t launch_onesweep(const unsigned long long *keys_in, const uint32_t *vals_in,
                            unsigned long long *keys_out, uint32_t *vals_out, uint32_t n,
                            int pass, const uint32_t *offsets, uint32_t *lookback,
                            uint32_t *ticket, unsigned *status, cudaStream_t stream,
                            uint32_t poll_limit) {
    static_assert(kLookbackPollLimit == kSpinLimit, "one bound for every device wait");
    static std::atomic<uint64_t> configured{0};
    const cudaError_t err = set_smem_limit_once(reinterpret_cast<const void *>(onesweep_kernel),
                                                static_cast<int>(onesweep_smem()), configured);
    if (err != cudaSuccess) {
        return err;
    }
    // Persistent CTAs: as many as fit on the device at once, at most one per tile.
    static std::atomic<int> resident{0};
    if (resident.load(std::memory_order_relaxed) == 0) {
        int per_sm = 0, sms = 0, device = 0;
        cudaError_t e = cudaGetDevice(&device);
        if (e == cudaSuccess) {
            e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        }
        if (e == cudaSuccess) {
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, onesweep_kernel,
                                                              kSortThreads, onesweep_smem());
        }
        if (e != cudaSuccess) {
            return e;
        }
        resident.store(std::max(1, per_sm) * std::max(1, sms), std::memory_order_relaxed);
    }
    const uint32_t tiles = sort_tiles(n);
    const uint32_t grid = std::min(tiles, static_cast<uint32_t>(resident.load()));
    onesweep_kernel<<<grid, kSortThreads, onesweep_smem(), stream>>>(
        keys_in, vals_in, keys_out, vals_out, n, tiles, static_cast<uint32_t>(kRadixBits * pass),
        offsets + pass * kRadix, lookback, ticket, status, poll_limit);
    return cudaGetLastError();
}

cudaError_t cooperative_grid(const void *kernel, int threads, size_t smem,
                             std::atomic<uint64_t> &configured, std::atomic<int> &resident,
                             uint32_t wanted, uint32_t &grid) {
    cudaError_t err = set_smem_limit_once(kernel, static_cast<int>(smem), configured);
    if (err == cudaSuccess && resident.load(std::memory_order_relaxed) == 0) {
        int per_sm = 0, sms = 0, device = 0;
        err = cudaGetDevice(&device);
        if (err == cudaSuccess) {
            err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        }
        if (err == cudaSuccess) {
            err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
        }
        if (err == cudaSuccess) {
            resident.store(std::max(1, per_sm) * std::max(1, sms), std::memory_order_relaxed);
        }
    }
    grid = std::max(1u, std::min(wanted, static_cast<uint32_t>(resident.load())));
    return err;
}

size_t order_partials_needed() { return 6ull * kMaxCooperativeBlocks; }

cudaError_t launch_order(const double *x, const double *y, const double *z, const double *m,
                         uint32_t n, unsigned long long *const *keys, uint32_t *const *perm,
                         uint32_t *hist, uint32_t *lookback, double *partials, double *sorted,
                         uint32_t *zeroed, size_t zeroed_words, TreeMeta *meta,
                         unsigned *barrier, unsigned *status, cudaStream_t stream,
                         SilentStage silent, uint32_t poll_limit) {
    static std::atomic<uint64_t> configured[2];
    static std::atomic<int> resident[2];
    const bool test = silent != SilentStage::none;
    const void *kernel = test ? reinterpret_cast<const void *>(order_kernel<true>)
                              : reinterpret_cast<const void *>(order_kernel<false>);
    const uint32_t tiles = sort_tiles(n);
    uint32_t grid = 0;
    const cudaError_t err =
        cooperative_grid(kernel, kSortThreads, sizeof(OrderSpace), configured[test], resident[test],
                         std::min(std::max(tiles, ceil_div(n, 1024u)), kMaxCooperativeBlocks),
                         grid);
    if (err != cudaSuccess) {
        return err;
    }
    OrderArgs a{x,        y,      z,      m,            n,    tiles,   {keys[0], keys[1]},
                {perm[0], perm[1]}, hist,   lookback,     partials, sorted, zeroed,
                zeroed_words,       meta,   barrier,      status,   silent, poll_limit};
    void *args[] = {&a};
    return cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kSortThreads), args,
                                       sizeof(OrderSpace), stream);
}

} // namespace ob
