// Direct O(N^2) force sum on sm_100a.
//
// Replaces the reference's direct_kernel (src/solvers/cuda_direct_kernel.cu:87-184)
// and the CPU DirectSolver it mirrors (src/solvers/direct_solver.cpp:20-80).
// The force law is the reference's Plummer-softened one,
// a_i = sum_{j != i} m_j d_ij (|d_ij|^2 + eps^2)^{-3/2}
// (include/orrery/core/softening.hpp:83-100), with G = 1.
//
// Layout and schedule (FP32 and split forms):
//   * sources are packed once per evaluation into float4 (x, y, z, m), padded
//     with zero-mass entries to a whole number of tiles;
//   * a CTA owns THREADS*R targets held in registers (R per thread) and walks a
//     contiguous range of source tiles, each 512-particle tile brought into
//     shared memory by one 1-D bulk copy (cp.async.bulk) on an mbarrier,
//     double-buffered so the next tile lands while this one is summed;
//   * every thread reads the same source at the same time, so each float4 read
//     is a shared-memory broadcast amortised over the R targets of the thread;
//   * tiles run a branch-free loop; with softening the target's own entry and
//     the zero-mass padding add exactly zero (self_term_vanishes), and
//     without it the tiles that hold them select zero mass for j == i and
//     j >= n, as the reference kernel masks (cuda_direct_kernel.cu:155-160);
//   * when the targets alone cannot fill 148 SMs evenly, S CTAs split the source
//     range of a target tile. Where the whole grid is resident at once they form
//     a thread-block cluster, whose partial sums are reduced through distributed
//     shared memory; otherwise each leaves its sums in memory and the last to
//     arrive adds them (a cluster waits for as many free slots of one GPC as it
//     has CTAs, which idles SMs once slots free up one by one). Either way the
//     parts are added in order, so the result does not depend on scheduling.
#include <algorithm>
#include <cooperative_groups.h>
#include <iterator>

#include "common.cuh"
#include "f64_math.cuh"
#include "f64_ordered.cuh"
#include "runtime.hpp"
#include "internal.hpp"
#include "split_math.cuh"

namespace cg = cooperative_groups;

namespace ob {
namespace {

struct DirectArgs {
    const float4 *hi;
    const float4 *lo;
    uint32_t n;
    uint32_t padded;
    float eps2;
    double *ax;
    double *ay;
    double *az;
    unsigned *status;
    double *partial;   // sums of the parts (a part is its own CTA, no cluster), or NULL
    unsigned *arrived; // per target tile: parts that have written theirs (zero between launches)
};

// Range of source tiles [tb, te) handled by split rank `rank`.
__device__ __forceinline__ void source_tiles(uint32_t n, uint32_t split, uint32_t rank,
                                             uint32_t &tb, uint32_t &te) {
    const uint32_t tiles = ceil_div(n, kDirectTile);
    const uint32_t per = ceil_div(tiles, split);
    tb = min(rank * per, tiles);
    te = min(tb + per, tiles);
}

// Sources per unrolled step of the tile loop: a thread with a single target
// pair (the shapes for small systems, few warps per SM) gets more independent
// chains to overlap.
template <int P> constexpr int kSourceUnroll = P == 1 ? 4 : 2;

// The same for the FP32 kernel, in pairs of sources per step.
template <int R> constexpr int kPairUnroll = R == 2 ? 4 : 2;
// Threads per SM that the FP32 kernel's registers are held to: 512 at 128
// registers with four targets and more (262,144 targets 26.8 ms; 768 at 80
// 27.4 ms, 1024 at 64 30.2 ms), 1024 at 64 with two.
template <int THREADS, int R> constexpr int kMinBlocksF32 = (R <= 2 ? 1024 : 512) / THREADS;

// Tiles holding the CTA's own targets or padding need no masks when those
// entries add exactly zero. A target's own entry is its packed position, so
// d = 0 exactly and r2 = eps2, and its term is f * 0 = 0 whenever
// f = (m y)(y y) at r2 = eps2 is finite; padded entries (zero mass, at the
// origin) have r2 >= eps2 and give (0 y)(y y) = 0. The masked loop adds f = 0
// for the same entries in the same order, so both loops give the same sums.
// `f_self` is that f for one target, computed as the loop computes it.
__device__ __forceinline__ bool self_term_vanishes(float eps2, float f_self) {
    return eps2 >= 1.17549435e-38f && isfinite(f_self); // eps2 normal: no flush to zero
}

// Source groups. With K > 1 the threads of a CTA form K groups of TP =
// THREADS / K: thread tid serves target lane tid % TP over the sources of
// slice tid / TP of every tile (kDirectTile / K consecutive sources), so a
// small system gets K times the warps. The K partial sums of a target are
// added in slice order, so the result does not depend on scheduling.
template <int THREADS, int K> struct SourceGroups {
    static_assert(THREADS % K == 0 && (THREADS / K) % 32 == 0, "groups are whole warps");
    static_assert(kDirectTile % K == 0, "a tile splits evenly");
    static constexpr uint32_t lanes = THREADS / K;       // target lanes per group
    static constexpr uint32_t sources = kDirectTile / K; // sources per slice of a tile
};


// Adds the parts of a CTA's target tile, whose 3 * bt sums ([component][slot])
// this part holds in shared memory. Kept out of line: inlined, it changes the
// registers the compiler gives the pair loops.
__device__ __noinline__ void add_parts(const DirectArgs &a, uint32_t t0, double *partial,
                                       uint32_t bt) {
    const uint32_t split = gridDim.x, rank = blockIdx.x, tid = threadIdx.x;
    const uint32_t block = 3u * bt; // one part's sums
    if (a.partial != nullptr) {
        __shared__ bool last;
        __syncthreads();
        double *sums = a.partial + static_cast<size_t>(blockIdx.y) * split * block;
        for (uint32_t k = tid; k < block; k += blockDim.x) {
            sums[rank * block + k] = partial[k];
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            last = atomicAdd(&a.arrived[blockIdx.y], 1u) == split - 1u;
        }
        __syncthreads();
        if (!last) {
            return;
        }
        __threadfence();
        for (uint32_t k = tid; k < block; k += blockDim.x) {
            double sum = 0.0;
            for (uint32_t q = 0; q < split; ++q) {
                sum += __ldcg(&sums[q * block + k]);
            }
            const uint32_t i = t0 + k % bt;
            if (i < a.n) {
                (k < bt ? a.ax : k < 2u * bt ? a.ay : a.az)[i] = sum;
            }
        }
        if (tid == 0) {
            a.arrived[blockIdx.y] = 0u; // for the next launch
        }
        return;
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const uint32_t per = bt / split;
    for (uint32_t k = tid; k < per; k += blockDim.x) {
        const uint32_t slot = rank * per + k;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
        for (uint32_t q = 0; q < split; ++q) {
            const double *remote = cluster.map_shared_rank(partial, q);
            s0 += remote[slot];
            s1 += remote[bt + slot];
            s2 += remote[2 * bt + slot];
        }
        const uint32_t i = t0 + slot;
        if (i < a.n) {
            a.ax[i] = s0;
            a.ay[i] = s1;
            a.az[i] = s2;
        }
    }
    cluster.sync();
}

// Writes the CTA's per-target sums, adding the parts' when the sources are
// split. `partial` holds 3*BT sums laid out [component][slot] (one such block
// per group). Target slot r*TP + lane.
template <int THREADS, int R, int K>
__device__ __forceinline__ void finish_targets(const DirectArgs &a, uint32_t t0, double *partial,
                                               const double (&sx)[R], const double (&sy)[R],
                                               const double (&sz)[R]) {
    constexpr uint32_t TP = SourceGroups<THREADS, K>::lanes;
    constexpr uint32_t BT = TP * R;
    const uint32_t split = gridDim.x;
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid % TP;
    const uint32_t group = tid / TP;
    if (K == 1 && split == 1) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t i = t0 + r * THREADS + tid;
            if (i < a.n) {
                a.ax[i] = sx[r];
                a.ay[i] = sy[r];
                a.az[i] = sz[r];
            }
        }
        return;
    }
    if constexpr (K == 1) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t slot = r * THREADS + tid;
            partial[slot] = sx[r];
            partial[BT + slot] = sy[r];
            partial[2 * BT + slot] = sz[r];
        }
    } else {
        // Each group's sums in its own block, then added in group order into
        // block 0 (each slot by one thread, which reads every group's value of
        // a component before it overwrites block 0's).
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t slot = r * TP + lane;
            partial[(group * 3 + 0) * BT + slot] = sx[r];
            partial[(group * 3 + 1) * BT + slot] = sy[r];
            partial[(group * 3 + 2) * BT + slot] = sz[r];
        }
        __syncthreads();
        for (uint32_t slot = tid; slot < BT; slot += THREADS) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double s = 0.0;
#pragma unroll
                for (int g = 0; g < K; ++g) {
                    s += partial[(g * 3 + c) * BT + slot];
                }
                partial[c * BT + slot] = s;
            }
        }
        __syncthreads();
        if (split == 1) {
            for (uint32_t slot = tid; slot < BT; slot += THREADS) {
                const uint32_t i = t0 + slot;
                if (i < a.n) {
                    a.ax[i] = partial[slot];
                    a.ay[i] = partial[BT + slot];
                    a.az[i] = partial[2 * BT + slot];
                }
            }
            return;
        }
    }
    add_parts(a, t0, partial, BT);
}

// Sources of the FP32 kernel are stored in pairs, two float4 per two
// particles: (x0, x1, y0, y1) and (z0, z1, m0, m1), so that each half is already
// a packed FP32x2 operand of two sources; a target's coordinates are held
// twice in registers. (With the values duplicated in memory and pairs of
// targets per instruction, a warp read twice the shared memory per
// interaction, two thirds of what the SM can deliver to four-target threads:
// 262,144 targets took 29.2 ms.)
template <int THREADS, int R, int K>
__global__ void __launch_bounds__(THREADS, kMinBlocksF32<THREADS, R>)
    direct_f32_kernel(const DirectArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr uint32_t TP = SourceGroups<THREADS, K>::lanes;
    constexpr uint32_t JS = SourceGroups<THREADS, K>::sources;
    constexpr uint32_t BT = TP * R;
    float4 *tiles = reinterpret_cast<float4 *>(smem); // 2 buffers x kDirectTile
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + 2 * kDirectTile * sizeof(float4));
    double *partial = reinterpret_cast<double *>(bars + 2);

    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid % TP;
    const uint32_t pb = (tid / TP) * (JS / 2); // this thread's slice of every tile, in pairs
    const uint32_t t0 = blockIdx.y * BT;
    const float2 eps2 = make_float2(a.eps2, a.eps2);

    // Target r is slot r * TP + lane.
    float2 nx[R], ny[R], nz[R], ax[R], ay[R], az[R];
    const float y_self = rsqrt_approx(a.eps2);
    bool vanish = true;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t i = t0 + r * TP + lane;
        const float4 u0 = a.hi[i & ~1u], u1 = a.hi[i | 1u];
        const bool odd = (i & 1u) != 0u;
        const float x = odd ? u0.y : u0.x, y = odd ? u0.w : u0.z, z = odd ? u1.y : u1.x;
        const float m = odd ? u1.w : u1.z;
        nx[r] = make_float2(-x, -x);
        ny[r] = make_float2(-y, -y);
        nz[r] = make_float2(-z, -z);
        ax[r] = ay[r] = az[r] = make_float2(0.0f, 0.0f);
        vanish = vanish && self_term_vanishes(a.eps2, (m * y_self) * (y_self * y_self));
    }

    uint32_t tb, te;
    source_tiles(a.n, gridDim.x, blockIdx.x, tb, te);
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_barrier_init();
    }
    const bool unmasked = __syncthreads_and(vanish ? 1 : 0) != 0;
    constexpr uint32_t tile_bytes = kDirectTile * sizeof(float4);
    auto stage = [&](uint32_t k, uint32_t buf) {
        mbar_arrive_expect_tx(&bars[buf], tile_bytes);
        bulk_copy_g2s(tiles + buf * kDirectTile, a.hi + static_cast<size_t>(k) * kDirectTile,
                      tile_bytes, &bars[buf]);
    };
    if (tid == 0) {
        for (uint32_t k = tb; k < min(tb + 2, te); ++k) {
            stage(k, k - tb);
        }
    }

    bool ok = true;
    for (uint32_t k = tb; k < te; ++k) {
        const uint32_t it = k - tb;
        const uint32_t buf = it & 1u;
        if (ok) {
            ok = mbar_wait_bounded(&bars[buf], (it >> 1) & 1u, a.status);
        }
        if (ok) {
            const float4 *tile = tiles + buf * kDirectTile;
            const uint32_t j0 = k * kDirectTile;
            const bool masked = !unmasked && ((j0 + kDirectTile > a.n) ||
                                              (j0 < t0 + BT && t0 < j0 + kDirectTile));
            if (!masked) {
#pragma unroll(kPairUnroll<R>)
                for (uint32_t p = pb; p < pb + JS / 2; ++p) {
                    const float4 s0 = tile[2 * p];     // (x0, x1, y0, y1)
                    const float4 s1 = tile[2 * p + 1]; // (z0, z1, m0, m1)
                    const float2 sx = make_float2(s0.x, s0.y);
                    const float2 sy = make_float2(s0.z, s0.w);
                    const float2 sz = make_float2(s1.x, s1.y);
                    const float2 sm = make_float2(s1.z, s1.w);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float2 dx = __fadd2_rn(sx, nx[r]);
                        const float2 dy = __fadd2_rn(sy, ny[r]);
                        const float2 dz = __fadd2_rn(sz, nz[r]);
                        float2 r2 = __ffma2_rn(dx, dx, eps2);
                        r2 = __ffma2_rn(dy, dy, r2);
                        r2 = __ffma2_rn(dz, dz, r2);
                        const float2 inv = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
                        const float2 f = __fmul2_rn(__fmul2_rn(sm, inv), __fmul2_rn(inv, inv));
                        ax[r] = __ffma2_rn(f, dx, ax[r]);
                        ay[r] = __ffma2_rn(f, dy, ay[r]);
                        az[r] = __ffma2_rn(f, dz, az[r]);
                    }
                }
            } else {
                for (uint32_t p = pb; p < pb + JS / 2; ++p) {
                    const float4 s0 = tile[2 * p];
                    const float4 s1 = tile[2 * p + 1];
                    const uint32_t j = j0 + 2 * p;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const uint32_t i = t0 + r * TP + lane;
                        const bool skip0 = (j == i) || (j >= a.n);
                        const bool skip1 = (j + 1 == i) || (j + 1 >= a.n);
                        const float2 dx = __fadd2_rn(make_float2(s0.x, s0.y), nx[r]);
                        const float2 dy = __fadd2_rn(make_float2(s0.z, s0.w), ny[r]);
                        const float2 dz = __fadd2_rn(make_float2(s1.x, s1.y), nz[r]);
                        float2 r2 = __ffma2_rn(dx, dx, eps2);
                        r2 = __ffma2_rn(dy, dy, r2);
                        r2 = __ffma2_rn(dz, dz, r2);
                        r2.x = skip0 ? 1.0f : r2.x;
                        r2.y = skip1 ? 1.0f : r2.y;
                        const float2 w = make_float2(skip0 ? 0.0f : s1.z, skip1 ? 0.0f : s1.w);
                        const float2 inv = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
                        const float2 f = __fmul2_rn(__fmul2_rn(w, inv), __fmul2_rn(inv, inv));
                        ax[r] = __ffma2_rn(f, dx, ax[r]);
                        ay[r] = __ffma2_rn(f, dy, ay[r]);
                        az[r] = __ffma2_rn(f, dz, az[r]);
                    }
                }
            }
        }
        __syncthreads();
        if (tid == 0 && ok && k + 2 < te) {
            fence_proxy_async_shared();
            stage(k + 2, buf);
        }
    }

    double sx[R], sy[R], sz[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        sx[r] = static_cast<double>(ax[r].x) + static_cast<double>(ax[r].y);
        sy[r] = static_cast<double>(ay[r].x) + static_cast<double>(ay[r].y);
        sz[r] = static_cast<double>(az[r].x) + static_cast<double>(az[r].y);
    }
    finish_targets<THREADS, R, K>(a, t0, partial, sx, sy, sz);
}

// Split (precision) form: targets r = 2p + h are packed in pairs p and every
// operation is an FP32x2 instruction (split_math.cuh). Tiles carry 512 sources
// of hi and lo parts (64 bytes per source).
template <int THREADS, int R, int K>
__global__ void __launch_bounds__(THREADS) direct_split_kernel(const DirectArgs a) {
    static_assert(R % 2 == 0, "targets are processed in packed pairs");
    constexpr int P = R / 2;
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr uint32_t TP = SourceGroups<THREADS, K>::lanes;
    constexpr uint32_t JS = SourceGroups<THREADS, K>::sources;
    constexpr uint32_t BT = TP * R;
    float4 *tiles_hi = reinterpret_cast<float4 *>(smem);     // 2 buffers x 2*kDirectTile
    float4 *tiles_lo = tiles_hi + 4 * kDirectTile;           // 2 buffers x 2*kDirectTile
    uint64_t *bars = reinterpret_cast<uint64_t *>(tiles_lo + 4 * kDirectTile);
    double *partial = reinterpret_cast<double *>(bars + 2);

    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid % TP;
    const uint32_t jb = (tid / TP) * JS; // this thread's slice of every tile
    const uint32_t t0 = blockIdx.y * BT;
    const float2 eps2 = make_float2(a.eps2, a.eps2);

    SplitTargets tg[P];
    double sx[R], sy[R], sz[R];
    const float2 y_self = refined_rsqrt2(eps2);
    bool vanish = true;
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const size_t i0 = t0 + (2 * p) * TP + lane;
        tg[p] = load_split_targets(a.hi, a.lo, i0, i0 + TP);
        const float2 m = make_float2(a.hi[2 * i0 + 1].z, a.hi[2 * (i0 + TP) + 1].z);
        const float2 f_self = __fmul2_rn(__fmul2_rn(m, y_self), __fmul2_rn(y_self, y_self));
        vanish = vanish && self_term_vanishes(a.eps2, f_self.x) &&
                 self_term_vanishes(a.eps2, f_self.y);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        sx[r] = sy[r] = sz[r] = 0.0;
    }

    uint32_t tb, te;
    source_tiles(a.n, gridDim.x, blockIdx.x, tb, te);
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_barrier_init();
    }
    const bool unmasked = __syncthreads_and(vanish ? 1 : 0) != 0;
    constexpr uint32_t tile_bytes = 2 * kDirectTile * sizeof(float4);
    auto stage = [&](uint32_t k, uint32_t buf) {
        mbar_arrive_expect_tx(&bars[buf], 2 * tile_bytes);
        const size_t off = 2ull * static_cast<size_t>(k) * kDirectTile;
        bulk_copy_g2s(tiles_hi + buf * 2 * kDirectTile, a.hi + off, tile_bytes, &bars[buf]);
        bulk_copy_g2s(tiles_lo + buf * 2 * kDirectTile, a.lo + off, tile_bytes, &bars[buf]);
    };
    if (tid == 0) {
        for (uint32_t k = tb; k < min(tb + 2, te); ++k) {
            stage(k, k - tb);
        }
    }

    bool ok = true;
    for (uint32_t k = tb; k < te; ++k) {
        const uint32_t it = k - tb;
        const uint32_t buf = it & 1u;
        if (ok) {
            ok = mbar_wait_bounded(&bars[buf], (it >> 1) & 1u, a.status);
        }
        if (ok) {
            const float4 *th = tiles_hi + buf * 2 * kDirectTile;
            const float4 *tl = tiles_lo + buf * 2 * kDirectTile;
            const uint32_t j0 = k * kDirectTile;
            const bool masked = !unmasked && ((j0 + kDirectTile > a.n) ||
                                              (j0 < t0 + BT && t0 < j0 + kDirectTile));
            float2 kx[P], ky[P], kz[P], cx[P], cy[P], cz[P];
#pragma unroll
            for (int p = 0; p < P; ++p) {
                kx[p] = ky[p] = kz[p] = cx[p] = cy[p] = cz[p] = make_float2(0.0f, 0.0f);
            }
            if (!masked) {
#pragma unroll(kSourceUnroll<P>)
                for (uint32_t jj = jb; jj < jb + JS; ++jj) {
                    const float4 h0 = th[2 * jj], h1 = th[2 * jj + 1];
                    const float4 l0 = tl[2 * jj], l1 = tl[2 * jj + 1];
#pragma unroll
                    for (int p = 0; p < P; ++p) {
                        float2 dx, dy, dz;
                        split_offsets(tg[p], h0, h1, l0, l1, dx, dy, dz);
                        const float2 r2 =
                            __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, eps2)));
                        const float2 y = refined_rsqrt2(r2);
                        const float2 f = __fmul2_rn(__fmul2_rn(pair_high(h1), y), __fmul2_rn(y, y));
                        kahan2(kx[p], cx[p], f, dx);
                        kahan2(ky[p], cy[p], f, dy);
                        kahan2(kz[p], cz[p], f, dz);
                    }
                }
            } else {
                for (uint32_t jj = jb; jj < jb + JS; ++jj) {
                    const float4 h0 = th[2 * jj], h1 = th[2 * jj + 1];
                    const float4 l0 = tl[2 * jj], l1 = tl[2 * jj + 1];
                    const uint32_t j = j0 + jj;
#pragma unroll
                    for (int p = 0; p < P; ++p) {
                        const uint32_t i0 = t0 + (2 * p) * TP + lane;
                        const bool skip0 = (j == i0) || (j >= a.n);
                        const bool skip1 = (j == i0 + TP) || (j >= a.n);
                        float2 dx, dy, dz;
                        split_offsets(tg[p], h0, h1, l0, l1, dx, dy, dz);
                        float2 r2 =
                            __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, eps2)));
                        r2 = make_float2(skip0 ? 1.0f : r2.x, skip1 ? 1.0f : r2.y);
                        const float2 w = make_float2(skip0 ? 0.0f : h1.z, skip1 ? 0.0f : h1.w);
                        const float2 y = refined_rsqrt2(r2);
                        const float2 f = __fmul2_rn(__fmul2_rn(w, y), __fmul2_rn(y, y));
                        kahan2(kx[p], cx[p], f, dx);
                        kahan2(ky[p], cy[p], f, dy);
                        kahan2(kz[p], cz[p], f, dz);
                    }
                }
            }
            // Fold the tile's compensated FP32 partials into FP64.
#pragma unroll
            for (int p = 0; p < P; ++p) {
                sx[2 * p] += static_cast<double>(kx[p].x) + static_cast<double>(cx[p].x);
                sx[2 * p + 1] += static_cast<double>(kx[p].y) + static_cast<double>(cx[p].y);
                sy[2 * p] += static_cast<double>(ky[p].x) + static_cast<double>(cy[p].x);
                sy[2 * p + 1] += static_cast<double>(ky[p].y) + static_cast<double>(cy[p].y);
                sz[2 * p] += static_cast<double>(kz[p].x) + static_cast<double>(cz[p].x);
                sz[2 * p + 1] += static_cast<double>(kz[p].y) + static_cast<double>(cz[p].y);
            }
        }
        __syncthreads();
        if (tid == 0 && ok && k + 2 < te) {
            fence_proxy_async_shared();
            stage(k + 2, buf);
        }
    }
    finish_targets<THREADS, R, K>(a, t0, partial, sx, sy, sz);
}

// FP64 direct sum in the order of accumulate_range_scalar
// (src/solvers/direct_kernel_scalar.cpp:31-59) with the split at i of
// DirectSolver::evaluate (src/solvers/direct_solver.cpp:49-56): every operation
// is an explicitly rounded FP64 intrinsic, so nothing is contracted and the
// result is bit-identical to the reference's scalar kernel. The terms of a
// target are formed by many warps and added in index order (f64_ordered.cuh).
struct ForceTerm {
    static constexpr int components = 3;
    static constexpr int warps = 16; // 4,096 targets: 78 us, with 8 warps 89 us
    static __device__ __forceinline__ void form(double m, double inv, double dx, double dy,
                                                double dz, double (&term)[3]) {
        const double f = __dmul_rn(m, __dmul_rn(__dmul_rn(inv, inv), inv));
        term[0] = __dmul_rn(f, dx);
        term[1] = __dmul_rn(f, dy);
        term[2] = __dmul_rn(f, dz);
    }
};

__global__ void __launch_bounds__(OrderedShape<ForceTerm>::threads)
    direct_f64_kernel(const double *__restrict__ x, const double *__restrict__ y,
                      const double *__restrict__ z, const double *__restrict__ m, uint32_t n,
                      double eps2, double *ax, double *ay, double *az) {
    extern __shared__ __align__(16) unsigned char smem[];
    auto &space = *reinterpret_cast<OrderedSpace<ForceTerm> *>(smem);
    const uint32_t own = blockIdx.x; // the chunk that holds this CTA's targets
    const uint32_t lane = threadIdx.x & 31u;
    double before = 0.0, sum = 0.0; // sources before the target, then after it
    ordered_terms<ForceTerm>(
        space, x, y, z, m, n, eps2, own, 0u,
        [&](uint32_t chunk, uint32_t count, const double2 *terms) {
            if (chunk != own) {
                add_chunk(sum, terms, count);
                return;
            }
            for (uint32_t k = 0; k < count; ++k) {
                const double t = chunk_term(terms, k);
                if (k == lane) {
                    before = sum;
                    sum = 0.0;
                } else {
                    sum = __dadd_rn(sum, t);
                }
            }
        });
    const uint32_t component = threadIdx.x >> 5;
    const uint32_t i = own * kOrderedTargets + lane;
    if (component < 3u && i < n) {
        (component == 0u ? ax : component == 1u ? ay : az)[i] = __dadd_rn(before, sum);
    }
}

// The same sums with one target per thread and no exchange between warps, for
// systems large enough to give every SM sub-partition a warp: the terms of
// kAhead sources are formed side by side, so that their dependent chains
// overlap, and added in index order. Each warp stages its own sources.
constexpr uint32_t kAhead = 4;
constexpr uint32_t kWideThreads = 64;
// From here on one target per thread: past two full waves of the other kernel's
// CTAs (three of 32 targets per SM, 148 SMs). With the terms formed by many warps,
// and one target per thread, an evaluation took 242 and 482 us at 8,192 targets,
// 904 and 958 us at 16,384, 1.62 and 1.93 ms at 23,680, 2.31 ms both at 28,416, 2.82
// and 2.44 ms at 30,000 (a third wave; shared memory carries 48 bytes per pair),
// 12.1 and 10.0 ms at 65,536. The former single kernel (one target per thread, the
// general root and division, 128-thread CTAs): 731 us at 4,096, 2.91 ms at 16,384,
// 15.3 ms at 65,536.
constexpr uint32_t kWideFrom = 2 * 3 * 148 * 32 + 1;

__global__ void __launch_bounds__(kWideThreads)
    direct_f64_wide_kernel(const double *__restrict__ x, const double *__restrict__ y,
                           const double *__restrict__ z, const double *__restrict__ m, uint32_t n,
                           double eps2, double *ax, double *ay, double *az) {
    __shared__ double staged[kWideThreads / 32][2][4][32];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t own = blockIdx.x * (kWideThreads / 32) + (threadIdx.x >> 5); // targets' chunk
    const uint32_t i = own * 32u + lane;
    if (own * 32u >= n) {
        return; // the whole warp lies past the last target; warps do not wait on one another
    }
    double(*tile)[4][32] = staged[threadIdx.x >> 5];
    const double px = i < n ? x[i] : 0.0, py = i < n ? y[i] : 0.0, pz = i < n ? z[i] : 0.0;
    double bx = 0.0, by = 0.0, bz = 0.0; // sources before i
    double sx = 0.0, sy = 0.0, sz = 0.0; // sources after the last reset
    const uint32_t chunks = (n + 31u) / 32u;
    double next[4] = {0.0, 0.0, 0.0, 0.0};
    auto fetch = [&](uint32_t chunk) {
        const uint32_t j = chunk * 32u + lane;
        const bool real = chunk < chunks && j < n;
        next[0] = real ? x[j] : 0.0;
        next[1] = real ? y[j] : 0.0;
        next[2] = real ? z[j] : 0.0;
        next[3] = real ? m[j] : 0.0;
    };
    fetch(0u);
    for (uint32_t c = 0; c < chunks; ++c) {
        double(*src)[32] = tile[c & 1u];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            src[a][lane] = next[a];
        }
        __syncwarp();
        fetch(c + 1u);
        const uint32_t count = min(32u, n - c * 32u);
        const uint32_t groups = count / kAhead * kAhead;
        auto one = [&](uint32_t k) {
            const double dx = __dsub_rn(src[0][k], px);
            const double dy = __dsub_rn(src[1][k], py);
            const double dz = __dsub_rn(src[2][k], pz);
            const double r2 = __dadd_rn(
                __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)),
                eps2);
            double t[3];
            ForceTerm::form(src[3][k], inverse_root(r2), dx, dy, dz, t);
            if (c == own && k == lane) { // the target itself: the sums start again
                bx = sx;
                by = sy;
                bz = sz;
                sx = sy = sz = 0.0;
            } else {
                sx = __dadd_rn(sx, t[0]);
                sy = __dadd_rn(sy, t[1]);
                sz = __dadd_rn(sz, t[2]);
            }
        };
        if (c == own) {
            for (uint32_t k = 0; k < count; ++k) {
                one(k);
            }
            continue;
        }
        for (uint32_t k0 = 0; k0 < groups; k0 += kAhead) {
            double dx[kAhead], dy[kAhead], dz[kAhead], r2[kAhead], inv[kAhead];
            bool in_range = true;
#pragma unroll
            for (uint32_t k = 0; k < kAhead; ++k) {
                dx[k] = __dsub_rn(src[0][k0 + k], px);
                dy[k] = __dsub_rn(src[1][k0 + k], py);
                dz[k] = __dsub_rn(src[2][k0 + k], pz);
                r2[k] = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx[k], dx[k]),
                                                      __dmul_rn(dy[k], dy[k])),
                                            __dmul_rn(dz[k], dz[k])),
                                  eps2);
                in_range = in_range && inverse_root_in_range(r2[k]);
            }
            if (__all_sync(0xffffffffu, in_range)) {
#pragma unroll
                for (uint32_t k = 0; k < kAhead; ++k) {
                    inv[k] = inverse_root_in_range_rn(r2[k]);
                }
            } else {
#pragma unroll
                for (uint32_t k = 0; k < kAhead; ++k) {
                    inv[k] = inverse_root_general(r2[k]);
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < kAhead; ++k) {
                double t[3];
                ForceTerm::form(src[3][k0 + k], inv[k], dx[k], dy[k], dz[k], t);
                sx = __dadd_rn(sx, t[0]);
                sy = __dadd_rn(sy, t[1]);
                sz = __dadd_rn(sz, t[2]);
            }
        }
        for (uint32_t k = groups; k < count; ++k) {
            one(k);
        }
    }
    if (i < n) {
        ax[i] = __dadd_rn(bx, sx);
        ay[i] = __dadd_rn(by, sy);
        az[i] = __dadd_rn(bz, sz);
    }
}

// Packs FP64 SoA into the split form's source layout: two float4 per particle,
// (x, x, y, y) and (z, z, m, m) rounded to FP32 in hi, and (x', x', y', y') and
// (z', z', 0, 0) with x' = x - FP32(x) in lo.
__global__ void pack_split_kernel(const double *__restrict__ x, const double *__restrict__ y,
                                  const double *__restrict__ z, const double *__restrict__ m,
                                  uint32_t n, uint32_t padded, float4 *hi, float4 *lo) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < padded;
         i += gridDim.x * blockDim.x) {
        const bool real = i < n;
        const double X = real ? x[i] : 0.0, Y = real ? y[i] : 0.0, Z = real ? z[i] : 0.0;
        const float hx = __double2float_rn(X);
        const float hy = __double2float_rn(Y);
        const float hz = __double2float_rn(Z);
        const float hm = real ? __double2float_rn(m[i]) : 0.0f;
        hi[2ull * i] = make_float4(hx, hx, hy, hy);
        hi[2ull * i + 1] = make_float4(hz, hz, hm, hm);
        // X - hx is exact in FP64; rounding it gives the low part.
        const float lx = __double2float_rn(X - static_cast<double>(hx));
        const float ly = __double2float_rn(Y - static_cast<double>(hy));
        const float lz = __double2float_rn(Z - static_cast<double>(hz));
        lo[2ull * i] = make_float4(lx, lx, ly, ly);
        lo[2ull * i + 1] = make_float4(lz, lz, 0.0f, 0.0f);
    }
}

// Packs FP64 SoA into the FP32 kernel's pairs, two float4 per two particles:
// (x0, x1, y0, y1) and (z0, z1, m0, m1); `padded` is even.
__global__ void pack_pairs_kernel(const double *__restrict__ x, const double *__restrict__ y,
                                  const double *__restrict__ z, const double *__restrict__ m,
                                  uint32_t n, uint32_t padded, float4 *pairs) {
    for (uint32_t i = 2u * (blockIdx.x * blockDim.x + threadIdx.x); i < padded;
         i += 2u * gridDim.x * blockDim.x) {
        const bool a = i < n, b = i + 1u < n;
        pairs[i] = make_float4(a ? __double2float_rn(x[i]) : 0.0f,
                               b ? __double2float_rn(x[i + 1u]) : 0.0f,
                               a ? __double2float_rn(y[i]) : 0.0f,
                               b ? __double2float_rn(y[i + 1u]) : 0.0f);
        pairs[i + 1u] = make_float4(a ? __double2float_rn(z[i]) : 0.0f,
                                    b ? __double2float_rn(z[i + 1u]) : 0.0f,
                                    a ? __double2float_rn(m[i]) : 0.0f,
                                    b ? __double2float_rn(m[i + 1u]) : 0.0f);
    }
}

template <int THREADS, int R, int K, bool SPLIT> size_t direct_smem_bytes() {
    const size_t tiles = (SPLIT ? 8 : 2) * kDirectTile * sizeof(float4);
    // 3 sums per target: THREADS * R / K targets, one block per group.
    const size_t partial = 3 * THREADS * R * sizeof(double);
    return tiles + 2 * sizeof(uint64_t) + partial;
}

template <int THREADS, int R, int K, bool SPLIT> auto direct_kernel_for() {
    if constexpr (SPLIT) {
        return direct_split_kernel<THREADS, R, K>;
    } else {
        return direct_f32_kernel<THREADS, R, K>;
    }
}

template <int THREADS, int R, int K, bool SPLIT>
cudaError_t launch_direct_t(const DirectArgs &args, int split, cudaStream_t stream) {
    const uint32_t bt = SourceGroups<THREADS, K>::lanes * R;
    const dim3 grid(static_cast<unsigned>(split), ceil_div(args.n, bt), 1);
    const size_t smem = direct_smem_bytes<THREADS, R, K, SPLIT>();
    auto kernel = direct_kernel_for<THREADS, R, K, SPLIT>();
    // Set once per device, on the first launch there (before any graph
    // capture reaches it: solvers evaluate once before they capture).
    static std::atomic<uint64_t> configured{0};
    const cudaError_t err = set_smem_limit_once(reinterpret_cast<const void *>(kernel),
                                                static_cast<int>(smem), configured);
    if (err != cudaSuccess) {
        return err;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = args.partial != nullptr ? 1u : static_cast<unsigned>(split);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args);
}

template <bool SPLIT>
cudaError_t dispatch_direct(const DirectArgs &args, const DirectConfig &c, cudaStream_t stream) {
#define OB_DIRECT_CASE(T, RR, KK)                                                                  \
    if (c.threads == T && c.targets_per_thread == RR && c.groups == KK)                            \
        return launch_direct_t<T, RR, KK, SPLIT>(args, c.split, stream);
    OB_DIRECT_CASE(64, 2, 1)
    OB_DIRECT_CASE(64, 4, 1)
    OB_DIRECT_CASE(128, 2, 1)
    OB_DIRECT_CASE(128, 4, 1)
    OB_DIRECT_CASE(256, 2, 1)
    OB_DIRECT_CASE(256, 4, 1)
    OB_DIRECT_CASE(128, 2, 2)
    OB_DIRECT_CASE(128, 2, 4)
    OB_DIRECT_CASE(256, 2, 4)
    OB_DIRECT_CASE(256, 2, 8)
    OB_DIRECT_CASE(256, 4, 4)
    OB_DIRECT_CASE(256, 4, 8)
    if constexpr (!SPLIT) {
        OB_DIRECT_CASE(128, 8, 1)
        OB_DIRECT_CASE(256, 8, 1)
    }
#undef OB_DIRECT_CASE
    return cudaErrorInvalidValue;
}

uint32_t targets_per_cta(const DirectConfig &c) {
    return static_cast<uint32_t>(c.threads * c.targets_per_thread / c.groups);
}

} // namespace

// Sums of all parts, were they to meet in memory.
static size_t parts_doubles(uint32_t n, const DirectConfig &c) {
    const uint32_t bt = targets_per_cta(c);
    return 3ull * bt * ceil_div(n, bt) * static_cast<size_t>(c.split);
}

bool direct_uses_cluster(uint32_t n, const DirectConfig &c) {
    // The parts fit a portable cluster, and either the grid fits the SMs at two
    // CTAs each or the sums would take more memory than parts may.
    const bool portable = c.split == 1 || c.split == 2 || c.split == 4 || c.split == 8;
    const uint64_t ctas = static_cast<uint64_t>(ceil_div(n, targets_per_cta(c))) *
                          static_cast<uint64_t>(c.split);
    return portable && (c.split == 1 || ctas <= 2u * 148u ||
                        parts_doubles(n, c) * sizeof(double) > kDirectPartsBytes);
}

size_t direct_partial_doubles(uint32_t n, const DirectConfig &c) {
    return direct_uses_cluster(n, c) ? 0 : parts_doubles(n, c);
}

size_t direct_arrival_words(uint32_t n, const DirectConfig &c) {
    return direct_uses_cluster(n, c) ? 0 : ceil_div(n, targets_per_cta(c));
}

uint32_t direct_padded_count(uint32_t n, const DirectConfig &config) {
    const uint32_t bt = targets_per_cta(config);
    const uint32_t unit = bt > kDirectTile ? bt : kDirectTile;
    const uint32_t padded = ceil_div(n, unit) * unit;
    return padded == 0 ? unit : padded;
}

cudaError_t pack_sources(const double *x, const double *y, const double *z, const double *m,
                         uint32_t n, uint32_t padded, float4 *hi, float4 *lo,
                         cudaStream_t stream) {
    if (padded == 0) {
        return cudaSuccess;
    }
    const uint32_t threads = 256;
    if (lo != nullptr) {
        const uint32_t blocks = min(ceil_div(padded, threads), 148u * 16u);
        pack_split_kernel<<<blocks, threads, 0, stream>>>(x, y, z, m, n, padded, hi, lo);
    } else {
        const uint32_t blocks = min(ceil_div(padded / 2u, threads), 148u * 16u);
        pack_pairs_kernel<<<blocks, threads, 0, stream>>>(x, y, z, m, n, padded, hi);
    }
    return cudaGetLastError();
}

cudaError_t launch_direct_f32(const float4 *sources, uint32_t n, uint32_t padded, float eps2,
                              double *ax, double *ay, double *az, const DirectConfig &config,
                              const DirectParts &parts, unsigned *status, cudaStream_t stream) {
    if (n == 0) {
        return cudaSuccess;
    }
    const bool cluster = direct_uses_cluster(n, config);
    if (config.split < 1 || padded < direct_padded_count(n, config) ||
        (!cluster && (parts.sums == nullptr || parts.arrived == nullptr))) {
        return cudaErrorInvalidValue;
    }
    const DirectArgs args{sources, nullptr, n, padded, eps2, ax, ay, az, status,
                          cluster ? nullptr : parts.sums, parts.arrived};
    return dispatch_direct<false>(args, config, stream);
}

cudaError_t launch_direct_split(const float4 *hi, const float4 *lo, uint32_t n, uint32_t padded,
                                float eps2, double *ax, double *ay, double *az,
                                const DirectConfig &config, const DirectParts &parts,
                                unsigned *status, cudaStream_t stream) {
    if (n == 0) {
        return cudaSuccess;
    }
    const bool cluster = direct_uses_cluster(n, config);
    if (config.split < 1 || padded < direct_padded_count(n, config) ||
        (!cluster && (parts.sums == nullptr || parts.arrived == nullptr))) {
        return cudaErrorInvalidValue;
    }
    const DirectArgs args{hi, lo, n, padded, eps2, ax, ay, az, status,
                          cluster ? nullptr : parts.sums, parts.arrived};
    return dispatch_direct<true>(args, config, stream);
}

cudaError_t launch_direct_f64(const double *x, const double *y, const double *z, const double *m,
                              uint32_t n, double eps2, double *ax, double *ay, double *az,
                              cudaStream_t stream) {
    if (n == 0) {
        return cudaSuccess;
    }
    if (n >= kWideFrom) {
        direct_f64_wide_kernel<<<ceil_div(n, kWideThreads), kWideThreads, 0, stream>>>(
            x, y, z, m, n, eps2, ax, ay, az);
        return cudaGetLastError();
    }
    static std::atomic<uint64_t> configured{0};
    constexpr size_t smem = sizeof(OrderedSpace<ForceTerm>); // above the static 48 KB
    const cudaError_t err =
        set_smem_limit_once(reinterpret_cast<const void *>(direct_f64_kernel),
                            static_cast<int>(smem), configured);
    if (err != cudaSuccess) {
        return err;
    }
    direct_f64_kernel<<<ceil_div(n, kOrderedTargets), OrderedShape<ForceTerm>::threads, smem,
                        stream>>>(x, y, z, m, n, eps2, ax, ay, az);
    return cudaGetLastError();
}

// The shapes and parts among which direct_default_config chooses.
struct DefaultShape {
    int targets, groups;
    double per_pair; // cost per pair beside the cheapest one
};
struct DefaultShapes {
    const DefaultShape *shapes;
    int count;
};
constexpr int kDefaultThreads = 256;
static const int kDefaultParts[] = {1, 2, 4, 8, 3, 5, 6, 10, 12, 16, 24, 32};

static DefaultShapes default_shapes(bool split) {
    static const DefaultShape fp32_shapes[] = {{4, 8, 1.0}, {2, 8, 1.01}};
    static const DefaultShape split_shapes[] = {{4, 8, 1.0}, {4, 4, 0.985}, {2, 8, 1.06}};
    return split ? DefaultShapes{split_shapes, 3} : DefaultShapes{fp32_shapes, 2};
}

int direct_candidates(bool split, DirectConfig *out, int capacity) {
    // (threads, targets per thread, source groups). 64-thread CTAs and source
    // groups give small systems (a few thousand particles) enough warps to
    // occupy the SMs.
    static const int split_shapes[][3] = {{64, 2, 1},  {64, 4, 1},  {128, 2, 1}, {128, 4, 1},
                                          {256, 2, 1}, {256, 4, 1}, {128, 2, 2}, {128, 2, 4},
                                          {256, 2, 4}, {256, 2, 8}, {256, 4, 4}, {256, 4, 8}};
    static const int fp32_shapes[][3] = {{64, 2, 1},  {64, 4, 1},  {128, 2, 1}, {128, 4, 1},
                                         {128, 8, 1}, {256, 2, 1}, {256, 4, 1}, {256, 8, 1},
                                         {128, 2, 2}, {128, 2, 4}, {256, 2, 4}, {256, 2, 8},
                                         {256, 4, 4}, {256, 4, 8}};
    const int(*shapes)[3] = split ? split_shapes : fp32_shapes;
    const int shape_count = split ? 12 : 14;
    static const int splits[] = {1, 2, 4, 8};
    int count = 0;
    auto add = [&](int threads, int targets, int parts, int groups) {
        if (count < capacity) {
            out[count] = DirectConfig{threads, targets, parts, groups};
        }
        ++count;
    };
    for (int s = 0; s < shape_count; ++s) {
        for (const int parts : splits) {
            add(shapes[s][0], shapes[s][1], parts, shapes[s][2]);
        }
    }
    // The other parts that the default rule takes, with the shapes that it takes.
    const DefaultShapes rule = default_shapes(split);
    for (int s = 0; s < rule.count; ++s) {
        for (const int parts : kDefaultParts) {
            if (std::find(std::begin(splits), std::end(splits), parts) == std::end(splits)) {
                add(kDefaultThreads, rule.shapes[s].targets, parts, rule.shapes[s].groups);
            }
        }
    }
    return count;
}

// Estimated time of a shape, in units of one target against one tile of
// sources on one SM: the CTAs that an SM gets (half a one more than the mean,
// for the uneven end, where an SM is left with one of its two), times a CTA's
// work and its start and end, times what the shape costs per pair beside
// the cheapest one.
static double direct_cost(const DirectConfig &c, double per_pair, uint32_t n, uint32_t sms) {
    const uint32_t bt = targets_per_cta(c);
    const uint32_t tiles = ceil_div(n, kDirectTile);
    const auto parts = static_cast<uint32_t>(c.split);
    const uint64_t ctas = static_cast<uint64_t>(ceil_div(n, bt)) * parts;
    const bool alone = ctas <= sms; // one CTA per SM at most
    const double per_sm =
        alone ? 1.0 : ctas <= 2ull * sms ? 2.0 : static_cast<double>(ctas) / sms + 0.5;
    double cost = per_pair * per_sm * bt * (ceil_div(tiles, parts) + 0.15);
    if (alone) { // a CTA alone on its SM hides less latency
        cost /= c.targets_per_thread == 2 ? 0.83 : 0.95;
    }
    return cost;
}

DirectConfig direct_default_config(uint32_t n, bool split, int sm_count) {
    // The cheapest of a few 256-thread shapes by the estimate above, whose
    // constants are fitted to sweeps from 1,000 to 262,144 particles on B200.
    // What decides is how evenly the CTAs fill the SMs: with one cluster rule
    // for all sizes (parts until about four CTAs per SM) FP32 sums of 20,011,
    // 40,000 and 65,536 particles took 222, 862 and 1,931 us, now 179, 674 and
    // 1,737; split sums of 10,007 and 65,536 178 us and 5.0 ms, now 127 us and
    // 4.2 ms.
    const uint32_t sms = static_cast<uint32_t>(sm_count > 0 ? sm_count : 148);
    const DefaultShapes rule = default_shapes(split);
    DirectConfig best;
    double best_cost = 0.0;
    for (int k = 0; k < rule.count; ++k) {
        for (const int parts : kDefaultParts) {
            if (parts > 1 && static_cast<uint32_t>(parts) > ceil_div(n, kDirectTile)) {
                continue;
            }
            DirectConfig c;
            c.threads = kDefaultThreads;
            c.targets_per_thread = rule.shapes[k].targets;
            c.groups = rule.shapes[k].groups;
            c.split = parts;
            if (parts_doubles(n, c) * sizeof(double) > kDirectPartsBytes) {
                continue; // a large system gains nothing from parts
            }
            const double cost = direct_cost(c, rule.shapes[k].per_pair, n, sms);
            if (best_cost == 0.0 || cost < best_cost) {
                best = c;
                best_cost = cost;
            }
        }
    }
    return best;
}

} // namespace ob
