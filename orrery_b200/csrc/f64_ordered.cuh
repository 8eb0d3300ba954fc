// FP64 sums over all sources in index order, bit-identical to a sequential
// loop, with the terms formed in parallel.
//
// A target's sum has one fixed order, but its terms (a square root, a division
// and about twenty more FP64 operations each) do not depend on one another. A
// CTA owns 32 targets (one per lane) and walks the sources in chunks of 32:
// eight or sixteen term warps form the chunk's terms, four or two sources each
// for all 32 targets, and leave them in shared memory; one adder warp per component adds
// the previous chunk's terms meanwhile, in index order, one target per lane.
// Terms and sources are buffered so that a chunk costs one barrier.
//
// Why this split: one thread per target leaves the GPU idle below a few tens
// of thousands of targets and waits on each term's dependent chain (4,096
// targets: 32 CTAs, 734 us; potential energy of 32,768: 5.7 ms). Here the chain
// per source is one FP64 addition: 4,096 targets 77 us, potential 1.0 ms. What
// bounds it: at one CTA per SM the latency of a chunk (4,096 targets, 16 term
// warps: the FP64 pipe is 42 % busy, issue slots 58 %), at several the shared
// memory that carries the terms.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "f64_math.cuh"

namespace ob {

constexpr uint32_t kOrderedTargets = 32; // per CTA, one per lane
constexpr uint32_t kOrderedChunk = 32;   // sources per chunk
// Chunks of sources in shared memory; a chunk is asked for kSourceAhead chunks
// early (an iteration is shorter than the latency of L2).
constexpr uint32_t kSourceRing = 8;
constexpr uint32_t kSourceAhead = 6;
static_assert(kOrderedTargets == kOrderedChunk, "a CTA's targets are one chunk of sources");

template <typename Term> struct OrderedShape {
    static_assert(Term::warps * 32 >= 4 * kOrderedChunk, "the term warps load a chunk in one go");
    static_assert(kOrderedChunk % (2 * Term::warps) == 0, "a term warp takes whole pairs");
    static constexpr uint32_t threads = 32u * (Term::components + Term::warps);
};

template <typename Term> struct __align__(16) OrderedSpace {
    // Terms of sources 2k, 2k + 1 of a chunk for each component and target.
    double2 terms[2][Term::components][kOrderedChunk / 2][kOrderedTargets];
    double sources[kSourceRing][4][kOrderedChunk]; // x, y, z, m of chunk c in slot c % ring
};

// Eight bytes global -> shared, asynchronously, or zeros when `real` is false.
__device__ __forceinline__ void async_copy_8(double *dst, const double *src, bool real) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(real ? 8u : 0u)
                 : "memory");
}

// Term k of a chunk for this lane's target.
__device__ __forceinline__ double chunk_term(const double2 *terms, uint32_t k) {
    const double2 t = terms[(k >> 1) * kOrderedTargets];
    return (k & 1u) != 0u ? t.y : t.x;
}

// Adds the first `count` terms of a chunk in order.
__device__ __forceinline__ void add_chunk(double &sum, const double2 *terms, uint32_t count) {
    if (count == kOrderedChunk) {
#pragma unroll 8
        for (uint32_t p = 0; p < kOrderedChunk / 2; ++p) {
            const double2 t = terms[p * kOrderedTargets];
            sum = __dadd_rn(__dadd_rn(sum, t.x), t.y);
        }
    } else {
        for (uint32_t k = 0; k < count; ++k) {
            sum = __dadd_rn(sum, chunk_term(terms, k));
        }
    }
}

// Forms the terms of this CTA's targets (those of chunk `own`) with the chunks
// from `first` on and calls add(chunk, sources in it, this lane's terms) for
// each, in order, in the adder warps (warp c adds component c).
template <typename Term, typename Add>
__device__ __forceinline__ void ordered_terms(OrderedSpace<Term> &space,
                                              const double *__restrict__ x,
                                              const double *__restrict__ y,
                                              const double *__restrict__ z,
                                              const double *__restrict__ m, uint32_t n,
                                              double eps2, uint32_t own, uint32_t first, Add add) {
    constexpr uint32_t C = Term::components;
    constexpr uint32_t kTermSources = kOrderedChunk / Term::warps; // per term warp and chunk
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t chunks = (n + kOrderedChunk - 1u) / kOrderedChunk;
    const bool adder = warp < C;
    const uint32_t i = own * kOrderedTargets + lane;
    const uint32_t tid = threadIdx.x - 32u * C; // among the term warps
    // Term threads 0..127 each fetch one value of a chunk.
    const bool fetches = !adder && tid < 4u * kOrderedChunk;
    const uint32_t which = fetches ? tid / kOrderedChunk : 0u;
    const uint32_t slot = tid % kOrderedChunk;
    const double *array = which == 0u ? x : which == 1u ? y : which == 2u ? z : m;
    auto fetch = [&](uint32_t chunk) { // one group per call, whether it copies or not
        if (fetches && chunk < chunks) {
            const uint32_t j = chunk * kOrderedChunk + slot;
            async_copy_8(&space.sources[chunk % kSourceRing][which][slot], array + min(j, n - 1u),
                         j < n);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double px = 0.0, py = 0.0, pz = 0.0;
    if (!adder && i < n) {
        px = x[i];
        py = y[i];
        pz = z[i];
    }
    for (uint32_t c = first; c < first + kSourceAhead; ++c) {
        fetch(c);
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(kSourceAhead - 1) : "memory");
    __syncthreads();
    // Iteration c forms chunk c's terms, adds chunk c - 1's and asks for the
    // sources of chunk c + kSourceAhead (whose slot was read two iterations ago).
    for (uint32_t c = first; c <= chunks; ++c) {
        if (adder) {
            if (c > first) {
                const uint32_t count = min(kOrderedChunk, n - (c - 1u) * kOrderedChunk);
                add(c - 1u, count, &space.terms[(c - 1u) & 1u][warp][0][lane]);
            }
        } else if (c < chunks) {
            fetch(c + kSourceAhead);
            const double(*src)[kOrderedChunk] = space.sources[c % kSourceRing];
            const uint32_t k0 = (warp - C) * kTermSources;
            double dx[kTermSources], dy[kTermSources], dz[kTermSources], r2[kTermSources];
            bool in_range = true;
#pragma unroll
            for (uint32_t k = 0; k < kTermSources; ++k) {
                dx[k] = __dsub_rn(src[0][k0 + k], px);
                dy[k] = __dsub_rn(src[1][k0 + k], py);
                dz[k] = __dsub_rn(src[2][k0 + k], pz);
                // core::squared_norm, then the softening.
                r2[k] = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx[k], dx[k]),
                                                      __dmul_rn(dy[k], dy[k])),
                                            __dmul_rn(dz[k], dz[k])),
                                  eps2);
                in_range = in_range && inverse_root_in_range(r2[k]);
            }
            // The short root and division, unless a lane has an argument
            // outside their range.
            double inv[kTermSources];
            if (__all_sync(0xffffffffu, in_range)) {
#pragma unroll
                for (uint32_t k = 0; k < kTermSources; ++k) {
                    inv[k] = inverse_root_in_range_rn(r2[k]);
                }
            } else {
#pragma unroll
                for (uint32_t k = 0; k < kTermSources; ++k) {
                    inv[k] = inverse_root_general(r2[k]);
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < kTermSources; k += 2) {
                double t0[C], t1[C];
                Term::form(src[3][k0 + k], inv[k], dx[k], dy[k], dz[k], t0);
                Term::form(src[3][k0 + k + 1], inv[k + 1], dx[k + 1], dy[k + 1], dz[k + 1], t1);
#pragma unroll
                for (uint32_t q = 0; q < C; ++q) {
                    space.terms[c & 1u][q][(k0 + k) / 2u][lane] = make_double2(t0[q], t1[q]);
                }
            }
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(kSourceAhead - 1) : "memory");
        __syncthreads();
    }
}

} // namespace ob
