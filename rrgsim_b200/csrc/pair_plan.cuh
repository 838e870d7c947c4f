// The schedule of the kernels that evaluate each unordered pair of particles once (direct_sym.cu,
// adjoint.cu): i-tiles against j-tiles, cut into equal runs of rounds, one run per resident block.
#pragma once

#include <algorithm>

#include "direct_epi.cuh"

namespace rrg {

constexpr int kPairWarps = kDirectThreads / 32;
static_assert(kPairWarps == 8, "a j-tile is one chunk of 32 per warp, a unit eight rounds");

// The schedule: units of i-tile a are j-tiles a G .. nt - 1, numbered from first_unit(a); round
// 8 u + r is round r of unit u.
struct SymPlan {
    int n, nt, g, tiles;  // particles, j-tiles, i-particles per thread, i-tiles
    int64_t rounds;
    int blocks;           // runs: block b takes rounds [b rounds / blocks, (b + 1) rounds / blocks),
                          // at least the 8 of one unit
    int islots;           // i slots: the most blocks that share one i-tile

    __host__ __device__ int64_t first_unit(int64_t a) const {
        return a * nt - static_cast<int64_t>(g) * (a * (a - 1) / 2);
    }
    __host__ __device__ int64_t run_start(int64_t b) const { return b * rounds / blocks; }
    // the block whose run holds a round
    __host__ __device__ int block_of(int64_t round) const {
        return static_cast<int>(((round + 1) * blocks - 1) / rounds);
    }
    // the first and last block that work for i-tile a
    __host__ __device__ int first_block(int64_t a) const { return block_of(8 * first_unit(a)); }
    __host__ __device__ int last_block(int64_t a) const {
        return block_of(8 * (first_unit(a) + nt - a * g) - 1);
    }
};

inline SymPlan make_pair_plan(int64_t n, int g, int slots) {
    SymPlan p;
    p.n = static_cast<int>(n);
    p.g = g;
    p.nt = static_cast<int>((n + kDirectThreads - 1) / kDirectThreads);
    p.tiles = (p.nt + g - 1) / g;
    const int64_t units =
        p.first_unit(p.tiles - 1) + (p.nt - static_cast<int64_t>(p.tiles - 1) * g);
    p.rounds = 8 * units;
    p.blocks = static_cast<int>(std::min<int64_t>(slots, units));
    p.islots = 1;
    for (int a = 0; a < p.tiles; ++a)
        p.islots = std::max(p.islots, p.last_block(a) - p.first_block(a) + 1);
    return p;
}

__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float half_sum(float2 v) { return __fadd_rn(v.x, v.y); }

// resident blocks of kDirectThreads per SM with `smem` bytes of dynamic shared memory
template <typename Kern>
int pair_blocks_per_sm(Kern k, size_t smem) {
    return resident_blocks_per_sm(reinterpret_cast<const void*>(k), kDirectThreads, smem);
}

// From 32 j-tiles to 131,072 particles (the sizes at which the schedule fills the SMs and its slots
// stay in bounds).
inline bool pair_plan_range(int64_t n) { return n > 31 * kDirectThreads && n <= 131072; }

}  // namespace rrg
