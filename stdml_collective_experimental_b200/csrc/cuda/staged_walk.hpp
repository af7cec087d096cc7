// Who works on what in the staged all-reduce (staged_kernel.cuh): the tiles of a
// block in each round, the pieces of its staging ring, and the choice of grid
// and tile.  Host and device code: exercised on the CPU (tests/test_partition_cuda.cpp).
#pragma once
#include <algorithm>
#include <cstddef>

#include "comm.cuh"

namespace stdml::collective::cuda
{
struct StagedTile {
    unsigned long long lo, hi;  // flat vectors
};

struct StagedWalk {
    const unsigned long long *bound;  // shard s is [bound[s], bound[s + 1])
    int world, nb, b;
    int tile_shift;

    // First vector of shard s: 512-byte granules, spread evenly (s == world: the end).
    static STDML_HD unsigned long long shard_begin(unsigned long long nvec, int world, int s)
    {
        const unsigned long long groups = (nvec + 31ull) / 32ull;
        const unsigned long long v = groups * static_cast<unsigned long long>(s) / world * 32ull;
        return v < nvec ? v : nvec;
    }

    // Tile of shard s that this block handles in round k (empty past the shard's end).
    STDML_HD StagedTile tile_of(int s, int k) const
    {
        const unsigned long long end = bound[s + 1];
        StagedTile t;
        t.lo = bound[s] + ((static_cast<unsigned long long>(k) * nb + b) << tile_shift);
        t.lo = t.lo < end ? t.lo : end;
        t.hi = t.lo + (1ull << tile_shift);
        t.hi = t.hi < end ? t.hi : end;
        return t;
    }

    // Byte offset inside a staging slot of the ring piece of round k and shard s.
    STDML_HD unsigned long long piece(int k, int s) const
    {
        const unsigned long long i =
            (static_cast<unsigned long long>(b) * kStagedRing + k % kStagedRing) * world + s;
        return (i << tile_shift) * 16ull;
    }
};

struct StagedGeometry {
    int blocks = 0;  // 0: the slot cannot hold the ring of even one block
    int tile_shift = kStagedStepShift, rounds = 1;
};

// Grid and tile for `nvec` vectors.  A tile is kStagedRoundVec vectors over all shards
// of a round at most (the block's loads in flight), smaller where the message
// would otherwise leave blocks without a tile, and never so large that the
// rings of all blocks outgrow the staging slot.
inline StagedGeometry staged_geometry(int world, size_t nvec, size_t staging_bytes, int max_blocks)
{
    StagedGeometry g;
    size_t longest = 0;
    for (int s = 0; s < world; ++s) {
        longest = std::max<size_t>(longest, StagedWalk::shard_begin(nvec, world, s + 1) -
                                                StagedWalk::shard_begin(nvec, world, s));
    }
    const size_t want = kStagedRoundVec / static_cast<size_t>(world);
    const size_t most = static_cast<size_t>(max_blocks);
    const auto ring_bytes = [&](int shift) {
        return (static_cast<size_t>(kStagedRing) * world << shift) * 16;
    };
    while ((size_t{2} << g.tile_shift) <= want && (size_t{2} << g.tile_shift) * most <= longest &&
           ring_bytes(g.tile_shift + 1) * most <= staging_bytes) {
        ++g.tile_shift;
    }
    const size_t tiles = (longest + (size_t{1} << g.tile_shift) - 1) >> g.tile_shift;
    const size_t fit = staging_bytes / ring_bytes(g.tile_shift);
    g.blocks = static_cast<int>(std::min<size_t>({tiles, most, fit}));
    if (g.blocks > 0) { g.rounds = static_cast<int>((tiles + g.blocks - 1) / g.blocks); }
    return g;
}
}  // namespace stdml::collective::cuda
