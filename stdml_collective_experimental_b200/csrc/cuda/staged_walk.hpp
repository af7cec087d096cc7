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
    int tile_shift = kStagedMinShift, rounds = 1;
    // A message longer than the slot goes round in it in one launch: the slot holds the rings of enough blocks.
    bool full = false;
};

// Grid and tile for `nvec` vectors on `num_sms` SMs that `vranks` ranks share.  A tile is kStagedRoundVec
// vectors over all shards of a round at most, smaller where its buffers would outgrow the shared
// memory of a block or the rings of enough blocks the staging slot, and where the message would
// otherwise leave blocks without a tile.
inline StagedGeometry staged_geometry(int world, size_t nvec, size_t staging_bytes, int num_sms, int vranks,
                                      int want_blocks, bool user_f32)
{
    StagedGeometry g;
    size_t longest = 0;
    for (int s = 0; s < world; ++s) {
        longest = std::max<size_t>(longest, StagedWalk::shard_begin(nvec, world, s + 1) -
                                                StagedWalk::shard_begin(nvec, world, s));
    }
    const auto ring_bytes = [&](int shift) {
        return (static_cast<size_t>(kStagedRing) * world << shift) * 16;
    };
    // blocks per rank that are resident together
    const auto most = [&](int shift) {
        const int resident = std::min(kMaxBlocks, staged_per_sm(world, shift, user_f32) * num_sms / vranks);
        return static_cast<size_t>(std::max(1, want_blocks > 0 ? std::min(want_blocks, resident) : resident));
    };
    const auto tiles_of = [&](int shift) { return (longest + (size_t{1} << shift) - 1) >> shift; };
    // Rings of enough blocks: of most SMs, or of two on each for tiles from 256 vectors on among two or three ranks.  In
    // between a slot gives as many blocks as it holds.  Tensors of 96 MB, f32, us, one launch in tiles of 64 / 128 / 256 /
    // 512 vectors: 2 ranks, slots of 2 MB 447 / 410 / 532 / 663, 4 MB 331 / 252 / 267 / 336 (bf16 24 MB 65 / 92 with 128 / 256),
    // 8 MB 334 / 191 / 157 / 172, 16 MB 361 / 205 / 132 / 109; 3 ranks, 4 MB 382 / 274 / 286, 8 MB 407 / 243 / 180; 4 ranks,
    // 2 MB 579 / 483 / 598, 4 MB 424 / 329 / 308, 8 MB 480 / 300 / 239; 8 ranks, 2 MB 766 / 679, 4 MB 630 / 505.
    const auto enough = [&](int shift) {
        const int some = std::max(1, (shift < 8 || world > 3 ? 1 : 2) * num_sms * 3 / 4 / vranks);
        return ring_bytes(shift) * std::min<size_t>({tiles_of(shift), most(shift), static_cast<size_t>(some)}) <= staging_bytes;
    };
    // (where the smallest tiles do not fit so either, fewer blocks with larger ones)
    const bool cramped = !enough(kStagedMinShift);
    const size_t want = std::max<size_t>(kStagedRoundVec / static_cast<size_t>(world), size_t{1} << kStagedMinShift);
    const auto good = [&](int shift) {
        const size_t tile = size_t{1} << shift;
        if (tile > want || staged_smem(world, shift, user_f32) > kStagedSmem) { return false; }
        if (cramped ? tile > 256 || ring_bytes(shift) > staging_bytes : !enough(shift)) { return false; }
        // A short message has fewer blocks, not smaller tiles than about a vector per worker, and larger ones
        // rather than a second round (a set of ragged tensors pays several memory latencies per vector: 224 of
        // them, 4 ranks, 20.6 us with 256 vectors at least, 14.5 so).
        if (tile <= kStagedThreads && tile * (world - 1) <= 256) { return true; }
        if (tile <= 256) { return tile / 2 * most(shift - 1) < longest; }
        return tile * most(shift) <= longest;
    };
    while (good(g.tile_shift + 1)) { ++g.tile_shift; }
    const size_t tiles = tiles_of(g.tile_shift);
    const size_t fit = staging_bytes / ring_bytes(g.tile_shift);
    g.blocks = static_cast<int>(std::min<size_t>({tiles, most(g.tile_shift), fit}));
    // A launch per slot instead: 8 ranks, slots of 2 MB, 96 MB 1280 us (679 so); 2 ranks, 8 MB 286 (157).
    // Slots below 2 MB have a launch each, as callers may count on.
    g.full = !cramped && staging_bytes >= 2u << 20;
    if (g.blocks > 0) { g.rounds = static_cast<int>((tiles + g.blocks - 1) / g.blocks); }
    return g;
}
}  // namespace stdml::collective::cuda
