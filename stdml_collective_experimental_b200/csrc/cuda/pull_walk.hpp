// Who moves what in the all_gather and broadcast by pull (kernels_pull.cu): the tiles of
// a block, the ring pieces, the shift of a rank's data, and the grid.  Host and device code:
// exercised on the CPU (tests/test_partition_cuda.cpp).
#pragma once
#include <algorithm>
#include <cstddef>

#include "comm.cuh"

namespace stdml::collective::cuda
{
// A rank's block of `bytes` bytes is seen as vectors of 16 bytes in which it starts
// `phase` bytes after the beginning of vector 0, as it does in a 16-byte aligned destination.  Block b of the grid moves vectors [k * nb + b) * T, + T) in round k.
struct PullWalk {
    unsigned long long bytes, stride;  // destination blocks start `stride` bytes apart
    int nb, b;
    int tile_shift;  // T = 1 << tile_shift vectors

    STDML_HD unsigned int phase(int p) const
    {
        return static_cast<unsigned int>(p) * static_cast<unsigned int>(stride & 15ull) & 15u;
    }
    STDML_HD unsigned long long vectors(unsigned int ph) const { return (bytes + ph + 15ull) / 16ull; }
    STDML_HD unsigned long long first_vector(int k) const
    {
        return (static_cast<unsigned long long>(k) * nb + b) << tile_shift;
    }
    // Byte offset inside a staging slot of the ring piece of round k.
    STDML_HD unsigned long long piece(int k) const
    {
        return ((static_cast<unsigned long long>(b) * kPullRing + k % kPullRing) << tile_shift) * 16ull;
    }
};

struct PullGeometry {
    int blocks = 0;  // 0: the slot cannot hold the ring of even one block
    int tile_shift = kPullStepShift, rounds = 1;
    // of the staging slot, for all blocks
    size_t ring_bytes() const
    {
        return ((static_cast<size_t>(blocks) * kPullRing) << tile_shift) * 16;
    }
};

// Grid and tile for blocks of `bytes` bytes read from `sources` ranks: a tile gives
// each thread up to kPullVec vectors to copy per round over all sources, less where the
// message would otherwise leave blocks without a tile.
inline PullGeometry pull_geometry(int sources, size_t bytes, size_t staging_bytes, int max_blocks)
{
    PullGeometry g;
    const size_t most = static_cast<size_t>(max_blocks);
    const size_t nvec = (bytes + 15 + 15) / 16;  // with the largest shift
    const size_t want = static_cast<size_t>(kPullThreads) * kPullVec / static_cast<size_t>(std::max(1, sources));
    const auto ring_bytes = [&](int shift) { return (static_cast<size_t>(kPullRing) << shift) * 16; };
    while ((size_t{2} << g.tile_shift) <= want && (size_t{2} << g.tile_shift) * most <= nvec &&
           ring_bytes(g.tile_shift + 1) * most <= staging_bytes) {
        ++g.tile_shift;
    }
    const size_t tiles = (nvec + (size_t{1} << g.tile_shift) - 1) >> g.tile_shift;
    g.blocks = static_cast<int>(std::min<size_t>({tiles, most, staging_bytes / ring_bytes(g.tile_shift)}));
    if (g.blocks > 0) { g.rounds = static_cast<int>((tiles + g.blocks - 1) / g.blocks); }
    return g;
}
}  // namespace stdml::collective::cuda
