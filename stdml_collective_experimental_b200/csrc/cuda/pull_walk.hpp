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
// `phase` bytes after the beginning of vector 0, as it does in a 16-byte aligned destination.
struct PullLayout {
    unsigned long long bytes, stride;  // destination blocks start `stride` bytes apart

    STDML_HD unsigned int phase(int p) const
    {
        return static_cast<unsigned int>(p) * static_cast<unsigned int>(stride & 15ull) & 15u;
    }
    STDML_HD unsigned long long vectors(unsigned int ph) const { return (bytes + ph + 15ull) / 16ull; }
};

// Block b of the grid moves vectors [k * nb + b) * T, + T) in round k.
struct PullWalk : PullLayout {
    int nb, b;
    int tile_shift;  // T = 1 << tile_shift vectors

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

// The same for pull_long_kernel: tiles of any number of vectors, a longer ring.
struct PullLongWalk : PullLayout {
    int nb, b;
    unsigned int tile;

    STDML_HD unsigned long long first_vector(int k) const
    {
        return (static_cast<unsigned long long>(k) * nb + b) * tile;
    }
    STDML_HD unsigned long long piece(int k) const
    {
        return (static_cast<unsigned long long>(b) * kPullLongRing + k % kPullLongRing) * tile * 16ull;
    }
};

struct PullGeometry {
    int blocks = 0;  // 0: the slot cannot hold the ring of even one block
    unsigned int tile = 1u << kPullStepShift;
    int rounds = 1, ring = kPullRing;
    bool lng = false;  // for pull_long_kernel
    // of the staging slot, for all blocks
    size_t ring_bytes() const { return static_cast<size_t>(blocks) * ring * tile * 16; }
};

// Grid and tile for blocks of `bytes` bytes read from `sources` ranks, on `num_sms` SMs that `vranks` ranks
// share.  pull_kernel: a tile gives each thread up to kPullVec vectors to copy per round over
// all sources, less where the message would otherwise leave blocks without a tile.
inline PullGeometry pull_geometry(int sources, size_t bytes, size_t staging_bytes, int num_sms, int vranks,
                                  int want_blocks)
{
    const auto resident = [&](int per_sm) {
        const int n = std::max(1, std::min(kMaxBlocks, per_sm * num_sms / vranks));
        return static_cast<size_t>(want_blocks > 0 ? std::min(want_blocks, n) : n);
    };
    const size_t nvec = (bytes + 15 + 15) / 16;  // with the largest shift
    PullGeometry g;
    size_t most = resident(kPullPerSm);
    const size_t want = static_cast<size_t>(kPullThreads) * kPullVec / static_cast<size_t>(std::max(1, sources));
    while (g.tile * 2 <= want && g.tile * 2 * most <= nvec && kPullRing * g.tile * 2 * 16 * most <= staging_bytes) {
        g.tile *= 2;
    }
    const auto lay_out = [&]() {
        const size_t tiles = (nvec + g.tile - 1) / g.tile;
        g.blocks = static_cast<int>(std::min<size_t>({tiles, most, staging_bytes / (static_cast<size_t>(g.ring) * g.tile * 16)}));
        if (g.blocks > 0) { g.rounds = static_cast<int>((tiles + g.blocks - 1) / g.blocks); }
    };
    lay_out();
    // pull_long_kernel, wherever every block of its grid has some work: broadcast of 1 MB to 1 (422 vectors
    // per block) 6.2 us and 6.4 so, of 0.5 MB to 7 (844) 9.7 and 8.2, all_gather of 8 x 0.7 MB 25.5 and 18.  From eight
    // sources on its tiles and bulk copies get small (16 x 1 MB: 74 us, 81 so).
    const PullGeometry s = g;
    g.lng = true;
    g.ring = kPullLongRing;
    most = resident(kPullLongPerSm);
    // The largest tile of which the slot holds the rings of all blocks.  Broadcast of 94 MB, us, pull_kernel / so: 4 ranks,
    // tiles of 256 vectors (slots of 4 MB) 462 / 315, of 128 (2 MB) 508 / 621; 2 ranks, 512 (16 MB) 136 / 88, 256 (8 MB)
    // 220 / 160, 128 (4 MB) 246 / 311; 3 ranks, 192 (4 MB) 331 / 348; all_gather of 8 x 2.47 MB, 256 (2 MB) 57 / 46,
    // 128 (1 MB) 62 both.
    g.tile = static_cast<unsigned int>(
        std::min<size_t>(pull_long_tile(sources), staging_bytes / (kPullLongRing * 16 * most) / 32 * 32));
    // (a broadcast of 2.1 MB to 1 in tiles of 256: 10.4 us, in pull_kernel's 8.4)
    const size_t least = g.tile < std::min(512u, pull_long_tile(sources)) ? 2 * kPullLongMin : kPullLongMin;
    if (sources > kPullLongSources || nvec < least * most || g.tile < kPullLongMinTile) { return s; }
    lay_out();
    g.blocks = static_cast<int>(most);
    // tiles of equal size that just fill their rounds
    const size_t per_round = static_cast<size_t>(g.rounds) * g.blocks;
    g.tile = static_cast<unsigned int>((nvec + per_round - 1) / per_round + 31) / 32 * 32;
    lay_out();
    return g;
}
}  // namespace stdml::collective::cuda
