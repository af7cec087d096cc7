// all_gather and broadcast by pull, for destinations outside the arena, in ONE launch of
// any length: every rank (broadcast: root) packs its block tile by tile into
// a small ring in its staging slot, and the others read the tiles from there
// straight into their tensors.
//
// What bounds it: bytes.  A block that is packed whole, met at a barrier and then copied
// moves through HBM twice more than it has to; the ring (four pieces per
// block, a few MB in all) stays in the L2, so that HBM sees the source once and the
// destinations once.  Pass k of a block: pack tile k, arrive, wait until
// all ranks have packed tile k-1, copy tile k-1 of all sources; the wait is hidden by the
// pack.  Ring of four: tile k goes over tile k-4, whose readers said that they were
// done with it by arriving in their pass k-2.
//
// Blocks whose size is no multiple of 16 land on odd addresses: block p starts
// p * stride % 16 bytes after a vector boundary of an aligned destination.  The packer shifts its
// data by that much (two aligned loads and a funnel shift per vector), so that
// the world - 1 copies of each tile are aligned 16-byte accesses; only the vectors
// at a block's ends are moved byte by byte.
// Measured, us: all_gather of 8 x 2.47 MB (an odd size) 518 -> 65, broadcast of 94 MB
// to 3 others 345 -> 117.  By vectors per thread and round over all sources, four in
// flight: 8: 68 / 128, 16: 65 / 117, 32: 76 / 117; eight in flight at 80 registers: 73 / 139.
//
// The reference's counterparts are its full-mesh exchange
// (src/stdml/collective/all_gather.cpp:16-56 there) and its broadcast walk
// (src/stdml/collective/session.cpp:49-62 there).
#include "copy.cuh"
#include "pull_walk.hpp"

namespace stdml::collective::cuda
{
// A block of the destination in the vector numbering of PullWalk.
struct PullBlock {
    char *base;               // address of vector 0
    unsigned long long nvec;  // vectors that hold a byte of the block
    unsigned int phase;
    bool aligned;
    // all vectors of [v, v + kPullThreads) can be stored whole
    __device__ __forceinline__ bool inside(unsigned long long v) const
    {
        return aligned && v >= 1 && v + kPullThreads < nvec;
    }
};

__global__ void __launch_bounds__(kPullThreads, kPullPerSm)
    pull_kernel(const __grid_constant__ CommCtx ctx, const __grid_constant__ PullArgs a)
{
    constexpr int kBatch = 4;  // vectors of a thread in flight
    __shared__ BlockSync sync;
    __shared__ PullBlock blocks[kMaxRanks];
    const int vr = static_cast<int>(blockIdx.y);
    const int rank = ctx.rank + vr;
    const int world = ctx.world;
    const bool bcast = a.root >= 0;
    const bool packs = !bcast || a.root == rank;
    const PullWalk walk{a.bytes, a.stride, static_cast<int>(gridDim.x),
                        static_cast<int>(blockIdx.x), a.tile_shift};
    sync_begin(ctx, rank, &sync);
    const unsigned long long policy = evict_first_policy();
    // blocks[p]: where the data of source p goes (broadcast: the same place for every p)
    if (static_cast<int>(threadIdx.x) < world) {
        const int p = static_cast<int>(threadIdx.x);
        PullBlock d;
        d.phase = bcast ? 0u : walk.phase(p);
        char *first = static_cast<char *>(a.dst[vr]) +
                      (bcast ? 0ull : static_cast<unsigned long long>(p) * a.stride);
        d.base = first - d.phase;
        d.nvec = walk.vectors(d.phase);
        d.aligned = (reinterpret_cast<unsigned long long>(d.base) & 15ull) == 0ull;
        blocks[p] = d;
    }
    __syncthreads();

    const PullBlock &own = blocks[rank];
    const ShiftedSource src(a.src[vr], a.bytes, own.phase);
    const bool in_place = own.base + own.phase == a.src[vr];
    char *ring = ctx.base[rank] + a.off;
    const int per_tile = a.tile_shift - kPullStepShift;  // log2 of the steps in a tile
    const int sources = bcast ? (a.root == rank ? 0 : 1) : world - 1;
    const int steps = sources << per_tile;
    // steps go through one source after the other, starting with the next rank so that
    // peers do not all read the same GPU first; everything about a step but the
    // thread's own vector is uniform over the block
    auto source_at = [&](int q) {
        if (bcast) { return a.root; }
        const int p = rank + 1 + (q >> per_tile);
        return p < world ? p : p - world;
    };
    auto first_at = [&](int q) {
        return static_cast<unsigned int>(q & ((1 << per_tile) - 1)) << kPullStepShift;
    };

    for (int k = 0; k <= a.rounds; ++k) {
        if (k < a.rounds) {
            if (packs) {
                const unsigned long long v0 = walk.first_vector(k);
                char *to = ring + walk.piece(k);
                for (int q0 = 0; q0 < 1 << per_tile; q0 += kBatch) {
                    uint4 x[kBatch];
#pragma unroll
                    for (int u = 0; u < kBatch; ++u) {
                        const unsigned int i = (static_cast<unsigned int>(q0 + u) << kPullStepShift) + threadIdx.x;
                        if (q0 + u >= 1 << per_tile) { continue; }
                        if (own.inside(v0 + i - threadIdx.x)) {
                            x[u] = src.load_inside(v0 + i, policy);
                        } else if (v0 + i < own.nvec) {
                            x[u] = src.load(v0 + i, policy);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kBatch; ++u) {
                        const unsigned int i = (static_cast<unsigned int>(q0 + u) << kPullStepShift) + threadIdx.x;
                        if (q0 + u >= 1 << per_tile || v0 + i >= own.nvec) { continue; }
                        st_arena_v4(to + i * 16u, x[u]);
                        if (in_place) { continue; }
                        if (own.inside(v0 + i - threadIdx.x)) {
                            st_stream_v4(own.base + (v0 + i) * 16ull, x[u], policy);
                        } else {
                            store_virtual(own.base + own.phase, a.bytes, own.phase, v0 + i, x[u], policy);
                        }
                    }
                }
            }
            arrive_all(ctx, rank, &sync, k + 1);
        }
        if (k == 0) { continue; }
        if (!wait_all(ctx, rank, &sync, k)) { return; }
        // ---- tile k-1 of the other sources
        const unsigned long long v0 = walk.first_vector(k - 1);
        const unsigned long long from = a.off + walk.piece(k - 1) + threadIdx.x * 16u;
        bool ends = false;  // some step touches an end of its block
        for (int q0 = 0; q0 < steps; q0 += kBatch) {
            uint4 x[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                if (q0 + u >= steps) { continue; }
                const int p = source_at(q0 + u);
                const unsigned int i = first_at(q0 + u);
                if (blocks[p].inside(v0 + i)) {
                    x[u] = ld_arena_v4(ctx.base[p] + from + i * 16u);
                } else {
                    ends = true;
                }
            }
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                if (q0 + u >= steps) { continue; }
                const PullBlock &d = blocks[source_at(q0 + u)];
                const unsigned int i = first_at(q0 + u);
                if (d.inside(v0 + i)) {
                    st_stream_v4(d.base + (v0 + i + threadIdx.x) * 16ull, x[u], policy);
                }
            }
        }
        for (int q = 0; ends && q < steps; ++q) {
            const int p = source_at(q);
            const PullBlock &d = blocks[p];
            const unsigned int i = first_at(q);
            const unsigned long long v = v0 + i + threadIdx.x;
            if (d.inside(v0 + i) || v >= d.nvec) { continue; }
            store_virtual(d.base + d.phase, a.bytes, d.phase, v,
                          ld_arena_v4(ctx.base[p] + from + i * 16u), policy);
        }
    }
    advance_epoch(&sync, a.rounds);
    if (a.end_barrier && !peer_barrier(ctx, rank, &sync)) { return; }
    sync_end(ctx, rank, &sync);
}

int launch_pull(const CommCtx &ctx, const PullArgs &a, int blocks, int vranks, void *stream)
{
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid(blocks, vranks, 1);
    if (vranks > 1) {
        void *params[2] = {const_cast<CommCtx *>(&ctx), const_cast<PullArgs *>(&a)};
        return static_cast<int>(cudaLaunchCooperativeKernel(
            reinterpret_cast<const void *>(&pull_kernel), grid, dim3(kPullThreads), params, 0, s));
    }
    pull_kernel<<<grid, kPullThreads, 0, s>>>(ctx, a);
    return static_cast<int>(cudaGetLastError());
}
}  // namespace stdml::collective::cuda
