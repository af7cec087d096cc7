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
// Measured, us: all_gather of 8 x 2.47 MB (an odd size) 518 -> 58, broadcast of 94 MB
// to 3 others 345 -> 111 (108 by the second kernel).  By vectors per thread and round over all
// sources, four in flight, when 16 took 65 / 117: 8: 68 / 128, 32: 76 / 117; eight in flight at 80
// registers: 73 / 139.
//
// The reference's counterparts are its full-mesh exchange
// (src/stdml/collective/all_gather.cpp:16-56 there) and its broadcast walk
// (src/stdml/collective/session.cpp:49-62 there).
#include "ar_kernel.cuh"
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
    const bool packs = (!bcast || a.root == rank) && a.src[vr] != nullptr;
    const bool stores = a.dst[vr] != nullptr;
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
    const bool ring_only = !stores || own.base + own.phase == a.src[vr];  // own block: packed, not stored
    char *ring = ctx.base[rank] + a.off;
    const int per_tile = a.tile_shift - kPullStepShift;  // log2 of the steps in a tile
    const int sources = !stores ? 0 : bcast ? (a.root == rank ? 0 : 1) : world - 1;
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
                        if (ring_only) { continue; }
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

// The same for messages of several rounds.  What bounds them is bytes in flight, and
// registers hold too few: the copies from the rings to the tensors go through shared
// memory by bulk asynchronous copies in both directions, which one thread of an extra warp
// keeps under way while the other warps pack the next tile.  Pass k: tile k-1 is copied
// and tile k packed side by side; arrive; wait for the others.  (An arrival then also says that
// tile k-1 has been read.)  Vectors at a block's ends are stored byte by byte; a
// destination that is not 16-byte aligned is written by the packing warps.
// launch_pull says which messages it is for.
constexpr int kPullBufs = 5;  // of kPullBufVec vectors: four blocks of an SM fit
constexpr unsigned int kPullBufVec = 512;
constexpr int kPullLongThreads = kPullThreads + 32;
constexpr int kPullLongBatch = 4;  // vectors of a packing thread in flight

__device__ __forceinline__ void bulk_store(void *dst, uint32_t src_smem, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                 "r"(src_smem), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

__global__ void __launch_bounds__(kPullLongThreads, kPullPerSm)
    pull_long_kernel(const __grid_constant__ CommCtx ctx, const __grid_constant__ PullArgs a)
{
    extern __shared__ __align__(128) unsigned char bufs[];
    __shared__ BlockSync sync;
    __shared__ PullBlock blocks[kMaxRanks];
    __shared__ __align__(8) unsigned long long bars[kPullBufs];
    const int vr = static_cast<int>(blockIdx.y);
    const int rank = ctx.rank + vr;
    const int world = ctx.world;
    const bool bcast = a.root >= 0;
    const bool packs = (!bcast || a.root == rank) && a.src[vr] != nullptr;
    const bool stores = a.dst[vr] != nullptr;
    const PullWalk walk{a.bytes, a.stride, static_cast<int>(gridDim.x),
                        static_cast<int>(blockIdx.x), a.tile_shift};
    sync_begin(ctx, rank, &sync);
    const unsigned long long policy = evict_first_policy();
    const uint32_t bars_s = smem_addr(bars), bufs_s = smem_addr(bufs);
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
    if (threadIdx.x == 0) {
        for (int i = 0; i < kPullBufs; ++i) { mbar_init(bars_s + 8u * i, 1u); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_proxy();
    }
    __syncthreads();

    const PullBlock &own = blocks[rank];
    const ShiftedSource src(a.src[vr], a.bytes, own.phase);
    const bool ring_only = !stores || own.base + own.phase == a.src[vr];  // own block: packed, not stored
    const bool by_bulk = own.aligned;  // alike for all blocks of a destination
    char *ring = ctx.base[rank] + a.off;
    const unsigned long long tile = 1ull << a.tile_shift;
    const int steps = 1 << (a.tile_shift - kPullStepShift);
    const int sources = !stores ? 0 : bcast ? (a.root == rank ? 0 : 1) : world - 1;
    auto source_at = [&](int i) {
        if (bcast) { return a.root; }
        const int p = rank + 1 + i;
        return p < world ? p : p - world;
    };
    const bool copier = threadIdx.x == kPullThreads;
    int filled = 0;  // copier only: buffers filled so far

    for (int k = 0; k <= a.rounds; ++k) {
        bool ok = true;
        // broadcast: root's pack is what the others wait for, from an eighth or so of the
        // grid (94 MB to 3 others: 116 us without, 108 with it); in an all_gather every rank packs
        if (is_sync_thread() && bcast && packs && k + 1 < a.rounds) {
            src.prefetch(walk.first_vector(k + 1), tile);
        }
        if (threadIdx.x < kPullThreads && packs && k < a.rounds) {
            // ---- pack tile k
            const unsigned long long v0 = walk.first_vector(k);
            char *to = ring + walk.piece(k);
            for (int q0 = 0; q0 < steps; q0 += kPullLongBatch) {
                uint4 x[kPullLongBatch];
#pragma unroll
                for (int u = 0; u < kPullLongBatch; ++u) {
                    const unsigned int i = (static_cast<unsigned int>(q0 + u) << kPullStepShift) + threadIdx.x;
                    if (q0 + u >= steps) { continue; }
                    if (own.inside(v0 + i - threadIdx.x)) {
                        x[u] = src.load_inside(v0 + i, policy);
                    } else if (v0 + i < own.nvec) {
                        x[u] = src.load(v0 + i, policy);
                    }
                }
#pragma unroll
                for (int u = 0; u < kPullLongBatch; ++u) {
                    const unsigned int i = (static_cast<unsigned int>(q0 + u) << kPullStepShift) + threadIdx.x;
                    if (q0 + u >= steps || v0 + i >= own.nvec) { continue; }
                    st_arena_v4(to + i * 16u, x[u]);
                    if (ring_only) { continue; }
                    if (own.inside(v0 + i - threadIdx.x)) {
                        st_stream_v4(own.base + (v0 + i) * 16ull, x[u], policy);
                    } else {
                        store_virtual(own.base + own.phase, a.bytes, own.phase, v0 + i, x[u], policy);
                    }
                }
            }
            fence_async_proxy();  // the peers read the ring with bulk copies
        }
        if (k > 0) {
            const unsigned long long v0 = walk.first_vector(k - 1);
            const unsigned long long from = a.off + walk.piece(k - 1);
            if (!by_bulk) {
                for (int i = 0; threadIdx.x < kPullThreads && i < sources; ++i) {
                    const int p = source_at(i);
                    const PullBlock &d = blocks[p];
                    for (unsigned long long v = v0 + threadIdx.x; v < v0 + tile && v < d.nvec;
                         v += kPullThreads) {
                        store_virtual(d.base + d.phase, a.bytes, d.phase, v,
                                      ld_arena_v4(ctx.base[p] + from + (v - v0) * 16ull), policy);
                    }
                }
            } else if (copier) {
                // ---- copy tile k-1 of the other sources: whole vectors by bulk copies
                fence_async_proxy();
                int stored = filled;
                auto span_of_source = [&](const PullBlock &d, unsigned long long *lo, unsigned long long *hi) {
                    const unsigned long long end = (a.bytes + d.phase) % 16ull != 0ull ? d.nvec - 1 : d.nvec;
                    *lo = v0 == 0 && d.phase != 0u ? 1ull : v0;
                    *hi = v0 + tile < end ? v0 + tile : end;
                };
                // two walks over the same chunks, the loads ahead of the stores
                int li = 0, si = 0;
                unsigned long long lv = 0, lhi = 0, sv = 0, shi = 0;
                bool lopen = false, sopen = false;
                auto next = [&](int *i, bool *open, unsigned long long *v, unsigned long long *hi) {
                    while (*i < sources) {
                        if (!*open) {
                            span_of_source(blocks[source_at(*i)], v, hi);
                            *open = true;
                        }
                        if (*v < *hi) { return true; }
                        *open = false;
                        ++*i;
                    }
                    return false;
                };
                for (;;) {
                    while (ok && filled - stored < kPullBufs - 1 && next(&li, &lopen, &lv, &lhi)) {
                        const int j = filled % kPullBufs;
                        // the store of kPullBufs chunks ago must have read this buffer; at
                        // least one younger store has been issued since, which need not
                        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                        const unsigned long long n = lhi - lv < kPullBufVec ? lhi - lv : kPullBufVec;
                        const uint32_t bytes = static_cast<uint32_t>(n) * 16u;
                        mbar_expect_tx(bars_s + 8u * j, bytes);
                        bulk_load(bufs_s + j * kPullBufVec * 16u,
                                  ctx.base[source_at(li)] + from + (lv - v0) * 16ull, bytes,
                                  bars_s + 8u * j);
                        lv += n;
                        ++filled;
                    }
                    if (stored == filled) { break; }
                    const int j = stored % kPullBufs;
                    ok = mbar_wait(ctx, bars_s + 8u * j, static_cast<uint32_t>((stored / kPullBufs) & 1),
                                   ctx.timeout_ns) && ok;
                    if (!ok) {
                        report_timeout(ctx, rank, -1, 0u, 0u, 64);
                        // the others already under way: one more bounded chance each
                        for (int t = stored + 1; t < filled; ++t) {
                            (void)mbar_wait(ctx, bars_s + 8u * (t % kPullBufs),
                                            static_cast<uint32_t>((t / kPullBufs) & 1), ctx.timeout_ns / 4);
                        }
                        break;
                    }
                    (void)next(&si, &sopen, &sv, &shi);
                    const unsigned long long n = shi - sv < kPullBufVec ? shi - sv : kPullBufVec;
                    bulk_store(blocks[source_at(si)].base + sv * 16ull, bufs_s + j * kPullBufVec * 16u,
                               static_cast<uint32_t>(n) * 16u);
                    sv += n;
                    ++stored;
                }
            } else if (threadIdx.x > kPullThreads) {
                // the ends of the blocks: lanes of the copier's warp, a source each
                for (int i = static_cast<int>(threadIdx.x) - kPullThreads - 1; i < sources; i += 31) {
                    const int p = source_at(i);
                    const PullBlock &d = blocks[p];
                    const unsigned long long last = d.nvec - 1;
                    if (v0 == 0 && d.phase != 0u) {
                        store_virtual(d.base + d.phase, a.bytes, d.phase, 0,
                                      ld_arena_v4(ctx.base[p] + from), policy);
                    }
                    if ((a.bytes + d.phase) % 16ull != 0ull && last >= v0 && last < v0 + tile &&
                        !(last == 0 && d.phase != 0u)) {
                        store_virtual(d.base + d.phase, a.bytes, d.phase, last,
                                      ld_arena_v4(ctx.base[p] + from + (last - v0) * 16ull), policy);
                    }
                }
            }
        }
        if (__syncthreads_and(ok ? 1 : 0) == 0) {
            if (copier) { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
            return;
        }
        if (k < a.rounds) {
            tell_all(ctx, rank, &sync, k + 1);
            if (!wait_all(ctx, rank, &sync, k + 1)) {
                if (copier) { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
                return;
            }
        }
    }
    if (copier) { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
    advance_epoch(&sync, a.rounds);
    // the rings of the last tiles may only be reused when all have read them: the next
    // call uses the other slot, whose users of the call before this one are done
    if (a.end_barrier && !peer_barrier(ctx, rank, &sync)) { return; }
    sync_end(ctx, rank, &sync);
}

int launch_pull(const CommCtx &ctx, const PullArgs &a, int blocks, int vranks, void *stream)
{
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid(blocks, vranks, 1);
    // One or two rounds are a matter of latency, to which the way through shared memory adds.
    // From three on, us, pull_kernel / pull_long_kernel, tensors not in the L2: broadcast of
    // 100 MB to 3 121 / 117, 34 MB to 5 70 / 66, 100 MB to 7 228 / 216, 17 MB to 7 49 / 48.
    // all_gather, in which every rank copies and packs the whole time: 3 x 34 MB 110 / 103,
    // 4 x 17 MB 78 / 83, 4 x 100 MB 442 / 437, 8 x 2.47 MB 58 both, 8 x 8 MB 150 / 160.
    // Two ranks: the registers keep up (broadcast 100 MB 70 / 74, all_gather 34 MB 57 both).
    // (Destinations off a vector boundary do better in pull_kernel throughout, 34 MB to 3: 293 / 325,
    // but a rank does not know the others', and all have to run the same kernel.)
    const bool lng = a.rounds > 2 && ctx.world > 2 && (a.root >= 0 || ctx.world == 3);
    const void *kernel = lng ? reinterpret_cast<const void *>(&pull_long_kernel)
                             : reinterpret_cast<const void *>(&pull_kernel);
    const dim3 block(lng ? kPullLongThreads : kPullThreads);
    const size_t smem = lng ? kPullBufs * kPullBufVec * 16u : 0u;
    void *params[2] = {const_cast<CommCtx *>(&ctx), const_cast<PullArgs *>(&a)};
    if (vranks > 1) {
        return static_cast<int>(cudaLaunchCooperativeKernel(kernel, grid, block, params, smem, s));
    }
    return static_cast<int>(cudaLaunchKernel(kernel, grid, block, params, smem, s));
}
}  // namespace stdml::collective::cuda
