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
// Measured against a slot-sized region, us: all_gather of 8 x 2.47 MB (an odd size) 518 -> 58, broadcast of 94 MB
// to 3 others 345 -> 111 (both have gone to the second kernel since).  By vectors per thread and round over all
// sources, four in flight, when 16 took 65 / 117: 8: 68 / 128, 32: 76 / 117; eight in flight at 80
// registers: 73 / 139.
//
// The reference's counterparts are its full-mesh exchange
// (src/stdml/collective/all_gather.cpp:16-56 there) and its broadcast walk
// (src/stdml/collective/session.cpp:49-62 there).
#include <atomic>

#include "ar_kernel.cuh"
#include "copy.cuh"
#include "pull_walk.hpp"
#include "ring_sync.cuh"

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
        return whole(v, kPullThreads);
    }
    // so can all of [v, v + n)
    __device__ __forceinline__ bool whole(unsigned long long v, unsigned int n) const
    {
        return aligned && v >= 1 && v + n < nvec;
    }
};

// Where the data of source p goes (broadcast: the same place for every p).
__device__ __forceinline__ PullBlock pull_block(const PullArgs &a, const PullLayout &walk, int vr, int p)
{
    const bool bcast = a.root >= 0;
    PullBlock d;
    d.phase = bcast ? 0u : walk.phase(p);
    char *first = static_cast<char *>(a.dst[vr]) +
                  (bcast ? 0ull : static_cast<unsigned long long>(p) * a.stride);
    d.base = first - d.phase;
    d.nvec = walk.vectors(d.phase);
    d.aligned = (reinterpret_cast<unsigned long long>(d.base) & 15ull) == 0ull;
    return d;
}

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
    const PullWalk walk{{a.bytes, a.stride}, static_cast<int>(gridDim.x), static_cast<int>(blockIdx.x), a.tile_shift};
    sync_begin(ctx, rank, &sync);
    const unsigned long long policy = evict_first_policy();
    if (static_cast<int>(threadIdx.x) < world) {
        blocks[threadIdx.x] = pull_block(a, walk, vr, static_cast<int>(threadIdx.x));
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

// The same for messages of several rounds.  What bounds them is bytes in flight and the way of a flag
// (a fence for the block's stores, the flag, its poll, the first load behind it: 4 to 8 us under
// load, several times what the bytes of a round take).  So four warps of a block look after these
// (ring_sync.cuh, as in staged_kernel.cuh): the loader brings the tensor's tiles into shared memory by bulk
// copies, the teller sets the flags, the fetcher polls them and brings the ring pieces of all
// sources into shared memory, the storer takes them on to the destination, by bulk copies too.  The workers
// only pack: pass k takes tile k from shared memory to the ring (and to the own block of the destination), and
// waits for the pieces of tile k - lag.  An odd destination is theirs as well: its vectors are put together
// from two of the piece's.  Ring of 2 lag + 1: tile k goes over tile k - 2 lag - 1, which its readers had
// in their shared memory before the flags that the fetcher saw for pass k - 1.
// Measured among ranks of one GPU, us, against a kernel that copied by bulk copies in lockstep with the pack, or
// pull_kernel: broadcast in place of 94 MB to 3 others 108 / 93, into other tensors 144 / 116, of 100 MB to 7 284 / 234, 9 MB
// to 5 33 / 23; all_gather of 8 x 2.47 MB (an odd size) 54 / 42, 8 x 8 MB 142 / 125, 3 x 34 MB 104 / 98, 8 x 0.7 MB 25 / 18; to
// destinations off a vector boundary 8 x 2.47 MB 429 / 52, broadcast of 34 MB to 3 364 / 50.
// By lag, broadcast of 94 MB: 2: 143, 3: 121, 5: 100, 7: 95 (before there was a storer); no more from there on.
// Two blocks per SM and 100 KB each, or three and 64: 8 x 2.47 MB 42 / 44, 94 MB 91 / 89; buffers for three or four rounds
// of pieces, with smaller tiles: 49, 57 and 93, 102.
struct PullShared {
    PullBlock blocks[kMaxRanks];
    // A round's bytes are there: the tensor's, the ring pieces of all sources.
    Phases<2> tensor;
    Phases<kPullDepth> pieces;
    // Workers and storer are done with them.
    Phases<2> packed;
    Phases<kPullDepth> stored;
    Phases<8> done;  // passes: tile k packed, tile k - lag here
    Phases<1> left;  // workers and storer have come through
    uint32_t epoch;
    int dead;  // the block gives up
};
static_assert(kPullLongPerSm * (kPullLongSmem + other_smem(sizeof(PullShared))) <= kSmSmem, "so many blocks fit an SM");
static_assert(kPullLag <= 7, "passes that the workers may be ahead of the warp that tells the peers");

// n bytes of shared memory to a destination of any alignment: the lanes of `threads` threads that share a run
// (this one is `me`).  Aligned stores, put together from two vectors where the addresses differ.
__device__ __forceinline__ void store_run(char *dst, uint32_t src, unsigned int n, unsigned int me,
                                          unsigned int threads, unsigned long long policy)
{
    const unsigned int to_vec = static_cast<unsigned int>(-reinterpret_cast<long long>(dst)) & 15u;
    const unsigned int head = to_vec < n ? to_vec : n;
    const unsigned int vecs = (n - head) / 16u;
    const uint32_t from = src + head;
    const unsigned int odd = from & 15u;
    for (unsigned int j = me; j < vecs; j += threads) {
        const uint32_t at = (from & ~15u) + j * 16u;
        uint4 x = ld_shared_v4(at);
        if (odd != 0u) { x = shift_bytes(x, ld_shared_v4(at + 16u), odd); }
        st_stream_v4(dst + head + j * 16ull, x, policy);
    }
    const char *bytes = static_cast<const char *>(__cvta_shared_to_generic(src));
    const unsigned int rest = head + vecs * 16u;
    for (unsigned int j = me; j < head; j += threads) { dst[j] = bytes[j]; }
    for (unsigned int j = rest + me; j < n; j += threads) { dst[j] = bytes[j]; }
}

struct PullLong {
    const CommCtx &ctx;
    const PullArgs &a;
    PullShared &sh;
    PullLongWalk walk;
    uint32_t smem;
    int vr, rank, sources;
    bool packs, stores;

    __device__ __forceinline__ PullLong(const CommCtx &c, const PullArgs &args, PullShared &shared, uint32_t bufs)
        : ctx(c), a(args), sh(shared), walk{{args.bytes, args.stride}, static_cast<int>(gridDim.x),
                                            static_cast<int>(blockIdx.x), args.tile},
          smem(bufs), vr(static_cast<int>(blockIdx.y)), rank(c.rank + vr)
    {
        const bool bcast = a.root >= 0;
        packs = (!bcast || a.root == rank) && a.src[vr] != nullptr;
        stores = a.dst[vr] != nullptr;
        sources = !stores ? 0 : bcast ? (a.root == rank ? 0 : 1) : ctx.world - 1;
    }
    // starting with the next rank, so that peers do not all read the same GPU first
    __device__ __forceinline__ int source_at(int i) const
    {
        if (a.root >= 0) { return a.root; }
        const int p = rank + 1 + i;
        return p < ctx.world ? p : p - ctx.world;
    }
    __device__ __forceinline__ unsigned int vectors(int p, int k) const
    {
        const unsigned long long v0 = walk.first_vector(k), end = sh.blocks[p].nvec;
        return v0 >= end ? 0u : end - v0 < a.tile ? static_cast<unsigned int>(end - v0) : a.tile;
    }
    // two rounds of the tensor (a vector more: it may start anywhere in one), kPullDepth of all sources' pieces
    __device__ __forceinline__ uint32_t tensor(int k) const { return smem + (k & 1) * (a.tile + 1u) * 16u; }
    __device__ __forceinline__ uint32_t piece(int i, int k) const
    {
        return smem + (2u * (a.tile + 1u) + static_cast<unsigned int>(k % kPullDepth * sources + i) * a.tile) * 16u;
    }
    // where tile k lies in tensor memory (its first byte), and the aligned address that comes first in tensor(k)
    __device__ __forceinline__ unsigned long long tensor_at(int k) const
    {
        return reinterpret_cast<unsigned long long>(a.src[vr]) + 16ull * walk.first_vector(k) - sh.blocks[rank].phase;
    }

    __device__ __forceinline__ void load() const
    {
        if (!packs || (threadIdx.x & 31u) != 0u) { return; }
        const unsigned long long policy = evict_first_policy();
        const unsigned long long begin = reinterpret_cast<unsigned long long>(a.src[vr]) & ~15ull;
        const unsigned long long end = (reinterpret_cast<unsigned long long>(a.src[vr]) + a.bytes + 15ull) & ~15ull;
        for (int k = 0; k < a.rounds; ++k) {
            // whole aligned vectors that hold a byte of the tensor
            const unsigned int n = vectors(rank, k);
            const unsigned long long at = tensor_at(k), first = at & ~15ull;
            const unsigned long long lo = first > begin ? first : begin;
            const unsigned long long last = first + 16ull * n + (at != first ? 16ull : 0ull);
            const unsigned long long hi = last < end ? last : end;
            if (k >= 2 && !ring_wait(ctx, sh.dead, sh.packed, k - 2)) {
                drain(ctx, sh.tensor, k - 1);
                return;
            }
            ask_stream(sh.tensor.at(k), tensor(k) + static_cast<uint32_t>(lo - first), reinterpret_cast<const void *>(lo),
                       n != 0u && lo < hi ? static_cast<unsigned int>(hi - lo) : 0u, policy);
        }
    }

    __device__ __forceinline__ void fetch(int told) const
    {
        const int i = static_cast<int>(threadIdx.x & 31u);
        for (int t = 0; t < told; ++t) {
            const bool more = t < a.rounds;
            const unsigned int bytes = more && i < sources ? vectors(source_at(i), t) * 16u : 0u;
            const unsigned int all = __reduce_add_sync(0xffffffffu, bytes);
            const char *from = ctx.base[i < sources ? source_at(i) : rank] + a.off + walk.piece(t);
            const uint32_t to = piece(i, t);
            // (pass r + lag waits for round r)
            const int before = t - kPullDepth;
            bool ok = !more || before < 0 || (sources != 0 ? ring_wait(ctx, sh.dead, sh.stored, before)
                                                           : ring_wait(ctx, sh.dead, sh.done, before + kPullLag));
            if (ok && i < ctx.world) { ok = poll_acquire(ctx, rank, i, sh.epoch + static_cast<uint32_t>(t) + 1u, 0); }
            if (!warp_agrees(ok)) {
                ring_give_up(sh.dead);
                drain(ctx, sh.pieces, (t < a.rounds ? t : a.rounds) - 1);
                return;
            }
            if (!more) { continue; }
            fence_async_proxy_global();
            if (i == 0) { mbar_expect_tx(sh.pieces.at(t), all); }
            if (bytes != 0u) { bulk_load(to, from, bytes, sh.pieces.at(t)); }
        }
        if (i == 0) { pad_of(ctx, rank)->epoch[blockIdx.x] = sh.epoch + static_cast<uint32_t>(told); }
    }

    // Bytes of source p's tile t that its block has: from shared address `piece`, to where.
    struct Run {
        char *dst;
        uint32_t src;
        unsigned int n;
        // both start at the same byte of a vector
        __device__ __forceinline__ bool alike() const
        {
            return ((static_cast<uint32_t>(reinterpret_cast<unsigned long long>(dst)) ^ src) & 15u) == 0u;
        }
    };
    __device__ __forceinline__ Run run_of(int p, int t, uint32_t piece) const
    {
        const PullBlock &d = sh.blocks[p];
        const unsigned long long at = 16ull * walk.first_vector(t), end = a.bytes + d.phase;
        const unsigned long long lo = at < d.phase ? d.phase : at;
        const unsigned long long to = at + 16ull * a.tile, hi = to < end ? to : end;
        return Run{d.base + lo, piece + static_cast<uint32_t>(lo - at), lo < hi ? static_cast<unsigned int>(hi - lo) : 0u};
    }

    // Tile k of the own data: to the ring, and to its place in the own destination.
    __device__ __forceinline__ void pack(int k) const
    {
        const unsigned long long policy = evict_first_policy();
        const PullBlock &own = sh.blocks[rank];
        const unsigned long long v0 = walk.first_vector(k);
        const unsigned int odd = static_cast<unsigned int>(tensor_at(k) & 15ull);
        const unsigned int n = vectors(rank, k);
        char *to = ctx.base[rank] + a.off + walk.piece(k);
        const bool keeps = stores && own.base + own.phase != a.src[vr];  // else the own block is in place
        // all vectors but the block's ends, stored as they are packed
        const bool aligned = keeps && own.aligned;
#pragma unroll 2
        for (unsigned int i = threadIdx.x; i < n; i += kPullLongThreads) {
            const uint32_t at = tensor(k) + i * 16u;
            uint4 x = ld_shared_v4(at);
            if (odd != 0u) { x = shift_bytes(x, ld_shared_v4(at + 16u), odd); }
            st_arena_v4(to + i * 16u, x);
            if (aligned && own.whole(v0 + i, 1)) { st_stream_v4(own.base + (v0 + i) * 16ull, x, policy); }
        }
        if (!keeps) { return; }
        const Run run = run_of(rank, k, tensor(k) + odd);
        if (!aligned) {
            store_run(run.dst, run.src, run.n, threadIdx.x, kPullLongThreads, policy);
        } else if (n != 0u && (v0 == 0 || v0 + n == own.nvec)) {
            // the ends
            const unsigned int first = v0 == 0 ? (run.n < 16u - own.phase ? run.n : 16u - own.phase) : 0u;
            store_run(run.dst, run.src, first, threadIdx.x, kPullLongThreads, policy);
            if (v0 + n == own.nvec && n + v0 > 1) {
                const unsigned int last = (static_cast<unsigned int>(a.bytes + own.phase - 1ull) & 15u) + 1u;
                store_run(run.dst + run.n - last, run.src + run.n - last, last, threadIdx.x, kPullLongThreads, policy);
            }
        }
    }

    // The storer: a lane per source takes its tiles on to the destination.
    __device__ __forceinline__ void store() const
    {
        if (!stores || sources == 0) {
            warp_arrive(sh.left.at(0));
            return;
        }
        const int i = static_cast<int>(threadIdx.x & 31u);
        const unsigned long long policy = evict_first_policy();
        for (int t = 0; t < a.rounds; ++t) {
            if (!warp_agrees(ring_wait(ctx, sh.dead, sh.pieces, t))) {
                asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
                return;
            }
            if (i < sources) {
                const Run run = run_of(source_at(i), t, piece(i, t));
                if (run.n != 0u && run.alike()) {
                    const unsigned int to_vec = (16u - (run.src & 15u)) & 15u, head = to_vec < run.n ? to_vec : run.n;
                    const unsigned int whole = (run.n - head) & ~15u;
                    if (whole != 0u) {
                        asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;" ::"l"(
                                         run.dst + head),
                                     "r"(run.src + head), "r"(whole), "l"(policy)
                                     : "memory");
                    }
                    const char *bytes = static_cast<const char *>(__cvta_shared_to_generic(run.src));
                    for (unsigned int j = 0; j < head; ++j) { run.dst[j] = bytes[j]; }
                    for (unsigned int j = head + whole; j < run.n; ++j) { run.dst[j] = bytes[j]; }
                }
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            }
            warp_arrive(sh.stored.at(t));
        }
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        warp_arrive(sh.left.at(0));
    }

    __device__ __forceinline__ void work() const
    {
        const unsigned long long policy = evict_first_policy();
#pragma unroll 1
        for (int k = 0; k < a.rounds + kPullLag; ++k) {
            if (k < a.rounds && packs) {
                if (!ring_wait(ctx, sh.dead, sh.tensor, k)) { return; }
                pack(k);
                warp_arrive(sh.packed.at(k));
            }
            const int t = k - kPullLag;
            if (t >= 0 && !ring_wait(ctx, sh.dead, sh.pieces, t)) { return; }
            warp_arrive(sh.done.at(k));
            if (t >= 0 && sources != 0) {
                // what the storer cannot do
                for (int i = 0; i < sources; ++i) {
                    const Run run = run_of(source_at(i), t, piece(i, t));
                    if (!run.alike()) { store_run(run.dst, run.src, run.n, threadIdx.x, kPullLongThreads, policy); }
                }
                warp_arrive(sh.stored.at(t));
            }
        }
        warp_arrive(sh.left.at(0));
    }
};

__global__ void __launch_bounds__(kPullLongBlock, kPullLongPerSm)
    pull_long_kernel(const __grid_constant__ CommCtx ctx, const __grid_constant__ PullArgs a)
{
    extern __shared__ __align__(128) unsigned char bufs[];
    __shared__ __align__(16) PullShared sh;
    const PullLong pull(ctx, a, sh, smem_addr(bufs));
    const int tid = static_cast<int>(threadIdx.x);
    if (tid < ctx.world) { sh.blocks[tid] = pull_block(a, pull.walk, pull.vr, tid); }
    if (tid == 0) {
        sh.epoch = pad_of(ctx, pull.rank)->epoch[blockIdx.x];
        sh.dead = 0;
        sh.tensor.init(1u);
        sh.pieces.init(1u);
        sh.packed.init(kPullLongThreads / 32);
        sh.stored.init(kPullLongThreads / 32 + 1);
        sh.done.init(kPullLongThreads / 32);
        sh.left.init(kPullLongThreads / 32 + 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_proxy();
    }
    __syncthreads();
    // (the rings of the last tiles may only be reused when all have read them: the next
    // call uses the other slot, whose users of the call before this one are done)
    const int told = a.rounds + (a.end_barrier != 0 ? kPullLag : 0);
    if (tid < kPullLongThreads) {
        pull.work();
    } else if (tid < kPullLongThreads + 32) {
        pull.load();
    } else if (tid < kPullLongThreads + 64) {
        ring_tell(ctx, sh.dead, sh.epoch, sh.done, pull.rank, told, sh.left);
    } else if (tid < kPullLongThreads + 96) {
        pull.fetch(told);
    } else {
        pull.store();
    }
}

int launch_pull(const CommCtx &ctx, const PullArgs &a, int blocks, int vranks, void *stream)
{
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid(blocks, vranks, 1);
    const void *kernel = a.lng != 0 ? reinterpret_cast<const void *>(&pull_long_kernel)
                                    : reinterpret_cast<const void *>(&pull_kernel);
    const dim3 block(a.lng != 0 ? kPullLongBlock : kPullThreads);
    const size_t smem = a.lng != 0 ? pull_long_smem(pull_sources(ctx.world, a.root), a.tile) : 0u;
    if (smem != 0) {
        // the opt-in to more than 48 KB is per function and per device
        static std::atomic<bool> opted_in[64] = {};
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { dev = 0; }
        if (!opted_in[dev].load(std::memory_order_relaxed)) {
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       static_cast<int>(kPullLongSmem));
            if (e != cudaSuccess) { return static_cast<int>(e); }
            opted_in[dev].store(true, std::memory_order_relaxed);
        }
    }
    void *params[2] = {const_cast<CommCtx *>(&ctx), const_cast<PullArgs *>(&a)};
    if (vranks > 1) {
        return static_cast<int>(cudaLaunchCooperativeKernel(kernel, grid, block, params, smem, s));
    }
    return static_cast<int>(cudaLaunchKernel(kernel, grid, block, params, smem, s));
}
}  // namespace stdml::collective::cuda
