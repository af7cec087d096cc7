// The all-reduce of memory that the peers cannot see (ordinary tensors, single or
// a fused group), in ONE launch: the two-shot of ar_kernel.cuh, cut into rounds
// whose pack, reduce and unpack run one round apart from each other.
//
// What bounds it: bytes.  Pack -> barrier -> reduce -> barrier -> unpack over a whole
// staging slot moves every byte through HBM three times and leaves the links
// (or HBM) idle in turn.  Here a block goes through its part in rounds of a few tens of KB
// and its staging pieces form a ring of three that all rounds reuse, so that
// the whole ring (tens of MB over all blocks) stays in the L2: HBM sees
// the tensors' own bytes only.  The owner of a shard takes its own operand from the
// tensor itself and stores its own result there, which spares 1/world of the staging.
//
// Pass k of a block: pack tile k; wait until all ranks have packed tile k-1 and
// reduced tile k-2; reduce tile k-1 of the own shard and push it to the peers;
// arrive; unpack tile k-2.  One flag exchange per round, whose latency the
// pack and unpack beside it hide.
// Ring of three: tile k is packed over tile k-3, which the peers reduced and this rank unpacked in
// its pass k-1 at the latest.
//
// Tiles of the same round are neighbours in memory over the blocks: all blocks together
// work on one moving window per shard, which DRAM serves better than a
// contiguous span per block.
//
// Reduction order is rank-ascending and the wire type's rounding is applied
// to the own operand too: bit-identical to the other peer-load algorithms.
// The reference's counterpart is the chunked graph walk
// (src/stdml/collective/run_graph_pair_list_multi_thread.cpp:58-97 there).
#pragma once
#include "ar_kernel.cuh"
#include "copy.cuh"
#include "staged_walk.hpp"

namespace stdml::collective::cuda
{
// AllReduceArgs::debug_checks for this kernel: the slot is aligned and past the pad,
// the rings of all blocks fit into it, the rounds cover every shard, the table is in range.
template <int DT>
__device__ __forceinline__ bool staged_args_look_sane(const CommCtx &ctx, const StagedArgs &a,
                                                      const GroupEntry *tab, int blocks)
{
    bool ok = buffer_offset_ok(a.off) && a.off != 0ull && ctx.world > 1 && ctx.world <= kMaxRanks &&
              a.nvec > 0 && a.tile_shift >= kStagedStepShift && a.rounds > 0;
    ok = ok && ((static_cast<unsigned long long>(blocks) * kStagedRing * ctx.world) << a.tile_shift) *
                       16ull <= a.slot_bytes;
    for (int s = 0; ok && s < ctx.world; ++s) {
        ok = StagedWalk::shard_begin(a.nvec, ctx.world, s + 1) -
                 StagedWalk::shard_begin(a.nvec, ctx.world, s) <=
             (static_cast<unsigned long long>(blocks) * a.rounds) << a.tile_shift;
    }
    if (ok && tab != nullptr) {
        ok = a.ntable > 0 && tab[0].voff == 0;
        for (int i = threadIdx.x; ok && i < a.ntable; i += kStagedThreads) {
            ok = table_entry_in_range<DT>(tab, i, a.ntable, a.nvec);
        }
    }
    return __syncthreads_and(ok ? 1 : 0) != 0;
}

// What a round needs of one shard's tile, worked out once by one thread and read by
// all from shared memory.  `fast` vectors from src on (and to dst on) can be moved
// with aligned 16-byte accesses (32 bytes for f32 tensors with a 16-bit wire type);
// 0 of them: the tile touches several tensors, a ragged end or an odd address, and
// every vector looks for its own tensor between the entries first and last.
struct TileDesc {
    const char *src;
    char *dst;
    unsigned long long lo;
    unsigned int n, fast;
    int first, last;
};

// Vector i of a fast tile.
template <int DT>
__device__ __forceinline__ uint4 load_fast(const char *src, unsigned int i, bool user_f32,
                                           unsigned long long policy)
{
    if constexpr (Tr<DT>::is_half) {
        if (user_f32) {
            union {
                uint4 v[2];
                float f[8];
            } x;
            x.v[0] = ld_stream_v4(src + i * 32ull, policy);
            x.v[1] = ld_stream_v4(src + i * 32ull + 16, policy);
            VecU<DT> u;
#pragma unroll
            for (int j = 0; j < 8; ++j) { u.e[j] = Tr<DT>::narrow(x.f[j]); }
            return u.v;
        }
    }
    return ld_stream_v4(src + i * 16ull, policy);
}

template <int DT>
__device__ __forceinline__ void store_fast(char *dst, unsigned int i, bool user_f32,
                                           const uint4 &v, unsigned long long policy)
{
    if constexpr (Tr<DT>::is_half) {
        if (user_f32) {
            union {
                uint4 v[2];
                float f[8];
            } x;
            VecU<DT> u;
            u.v = v;
#pragma unroll
            for (int j = 0; j < 8; ++j) { x.f[j] = Tr<DT>::widen(u.e[j]); }
            st_stream_v4(dst + i * 32ull, x.v[0], policy);
            st_stream_v4(dst + i * 32ull + 16, x.v[1], policy);
            return;
        }
    }
    st_stream_v4(dst + i * 16ull, v, policy);
}

// Any vector of any tile.  Out of line: few tiles need it, and its code and registers
// would weigh on the loops of the many.
struct SlowTile {
    const GroupEntry *tab;
    const unsigned int *starts;  // first vectors of the entries, in shared memory (or null)
    const void *src;
    void *dst;
    unsigned long long count;
    int first, last;
    int user_f32;
};

// Entry that holds vector v, between the tile's first and last.
__device__ __forceinline__ const GroupEntry &slow_entry(const SlowTile &t, unsigned long long v)
{
    if (t.starts == nullptr) {
        return t.tab[t.first + find_entry(t.tab + t.first, t.last - t.first + 1, v)];
    }
    int lo = t.first, hi = t.last;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (t.starts[mid] <= static_cast<unsigned int>(v)) {
            lo = mid;
        } else {
            hi = mid - 1;
        }
    }
    return t.tab[lo];
}

template <int DT>
static __device__ __noinline__ uint4 load_slow(const SlowTile &t, unsigned long long v)
{
    if (t.tab == nullptr) {
        return load_user_vec<DT>(t.src, t.user_f32 != 0, v, t.count, ptr_aligned16(t.src));
    }
    const GroupEntry &e = slow_entry(t, v);
    return load_user_vec<DT>(e.src, t.user_f32 != 0, v - e.voff, e.count, ptr_aligned16(e.src));
}

template <int DT>
static __device__ __noinline__ void store_slow(const SlowTile &t, unsigned long long v, uint4 x)
{
    if (t.tab == nullptr) {
        store_user_vec<DT>(t.dst, t.user_f32 != 0, v, t.count, ptr_aligned16(t.dst), x);
        return;
    }
    const GroupEntry &e = slow_entry(t, v);
    store_user_vec<DT>(e.dst, t.user_f32 != 0, v - e.voff, e.count, ptr_aligned16(e.dst), x);
}

// Four blocks of 256 threads per SM: while one waits for its flags or drains its loads the
// others move bytes.  Measured, 102 MB of f32 in 161 tensors, 4 ranks, us per call
// (vectors per block and round over all shards): 256 threads 403 (1024), 354 (2048),
// 388 (4096: the rings, 117 MB, no longer fit the L2); 512 threads, two blocks: 368 (4096).
// Those with four vectors of a thread in flight in pack and unpack, whose registers spill
// around the out-of-line calls; two in flight 310, one (no spills) 300: the other 31 warps
// of the SM's share hide a load better than spilled registers do.  Three, five and six blocks
// per SM: 333, 367, 445.  The three-phase kernel took 457; with every vector looking for
// its own tensor (no tile descriptors) this one took 432.
template <int DT, int OP>
__global__ void __launch_bounds__(kStagedThreads, kStagedPerSm)
    staged_kernel(const __grid_constant__ CommCtx ctx, const __grid_constant__ StagedArgs a)
{
    __shared__ BlockSync sync;
    __shared__ unsigned long long bound[kMaxRanks + 1];
    __shared__ TileDesc descs[4][kMaxRanks];
    __shared__ unsigned int slow_shards[4];  // bit s: shard s's tile has vectors past the fast ones
    // first vectors of the table's entries, for the searches of every round
    __shared__ unsigned int starts[kStagedStarts];
    const int vr = static_cast<int>(blockIdx.y);
    const int rank = ctx.rank + vr;
    const int world = ctx.world;
    const StagedWalk walk{bound, world, static_cast<int>(gridDim.x), static_cast<int>(blockIdx.x),
                          a.tile_shift};
    const int rounds = a.rounds;
    const bool user_f32 = Tr<DT>::is_half && a.user_dtype == DT_F32;
    const GroupEntry *tab = a.table[vr];
    if (a.debug_checks != 0 &&
        !staged_args_look_sane<DT>(ctx, a, tab, static_cast<int>(gridDim.x))) {
        report_bad_args(ctx, rank);
        return;
    }
    sync_begin(ctx, rank, &sync);
    const unsigned long long policy = evict_first_policy();
    SlowTile slow;
    slow.tab = tab;
    slow.src = a.src[vr];
    slow.dst = a.dst[vr];
    slow.count = a.count;
    slow.first = slow.last = 0;
    slow.user_f32 = user_f32 ? 1 : 0;
    // a rank without a destination serves its shard for the others and stores nothing of its own
    const bool stores = tab != nullptr || slow.dst != nullptr;

    const bool searchable = tab != nullptr && a.ntable <= kStagedStarts && a.nvec >> 32 == 0;
    slow.starts = searchable ? starts : nullptr;
    auto entry_at = [&](unsigned long long v) {
        if (!searchable) { return find_entry(tab, a.ntable, v); }
        int lo = 0, hi = a.ntable - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (starts[mid] <= static_cast<unsigned int>(v)) {
                lo = mid;
            } else {
                hi = mid - 1;
            }
        }
        return lo;
    };
    // The tiles of round k (one thread of the last warp per shard), for whoever comes
    // after the next block sync.  Called for k + 1 after the wait of pass k, when
    // no thread looks at slot (k + 1) & 3 any more (tile k - 3's unpack was the last to).
    auto look_up = [&](int k) {
        const int s = static_cast<int>(threadIdx.x) - (kStagedThreads - 32);
        if (s < 0 || k >= rounds) { return; }
        StagedTile t{0, 0};
        if (s < world) { t = walk.tile_of(s, k); }
        TileDesc d;
        d.src = nullptr;
        d.dst = nullptr;
        d.lo = t.lo;
        d.n = static_cast<unsigned int>(t.hi - t.lo);
        d.fast = 0;
        d.first = d.last = 0;
        if (d.n > 0) {
            GroupEntry e;
            if (tab != nullptr) {
                d.first = entry_at(t.lo);
                d.last = entry_at(t.hi - 1);
                e = tab[d.first];
            } else {
                e.src = slow.src;
                e.dst = slow.dst;
                e.voff = 0;
                e.count = slow.count;
            }
            constexpr unsigned long long N = lanes_of<DT>();
            const unsigned long long at = t.lo - e.voff;
            const unsigned long long whole = e.count / N;  // without the ragged last vector
            if (ptr_aligned16(e.src) && ptr_aligned16(e.dst) && whole > at) {
                const unsigned long long left = whole - at;
                d.fast = left < d.n ? static_cast<unsigned int>(left) : d.n;
                const unsigned long long byte = at * (user_f32 ? 32ull : 16ull);
                d.src = static_cast<const char *>(e.src) + byte;
                d.dst = static_cast<char *>(e.dst) + byte;
                // Wanted in a pass from now (own shard: two).  161 f32 tensors, 4 ranks:
                // 299 -> 284 us; not for f32 tensors with a 16-bit wire type, whose tiles are
                // twice as long as their ring pieces and push the rings out of the L2
                // (435 -> 499 us).
                if (k > 0 && !user_f32) { prefetch_l2(d.src, d.fast * 16u); }
            }
        }
        if (s < world) { descs[k & 3][s] = d; }
        const unsigned int mask = __ballot_sync(0xffffffffu, d.fast < d.n && s != rank);
        if (s == 0) { slow_shards[k & 3] = mask; }
    };

    char *mine = ctx.base[rank] + a.off;
    // Pack and unpack go through the tiles of all the other shards in steps of kStagedThreads
    // vectors, a step inside one tile; everything about a step but the thread's own vector
    // is uniform over the block.  A thread takes the same vectors of a piece in every
    // round: tile k is packed right after tile k - 3 was unpacked from the same piece, with no
    // block sync between.
    const int per_tile = a.tile_shift - kStagedStepShift;  // log2 of the steps in a tile
    const int steps = (world - 1) << per_tile;
    auto shard_at = [&](int q) {
        const int i = q >> per_tile;
        return i + (i >= rank ? 1 : 0);
    };
    auto vector_at = [&](int q) {
        return (static_cast<unsigned int>(q & ((1 << per_tile) - 1)) << kStagedStepShift) + threadIdx.x;
    };
    auto piece_byte = [&](int sh, unsigned int i) {
        return ((static_cast<unsigned int>(sh) << a.tile_shift) + i) * 16u;
    };
    if (static_cast<int>(threadIdx.x) <= world) {
        bound[threadIdx.x] = StagedWalk::shard_begin(a.nvec, world, static_cast<int>(threadIdx.x));
    }
    if (searchable) {
        for (int i = static_cast<int>(threadIdx.x); i < a.ntable; i += kStagedThreads) {
            starts[i] = static_cast<unsigned int>(tab[i].voff);
        }
    }
    __syncthreads();
    look_up(0);
    __syncthreads();
    for (int k = 0; k <= rounds + 1; ++k) {
        if (k < rounds) {
            // ---- pack tile k of every shard but the own one
            char *to = mine + walk.piece(k, 0);
            const TileDesc *ds = descs[k & 3];
            for (int q = 0; q < steps; ++q) {
                const int s = shard_at(q);
                const TileDesc &d = ds[s];
                const unsigned int i = vector_at(q);
                if (i < d.fast) {
                    st_arena_v4(to + piece_byte(s, i), load_fast<DT>(d.src, i, user_f32, policy));
                }
            }
            for (int q = 0; slow_shards[k & 3] != 0u && q < steps; ++q) {
                const int s = shard_at(q);
                const TileDesc &d = ds[s];
                const unsigned int i = vector_at(q);
                if (i < d.fast || i >= d.n) { continue; }
                slow.first = d.first;
                slow.last = d.last;
                st_arena_v4(to + piece_byte(s, i), load_slow<DT>(slow, d.lo + i));
            }
        }
        if (k > 0 && !wait_all(ctx, rank, &sync, k)) { return; }
        look_up(k + 1);
        if (k > 0 && k <= rounds) {
            // ---- reduce tile k-1 of the own shard
            const TileDesc &d = descs[(k - 1) & 3][rank];
            const unsigned long long at = a.off + walk.piece(k - 1, rank);
            slow.first = d.first;
            slow.last = d.last;
            for (unsigned int i = threadIdx.x; i < d.n; i += kStagedThreads) {
                const unsigned long long byte = at + i * 16ull;
                const bool fast = i < d.fast;
                Accum<DT> acc;
                for (int r0 = 0; r0 < world; r0 += 4) {
                    uint4 x[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (r0 + j < world) {
                            if (r0 + j != rank) {
                                x[j] = ld_arena_v4(ctx.base[r0 + j] + byte);
                            } else if (fast) {
                                x[j] = load_fast<DT>(d.src, i, user_f32, policy);
                            } else {
                                x[j] = load_slow<DT>(slow, d.lo + i);
                            }
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (r0 + j < world) {
                            if (r0 + j == 0) {
                                acc.init(x[j]);
                            } else {
                                acc.template add<OP>(x[j]);
                            }
                        }
                    }
                }
                const uint4 res = acc.finish(a.scale, a.has_scale != 0);
                for (int r = 0; r < world; ++r) {
                    if (r != rank) { st_arena_v4(ctx.base[r] + byte, res); }
                }
                if (!stores) { continue; }
                if (fast) {
                    store_fast<DT>(d.dst, i, user_f32, res, policy);
                } else {
                    store_slow<DT>(slow, d.lo + i, res);
                }
            }
        }
        if (k <= rounds) { arrive_all(ctx, rank, &sync, k + 1); }
        if (k > 1 && stores) {
            // ---- unpack tile k-2 of every shard but the own one
            const char *from = mine + walk.piece(k - 2, 0);
            const TileDesc *ds = descs[(k - 2) & 3];
            for (int q = 0; q < steps; ++q) {
                const int s = shard_at(q);
                const TileDesc &d = ds[s];
                const unsigned int i = vector_at(q);
                if (i < d.fast) {
                    store_fast<DT>(d.dst, i, user_f32, ld_arena_v4(from + piece_byte(s, i)), policy);
                }
            }
            for (int q = 0; slow_shards[(k - 2) & 3] != 0u && q < steps; ++q) {
                const int s = shard_at(q);
                const TileDesc &d = ds[s];
                const unsigned int i = vector_at(q);
                if (i < d.fast || i >= d.n) { continue; }
                slow.first = d.first;
                slow.last = d.last;
                store_slow<DT>(slow, d.lo + i, ld_arena_v4(from + piece_byte(s, i)));
            }
        }
    }
    advance_epoch(&sync, rounds + 1);
    sync_end(ctx, rank, &sync);
}

template <int DT>
int launch_staged_ops(const CommCtx &ctx, const StagedArgs &a, int op, int blocks, int vranks,
                      cudaStream_t stream)
{
    auto go = [&](auto *kernel) {
        const dim3 grid(blocks, vranks, 1);
        // the rows of a loopback world wait on one another: all blocks resident at once
        if (vranks > 1) {
            void *params[2] = {const_cast<CommCtx *>(&ctx), const_cast<StagedArgs *>(&a)};
            return static_cast<int>(cudaLaunchCooperativeKernel(
                reinterpret_cast<const void *>(kernel), grid, dim3(kStagedThreads), params, 0, stream));
        }
        kernel<<<grid, kStagedThreads, 0, stream>>>(ctx, a);
        return static_cast<int>(cudaGetLastError());
    };
    switch (op) {
    case OP_SUM:
        return go(&staged_kernel<DT, OP_SUM>);
    case OP_MIN:
        return go(&staged_kernel<DT, OP_MIN>);
    case OP_MAX:
        return go(&staged_kernel<DT, OP_MAX>);
    case OP_PROD:
        return go(&staged_kernel<DT, OP_PROD>);
    case OP_XOR:
        if constexpr (!Tr<DT>::is_float) { return go(&staged_kernel<DT, OP_XOR>); }
        return -1;
    }
    return -1;
}
}  // namespace stdml::collective::cuda
