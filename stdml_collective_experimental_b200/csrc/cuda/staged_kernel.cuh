// The all-reduce of memory that the peers cannot see (ordinary tensors, single or
// a fused group), in ONE launch of any length: the two-shot of ar_kernel.cuh, cut into rounds
// whose pack, reduce and unpack run `lag` rounds apart from each other.
//
// What bounds it: bytes.  Pack -> barrier -> reduce -> barrier -> unpack over a whole
// staging slot moves every byte through HBM three times and leaves the links
// (or HBM) idle in turn.  Here a block goes through its part in rounds of 16 KB
// and its staging pieces form a small ring that all rounds reuse, so that
// the whole ring (tens of MB over all blocks) stays in the L2: HBM sees
// the tensors' own bytes only.  The owner of a shard takes its own operand from the
// tensor itself and stores its own result there, which spares 1/world of the staging.
// The ring's bytes still cross the L2 four times, and stores to it run at 7.4 TB/s (loads at 18): 161 f32
// tensors of 102 MB among 4 ranks of one GPU cannot go below 165 us (HBM alone: 125).
//
// Next to it: the way of a flag.  A fence that waits for the block's stores, the flag, its
// poll and the first load behind it take 4 to 8 us under load, longer than a round's
// bytes.  So the rounds of pack, reduce and unpack are kStagedLag apart, and nobody who moves bytes
// waits for any of that: three warps of their own look after it.  The loader finds each
// tile's tensor (a chain of dependent loads) and brings its bytes into shared memory by bulk copies; the
// teller fences and sets the flags; the fetcher polls the flags and brings the ring pieces of a round
// into shared memory.  The workers then have loads of shared memory and stores only:
// pass k packs tile k, reduces tile k - lag of the own shard and pushes it to the peers, unpacks tile
// k - 2 lag.  They sync with the other warps by mbarriers, and with each other not at all.
// Ring of 2 lag + 1: tile k is packed over tile k - 2 lag - 1, which this rank unpacked in its pass
// k - 1 and the peers reduced before the flags that the fetcher saw for that.
//
// Last: registers.  Nothing may spill: the polls empty the L1, so that a spilled value comes back from the L2.
//
// Measured among ranks of one GPU, us, against the kernel whose blocks packed, exchanged flags, reduced and
// unpacked by turns, a load per thread in flight, a launch per slot: 161 f32 tensors, 2 / 4 / 8 ranks
// 150 / 285 / 607, now 103 / 239 / 507 (4 ranks, inputs that change: 287, 245); BERT-base as bf16 wire, 2 ranks 437, now
// 335 (438, 344).  Messages of a few rounds, which gain nothing: staged_oneshot_limit.  By lag, 4 ranks: 1: 398, 2: 249,
// 3: 242 (a lag of 1 with the polls and fences in the workers' own warps 380).
// By workers 128 / 192 / 256 of 3 blocks per SM: 253 / 243 / 242 (f32), 373 / 328 / 345 (bf16 wire).
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
#include "ring_sync.cuh"
#include "staged_walk.hpp"

#include <atomic>

namespace stdml::collective::cuda
{
// AllReduceArgs::debug_checks for this kernel: the slot is aligned and past the pad,
// the rings of all blocks fit into it, the rounds cover every shard, the table is in range.
template <int DT>
__device__ __forceinline__ bool staged_args_look_sane(const CommCtx &ctx, const StagedArgs &a,
                                                      const GroupEntry *tab, int blocks)
{
    bool ok = buffer_offset_ok(a.off) && a.off != 0ull && ctx.world > 1 && ctx.world <= kMaxRanks &&
              a.nvec > 0 && a.tile_shift >= kStagedMinShift && a.rounds > 0;
    ok = ok && ((static_cast<unsigned long long>(blocks) * kStagedRing * ctx.world) << a.tile_shift) *
                       16ull <= a.slot_bytes;
    for (int s = 0; ok && s < ctx.world; ++s) {
        ok = StagedWalk::shard_begin(a.nvec, ctx.world, s + 1) -
                 StagedWalk::shard_begin(a.nvec, ctx.world, s) <=
             (static_cast<unsigned long long>(blocks) * a.rounds) << a.tile_shift;
    }
    if (ok && tab != nullptr) {
        ok = a.ntable > 0 && tab[0].voff == 0;
        for (int i = threadIdx.x; ok && i < a.ntable; i += kStagedBlock) {
            ok = table_entry_in_range<DT>(tab, i, a.ntable, a.nvec);
        }
    }
    return __syncthreads_and(ok ? 1 : 0) != 0;
}

__device__ __forceinline__ bool staged_searchable(const StagedArgs &a)
{
    return a.ntable <= kStagedStarts && a.nvec >> 32 == 0;
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

__device__ __forceinline__ void *generic_of(uint32_t at) { return __cvta_shared_to_generic(at); }

// Vector i of a tile of tensor memory (ring pieces: user_f32 is false) at shared address `from`.
template <int DT>
__device__ __forceinline__ uint4 load_fast(uint32_t from, unsigned int i, bool user_f32)
{
    if constexpr (Tr<DT>::is_half) {
        if (user_f32) {
            union {
                uint4 v[2];
                float f[8];
            } x;
            x.v[0] = ld_shared_v4(from + i * 32u);
            x.v[1] = ld_shared_v4(from + i * 32u + 16u);
            VecU<DT> u;
#pragma unroll
            for (int j = 0; j < 8; ++j) { u.e[j] = Tr<DT>::narrow(x.f[j]); }
            return u.v;
        }
    }
    return ld_shared_v4(from + i * 16u);
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

// Vectors past a tile's fast ones, one at a time.  In line, and element by element where a vector
// is not whole: a call, or a vector put together in registers, makes the loops of the many spill,
// and what is spilled comes back from the L2, since the flags' acquires empty the L1 (161 f32 tensors, 4
// ranks: 387 us with calls, 286 without).
struct SlowVec {
    const char *src;  // the tensor's memory (elements of the user's type)
    char *dst;
    unsigned long long first, count;  // the vector's first element, the tensor's elements
};

// What holds vector i of tile d.
template <int DT>
__device__ __forceinline__ SlowVec slow_vec(const StagedArgs &a, int vr, const unsigned int *starts,
                                            const TileDesc &d, unsigned int i)
{
    const unsigned long long v = d.lo + i;
    const GroupEntry *tab = a.table[vr];
    SlowVec s{static_cast<const char *>(a.src[vr]), static_cast<char *>(a.dst[vr]), v, a.count};
    if (tab != nullptr) {
        int lo = d.first, hi = d.last;
        const bool searchable = staged_searchable(a);
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if ((searchable ? starts[mid] : tab[mid].voff) <= v) {
                lo = mid;
            } else {
                hi = mid - 1;
            }
        }
        s.src = static_cast<const char *>(tab[lo].src);
        s.dst = static_cast<char *>(tab[lo].dst);
        s.first = v - tab[lo].voff;
        s.count = tab[lo].count;
    }
    s.first *= lanes_of<DT>();
    return s;
}

// The elements of a vector that is not whole, eight at a time: one after the other they cost a memory latency
// each (187 ragged bf16 tensors, 3 ranks 22.7 us, so 19.6; four at a time 20.6).
template <int N, typename Load, typename Store>
__device__ __forceinline__ void copy_elements(Load load, Store store)
{
    constexpr int B = N < 8 ? N : 8;
#pragma unroll 1
    for (int i = 0; i < N; i += B) {
        decltype(load(0)) x[B];
#pragma unroll
        for (int j = 0; j < B; ++j) { x[j] = load(i + j); }
#pragma unroll
        for (int j = 0; j < B; ++j) { store(i + j, x[j]); }
    }
}

// The vector in the wire type, to `to` (elements past the tensor's end: zero).
template <int DT>
__device__ __forceinline__ void slow_load(const SlowVec &s, bool user_f32, void *to)
{
    using S = typename Tr<DT>::storage;
    constexpr int N = lanes_of<DT>();
    S *out = static_cast<S *>(to);
    if constexpr (Tr<DT>::is_half) {
        if (user_f32) {
            const float *f = reinterpret_cast<const float *>(s.src) + s.first;
            if (ptr_aligned16(f) && s.first + N <= s.count) {
#pragma unroll
                for (int i = 0; i < N; i += 4) {
                    const float4 x = *reinterpret_cast<const float4 *>(f + i);
                    const S e[4] = {Tr<DT>::narrow(x.x), Tr<DT>::narrow(x.y), Tr<DT>::narrow(x.z), Tr<DT>::narrow(x.w)};
                    *reinterpret_cast<uint2 *>(out + i) =
                        make_uint2(e[0] | static_cast<uint32_t>(e[1]) << 16, e[2] | static_cast<uint32_t>(e[3]) << 16);
                }
                return;
            }
            copy_elements<N>([&](int i) { return s.first + i < s.count ? Tr<DT>::narrow(f[i]) : S(0); },
                             [&](int i, S x) { out[i] = x; });
            return;
        }
    }
    const S *p = reinterpret_cast<const S *>(s.src) + s.first;
    if (ptr_aligned16(p) && s.first + N <= s.count) {
        *reinterpret_cast<uint4 *>(out) = *reinterpret_cast<const uint4 *>(p);
        return;
    }
    copy_elements<N>([&](int i) { return s.first + i < s.count ? p[i] : S(0); }, [&](int i, S x) { out[i] = x; });
}

// A vector of the wire type in shared memory to the tensor.
template <int DT>
__device__ __forceinline__ void slow_store(const SlowVec &s, bool user_f32, const void *from)
{
    using S = typename Tr<DT>::storage;
    constexpr int N = lanes_of<DT>();
    const S *in = static_cast<const S *>(from);
    const int n = s.first + N <= s.count ? N : static_cast<int>(s.count - s.first);
    if constexpr (Tr<DT>::is_half) {
        if (user_f32) {
            float *f = reinterpret_cast<float *>(s.dst) + s.first;
            if (ptr_aligned16(f) && n == N) {
#pragma unroll
                for (int i = 0; i < N; i += 4) {
                    const uint2 e = *reinterpret_cast<const uint2 *>(in + i);
                    *reinterpret_cast<float4 *>(f + i) =
                        make_float4(Tr<DT>::widen(static_cast<S>(e.x)), Tr<DT>::widen(static_cast<S>(e.x >> 16)),
                                    Tr<DT>::widen(static_cast<S>(e.y)), Tr<DT>::widen(static_cast<S>(e.y >> 16)));
                }
                return;
            }
            copy_elements<N>([&](int i) { return in[i]; },
                             [&](int i, S x) {
                                 if (i < n) { f[i] = Tr<DT>::widen(x); }
                             });
            return;
        }
    }
    S *p = reinterpret_cast<S *>(s.dst) + s.first;
    if (ptr_aligned16(p) && n == N) {
        *reinterpret_cast<uint4 *>(p) = *reinterpret_cast<const uint4 *>(in);
        return;
    }
    copy_elements<N>([&](int i) { return in[i]; },
                     [&](int i, S x) {
                         if (i < n) { p[i] = x; }
                     });
}

constexpr int kStagedUnroll = 4;  // vectors of a worker in flight, shared memory to global
constexpr int kStagedDescs = 8;  // rounds whose tiles somebody may look at, from the load to the unpack
static_assert(kStagedDescs >= 2 * kStagedLag + 2, "descriptors of all rounds under way");

// Tile buffers of a block's shared memory: tensor tiles of the other shards; two rounds of the own
// shard's and of the peers' ring pieces of it (operands); ring pieces of the other shards (results).
struct StagedBuffers {
    uint32_t base;
    unsigned int others;      // world - 1
    unsigned int unit_tile;   // bytes of a tile in tensor memory
    unsigned int piece;       // bytes of a ring piece
    int rank;

    __device__ __forceinline__ unsigned int slot(int s) const
    {
        return static_cast<unsigned int>(s - (s > rank ? 1 : 0));
    }
    __device__ __forceinline__ uint32_t tensor(int s) const { return base + slot(s) * unit_tile; }
    __device__ __forceinline__ uint32_t own(int t) const { return base + (others + (t & 1)) * unit_tile; }
    __device__ __forceinline__ uint32_t operand(int r, int t) const
    {
        return base + (others + 2u) * unit_tile + ((t & 1) * others + slot(r)) * piece;
    }
    __device__ __forceinline__ uint32_t result(int s) const
    {
        return base + (others + 2u) * unit_tile + (2u * others + slot(s)) * piece;
    }
};

// What the warps of a block share.
struct StagedShared {
    TileDesc descs[kStagedDescs][kMaxRanks];
    int whole[kStagedDescs];  // all tiles of the round are whole and fast
    unsigned long long bound[kMaxRanks + 1];
    // A round's bytes are there: the tensor's, of the other shards and of the own one; the
    // peers' operands of the own shard; the results of the other shards.
    Phases<1> tensor;
    Phases<2> own, operands;
    Phases<1> results;
    // The workers are done with them.  `reduced` counts passes: everything that
    // pass k packs and reduces is stored.
    Phases<1> packed, unpacked;
    Phases<4> reduced;
    Phases<1> left;  // the workers have come through
    uint32_t epoch;
    int dead;  // the block gives up
    // first vectors of the table's entries, for the searches of every round
    unsigned int starts[kStagedStarts];
};
static_assert(other_smem(sizeof(StagedShared)) <= kStagedOtherSmem, "the blocks that staged_per_sm() promises fit an SM");
static_assert(kStagedLag <= 3, "passes that the workers may be ahead of the warp that tells the peers");

// The loader warp: a lane per shard finds the tensor of each of its tiles, a chain of dependent
// loads, and asks for the tile's bytes as soon as the buffer is free.
template <int DT>
__device__ __forceinline__ void staged_load(const CommCtx &ctx, const StagedArgs &a, StagedShared &sh,
                                            const StagedWalk &walk, const StagedBuffers &bufs, int vr)
{
    const int s = static_cast<int>(threadIdx.x & 31u);
    const int world = ctx.world, rank = bufs.rank;
    const unsigned long long policy = evict_first_policy();
    const unsigned int unit = Tr<DT>::is_half && a.user_dtype == DT_F32 ? 32u : 16u;
    const GroupEntry *tab = a.table[vr];
    const bool searchable = tab != nullptr && staged_searchable(a);
    auto entry_at = [&](unsigned long long v) {
        if (!searchable) { return find_entry(tab, a.ntable, v); }
        int lo = 0, hi = a.ntable - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sh.starts[mid] <= static_cast<unsigned int>(v)) {
                lo = mid;
            } else {
                hi = mid - 1;
            }
        }
        return lo;
    };
    int asked = -1, asked_own = -1;  // last rounds asked for
    for (int k = 0; k < a.rounds + kStagedLag - 1 || k < 2; ++k) {
        TileDesc d;
        d.src = nullptr;
        d.dst = nullptr;
        d.fast = d.n = 0;
        d.lo = 0;
        d.first = d.last = 0;
        if (s < world && k < a.rounds) {
            const StagedTile t = walk.tile_of(s, k);
            d.lo = t.lo;
            d.n = static_cast<unsigned int>(t.hi - t.lo);
        }
        if (d.n > 0) {
            GroupEntry e;
            if (tab != nullptr) {
                d.first = entry_at(d.lo);
                d.last = entry_at(d.lo + d.n - 1);
                e = tab[d.first];
            } else {
                e.src = a.src[vr];
                e.dst = a.dst[vr];
                e.voff = 0;
                e.count = a.count;
            }
            constexpr unsigned long long N = lanes_of<DT>();
            const unsigned long long at = d.lo - e.voff;
            const unsigned long long whole = e.count / N;  // without the ragged last vector
            if (ptr_aligned16(e.src) && ptr_aligned16(e.dst) && whole > at) {
                const unsigned long long left = whole - at;
                d.fast = left < d.n ? static_cast<unsigned int>(left) : d.n;
                d.src = static_cast<const char *>(e.src) + at * unit;
                d.dst = static_cast<char *>(e.dst) + at * unit;
            }
        }
        bool ok = true;
        if (k > 0 && k < a.rounds) { ok = warp_agrees(ring_wait(ctx, sh.dead, sh.packed, k - 1)); }
        if (ok && k < a.rounds) {
            if (s < world) { sh.descs[k % kStagedDescs][s] = d; }
            const bool whole = warp_agrees(s >= world || d.fast == 1u << a.tile_shift);
            if (s == 0) { sh.whole[k % kStagedDescs] = whole ? 1 : 0; }
            ask_stream(sh.tensor.at(k), bufs.tensor(s), d.src, s != rank ? d.fast * unit : 0u, policy);
            asked = k;
        }
        // The own tiles, the first two of them at once: pass k - 1 reduced the one that was in the buffer.
        const int t = k < 2 ? k : k - kStagedLag + 1;
        if (ok && t < a.rounds && (k < 2 || t >= 2)) {
            ok = k < 2 || warp_agrees(ring_wait(ctx, sh.dead, sh.reduced, k - 1));
            if (ok && s == rank) {
                const TileDesc &o = sh.descs[t % kStagedDescs][rank];
                ask_stream(sh.own.at(t), bufs.own(t), o.src, o.fast * unit, policy);
            }
            if (ok) { asked_own = t; }
        }
        if (!ok) {
            drain(ctx, sh.tensor, asked);
            drain(ctx, sh.own, asked_own);
            return;
        }
    }
}

// The fetcher: waits until all ranks have packed tile t and reduced tile t - lag, and asks for the pieces
// that pass t + lag reduces and unpacks.  A lane per rank or shard; all that can be known
// before the wait is worked out before it.
__device__ __forceinline__ void staged_fetch(const CommCtx &ctx, const StagedArgs &a, StagedShared &sh,
                                             const StagedWalk &walk, const StagedBuffers &bufs, bool stores)
{
    const int p = static_cast<int>(threadIdx.x & 31u);
    const int rank = bufs.rank;
    const bool peer = p < ctx.world && p != rank;
    const char *theirs = ctx.base[peer ? p : rank] + a.off, *mine = ctx.base[rank] + a.off;
    const int passes = a.rounds + kStagedLag;
    auto bytes_of = [&](int s, int t) {
        const StagedTile tile = walk.tile_of(s, t);
        return static_cast<unsigned int>(tile.hi - tile.lo) * 16u;
    };
    int asked_op = -1, asked_res = -1;  // last rounds asked for
    for (int t = 0; t < passes; ++t) {
        const int u = t - kStagedLag;
        const bool reduces = t < a.rounds, unpacks = u >= 0 && stores;
        const unsigned int n_op = reduces ? bytes_of(rank, t) : 0u;
        const unsigned int n_res = unpacks && peer ? bytes_of(p, u) : 0u;
        const unsigned int all_res = __reduce_add_sync(0xffffffffu, n_res);
        const char *from_op = theirs + walk.piece(t, rank), *from_res = mine + walk.piece(u < 0 ? 0 : u, peer ? p : rank);
        const uint32_t to_op = bufs.operand(p, t), to_res = bufs.result(p);
        bool ok = !reduces || t < 2 || ring_wait(ctx, sh.dead, sh.reduced, t - 2 + kStagedLag);
        if (ok && p < ctx.world) { ok = poll_acquire(ctx, rank, p, sh.epoch + static_cast<uint32_t>(t) + 1u, 0); }
        ok = warp_agrees(ok);
        fence_async_proxy_global();
        if (ok && reduces) {
            if (p == 0) { mbar_expect_tx(sh.operands.at(t), n_op * bufs.others); }
            if (peer && n_op != 0u) { bulk_load(to_op, from_op, n_op, sh.operands.at(t)); }
            asked_op = t;
        }
        if (ok && unpacks) {
            ok = u < 1 || warp_agrees(ring_wait(ctx, sh.dead, sh.unpacked, u - 1));
            if (ok && p == 0) { mbar_expect_tx(sh.results.at(u), all_res); }
            if (ok && n_res != 0u) { bulk_load(to_res, from_res, n_res, sh.results.at(u)); }
            if (ok) { asked_res = u; }
        }
        if (!ok) {
            ring_give_up(sh.dead);
            drain(ctx, sh.operands, asked_op);
            drain(ctx, sh.results, asked_res);
            return;
        }
    }
    if (p == 0) { pad_of(ctx, rank)->epoch[blockIdx.x] = sh.epoch + static_cast<uint32_t>(passes); }
}

// What a worker needs to know.  Made anew from the special registers in every phase of a pass,
// so that nothing of it takes a register in between.
template <int DT>
struct StagedWorker {
    const CommCtx &ctx;
    const StagedArgs &a;
    StagedShared &sh;
    unsigned int tid;
    int vr, rank;
    bool user_f32;
    StagedBuffers bufs;

    __device__ __forceinline__ StagedWorker(const CommCtx &c, const StagedArgs &args, StagedShared &shared,
                                            uint32_t smem)
        : ctx(c), a(args), sh(shared)
    {
        asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
        asm volatile("mov.u32 %0, %%ctaid.y;" : "=r"(vr));
        rank = ctx.rank + vr;
        user_f32 = Tr<DT>::is_half && a.user_dtype == DT_F32;
        bufs = StagedBuffers{smem, static_cast<unsigned int>(ctx.world - 1),
                             (user_f32 ? 32u : 16u) << a.tile_shift, 16u << a.tile_shift, rank};
    }
    __device__ __forceinline__ StagedWalk walk() const
    {
        return StagedWalk{sh.bound, ctx.world, static_cast<int>(gridDim.x), static_cast<int>(blockIdx.x), a.tile_shift};
    }
    // a rank without a destination serves its shard for the others and stores nothing of its own
    __device__ __forceinline__ bool stores() const { return a.table[vr] != nullptr || a.dst[vr] != nullptr; }
    // vectors of the tiles of all the other shards
    __device__ __forceinline__ unsigned int others() const { return bufs.others << a.tile_shift; }

    // Calls f(s, i) for all of them, kStagedThreads at a time; a warp's vectors lie in one tile.
    template <typename F>
    __device__ __forceinline__ void for_others(F f) const
    {
#pragma unroll 1
        for (unsigned int j = tid; j < others(); j += kStagedThreads) {
            const int s = static_cast<int>(j >> a.tile_shift);
            f(s + (s >= rank ? 1 : 0), j & ((1u << a.tile_shift) - 1u));
        }
    }
};

// Every phase below has two forms: for a round all of whose tiles are whole and fast, in which a
// vector costs little more than its load and its store (what bounds the kernel after its
// bytes is instructions: 180 a warp and vector in the other form alone, 54 % of the issue slots), and for any.

// Tile k of every shard but the own one, to the ring.  False: the block gives up.
template <int DT>
__device__ __forceinline__ bool staged_pack(const CommCtx &ctx, const StagedArgs &a, StagedShared &sh, uint32_t smem,
                                            int k)
{
    if (!ring_wait(ctx, sh.dead, sh.tensor, k)) { return false; }
    const StagedWorker<DT> w(ctx, a, sh, smem);
    char *to = ctx.base[w.rank] + a.off + w.walk().piece(k, 0);
    if (sh.whole[k % kStagedDescs] != 0) {
        const unsigned int n = w.others(), own = static_cast<unsigned int>(w.rank) << a.tile_shift;
        const uint32_t from = w.bufs.base;  // tile after tile
#pragma unroll kStagedUnroll
        for (unsigned int j = w.tid; j < n; j += kStagedThreads) {
            // (in the ring the own shard has a piece too)
            st_arena_v4(to + (j + (j >= own ? 1u << a.tile_shift : 0u)) * 16u, load_fast<DT>(from, j, w.user_f32));
        }
    } else {
        const TileDesc *ds = sh.descs[k % kStagedDescs];
        w.for_others([&](int s, unsigned int i) {
            char *at = to + ((static_cast<unsigned int>(s) << a.tile_shift) + i) * 16u;
            if (i < ds[s].fast) {
                st_arena_v4(at, load_fast<DT>(w.bufs.tensor(s), i, w.user_f32));
            } else if (i < ds[s].n) {
                slow_load<DT>(slow_vec<DT>(a, w.vr, sh.starts, ds[s], i), w.user_f32, at);
            }
        });
    }
    warp_arrive(sh.packed.at(k));
    return true;
}

// Vector i of the own shard's tile t: the ranks' operands, in ascending order, to the result.
// `own`: the vector of the own operand.
template <int DT, int OP>
__device__ __forceinline__ uint4 staged_sum(const StagedWorker<DT> &w, int t, unsigned int i, const uint4 &own)
{
    Accum<DT> acc;
    const int world = w.ctx.world;
    const uint32_t from = w.bufs.operand(0, t) + i * 16u;
#pragma unroll 1
    for (int r0 = 0; r0 < world; r0 += 4) {
        uint4 x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = r0 + j;
            if (r < world) { x[j] = r == w.rank ? own : ld_shared_v4(from + w.bufs.slot(r) * w.bufs.piece); }
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
    return acc.finish(w.a.scale, w.a.has_scale != 0);
}

// Tile t of the own shard: reduced, to every peer's ring and the own tensor.
template <int DT, int OP>
__device__ __forceinline__ bool staged_reduce(const CommCtx &ctx, const StagedArgs &a, StagedShared &sh, uint32_t smem,
                                              int t)
{
    if (!ring_wait(ctx, sh.dead, sh.own, t)) { return false; }
    const StagedWorker<DT> w(ctx, a, sh, smem);
    const unsigned long long policy = evict_first_policy();
    const TileDesc &d = sh.descs[t % kStagedDescs][w.rank];
    const unsigned long long at = a.off + w.walk().piece(t, w.rank);
    const uint32_t own = w.bufs.own(t);
    const unsigned int fast = d.fast, n = d.n, unit = w.user_f32 ? 32u : 16u;
    // Slow vectors: the own operand, then the result, by way of the own tile's buffer, in the wire type.  Their
    // chains of loads run while the peers' operands are on their way.
#pragma unroll 1
    for (unsigned int i = w.tid; fast < n && i < n; i += kStagedThreads) {
        if (i >= fast) { slow_load<DT>(slow_vec<DT>(a, w.vr, sh.starts, d, i), w.user_f32, generic_of(own + i * unit)); }
    }
    if (!ring_wait(ctx, sh.dead, sh.operands, t)) { return false; }
#pragma unroll 1
    for (unsigned int i = w.tid; i < n; i += kStagedThreads) {
        const uint32_t here = own + i * unit;
        const uint4 res = staged_sum<DT, OP>(w, t, i, i < fast ? load_fast<DT>(own, i, w.user_f32) : ld_shared_v4(here));
#pragma unroll 4
        for (int r = 0; r < ctx.world; ++r) {
            if (r != w.rank) { st_arena_v4(ctx.base[r] + at + i * 16u, res); }
        }
        if (i >= fast) {
            *static_cast<uint4 *>(generic_of(here)) = res;
            if (w.stores()) { slow_store<DT>(slow_vec<DT>(a, w.vr, sh.starts, d, i), w.user_f32, generic_of(here)); }
            // a bulk copy comes over these writes next
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        } else if (w.stores()) {
            store_fast<DT>(d.dst, i, w.user_f32, res, policy);
        }
    }
    return true;
}

// Tile t of every shard but the own one, from the ring to the tensors.
template <int DT>
__device__ __forceinline__ bool staged_unpack(const CommCtx &ctx, const StagedArgs &a, StagedShared &sh, uint32_t smem,
                                              int t)
{
    if (!ring_wait(ctx, sh.dead, sh.results, t)) { return false; }
    const StagedWorker<DT> w(ctx, a, sh, smem);
    const unsigned long long policy = evict_first_policy();
    const TileDesc *ds = sh.descs[t % kStagedDescs];
    if (sh.whole[t % kStagedDescs] != 0) {
        const unsigned int n = w.others(), in_tile = (1u << a.tile_shift) - 1u;
        const uint32_t from = w.bufs.result(0);
#pragma unroll kStagedUnroll
        for (unsigned int j = w.tid; j < n; j += kStagedThreads) {
            const int s = static_cast<int>(j >> a.tile_shift);
            store_fast<DT>(ds[s + (s >= w.rank ? 1 : 0)].dst, j & in_tile, w.user_f32, ld_shared_v4(from + j * 16u), policy);
        }
    } else {
        w.for_others([&](int s, unsigned int i) {
            const uint32_t from = w.bufs.result(s) + i * 16u;
            if (i < ds[s].fast) {
                store_fast<DT>(ds[s].dst, i, w.user_f32, ld_shared_v4(from), policy);
            } else if (i < ds[s].n) {
                slow_store<DT>(slow_vec<DT>(a, w.vr, sh.starts, ds[s], i), w.user_f32, generic_of(from));
            }
        });
    }
    warp_arrive(sh.unpacked.at(t));
    return true;
}

template <int DT, int OP>
__global__ void __launch_bounds__(kStagedBlock, kStagedMinPerSm)
    staged_kernel(const __grid_constant__ CommCtx ctx, const __grid_constant__ StagedArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(16) StagedShared sh;
    const int vr = static_cast<int>(blockIdx.y);
    const int rank = ctx.rank + vr;
    const int tid = static_cast<int>(threadIdx.x);
    const GroupEntry *tab = a.table[vr];
    if (a.debug_checks != 0 &&
        !staged_args_look_sane<DT>(ctx, a, tab, static_cast<int>(gridDim.x))) {
        report_bad_args(ctx, rank);
        return;
    }
    if (tid == 0) {
        sh.epoch = pad_of(ctx, rank)->epoch[blockIdx.x];
        sh.dead = 0;
        sh.tensor.init(32u);
        sh.own.init(1u);
        sh.operands.init(1u);
        sh.results.init(1u);
        sh.packed.init(kStagedThreads / 32);
        sh.reduced.init(kStagedThreads / 32);
        sh.unpacked.init(kStagedThreads / 32);
        sh.left.init(kStagedThreads / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_proxy();
    }
    if (tid <= ctx.world) { sh.bound[tid] = StagedWalk::shard_begin(a.nvec, ctx.world, tid); }
    if (tab != nullptr && staged_searchable(a)) {
        for (int i = tid; i < a.ntable; i += kStagedBlock) {
            sh.starts[i] = static_cast<unsigned int>(tab[i].voff);
        }
    }
    __syncthreads();

    const StagedWalk walk{sh.bound, ctx.world, static_cast<int>(gridDim.x), static_cast<int>(blockIdx.x),
                          a.tile_shift};
    const bool user_f32 = Tr<DT>::is_half && a.user_dtype == DT_F32;
    const StagedBuffers bufs{smem_addr(smem), static_cast<unsigned int>(ctx.world - 1),
                             (user_f32 ? 32u : 16u) << a.tile_shift, 16u << a.tile_shift, rank};
    // a rank without a destination serves its shard for the others and stores nothing of its own
    const bool stores = tab != nullptr || a.dst[vr] != nullptr;
    if (tid >= kStagedThreads) {
        const int role = (tid - kStagedThreads) / 32;
        if (role == 0) { staged_load<DT>(ctx, a, sh, walk, bufs, vr); }
        if (role == 1) { ring_tell(ctx, sh.dead, sh.epoch, sh.reduced, rank, a.rounds + kStagedLag, sh.left); }
        if (role == 2) { staged_fetch(ctx, a, sh, walk, bufs, stores); }
        return;
    }

    // ---- the workers
#pragma unroll 1
    for (int k = 0; k < a.rounds + 2 * kStagedLag; ++k) {
        if (k < a.rounds && !staged_pack<DT>(ctx, a, sh, smem_addr(smem), k)) { return; }
        if (k < a.rounds + kStagedLag) {
            if (k >= kStagedLag && !staged_reduce<DT, OP>(ctx, a, sh, smem_addr(smem), k - kStagedLag)) { return; }
            warp_arrive(sh.reduced.at(k));
        }
        if (k >= 2 * kStagedLag && stores && !staged_unpack<DT>(ctx, a, sh, smem_addr(smem), k - 2 * kStagedLag)) {
            return;
        }
    }
    warp_arrive(sh.left.at(0));
}

template <int DT, int OP>
int launch_staged_op(const CommCtx &ctx, const StagedArgs &a, int blocks, int vranks, cudaStream_t stream)
{
    const void *kernel = reinterpret_cast<const void *>(&staged_kernel<DT, OP>);
    // the opt-in to more than 48 KB (with the static part) is per function and per device
    static std::atomic<bool> opted_in[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { dev = 0; }
    if (!opted_in[dev].load(std::memory_order_relaxed)) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(kStagedSmem));
        if (e != cudaSuccess) { return static_cast<int>(e); }
        opted_in[dev].store(true, std::memory_order_relaxed);
    }
    const dim3 grid(blocks, vranks, 1);
    const dim3 block(kStagedBlock);
    const size_t smem = staged_smem(ctx.world, a.tile_shift, Tr<DT>::is_half && a.user_dtype == DT_F32);
    void *params[2] = {const_cast<CommCtx *>(&ctx), const_cast<StagedArgs *>(&a)};
    // the rows of a loopback world wait on one another: all blocks resident at once
    if (vranks > 1) {
        return static_cast<int>(cudaLaunchCooperativeKernel(kernel, grid, block, params, smem, stream));
    }
    return static_cast<int>(cudaLaunchKernel(kernel, grid, block, params, smem, stream));
}

template <int DT>
int launch_staged_ops(const CommCtx &ctx, const StagedArgs &a, int op, int blocks, int vranks,
                      cudaStream_t stream)
{
    switch (op) {
    case OP_SUM:
        return launch_staged_op<DT, OP_SUM>(ctx, a, blocks, vranks, stream);
    case OP_MIN:
        return launch_staged_op<DT, OP_MIN>(ctx, a, blocks, vranks, stream);
    case OP_MAX:
        return launch_staged_op<DT, OP_MAX>(ctx, a, blocks, vranks, stream);
    case OP_PROD:
        return launch_staged_op<DT, OP_PROD>(ctx, a, blocks, vranks, stream);
    case OP_XOR:
        if constexpr (!Tr<DT>::is_float) {
            return launch_staged_op<DT, OP_XOR>(ctx, a, blocks, vranks, stream);
        }
        return -1;
    }
    return -1;
}
}  // namespace stdml::collective::cuda
