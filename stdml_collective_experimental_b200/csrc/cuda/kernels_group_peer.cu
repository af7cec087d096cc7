// Fused group all-reduce on registered tensors: the two-shot of ar_kernel.cuh
// walking a table of per-rank tensor pointers instead of one flat buffer.  The
// owner of a span loads every rank's piece of every tensor that intersects it
// (rank-ascending reduce in registers, scale fused) and stores the result into
// every rank's output tensor.  Nothing is packed or unpacked, so loose gradient
// tensors cost one launch and no extra HBM pass.  Two ways of loading: 16-byte
// peer loads, each vector finding its own tensor (small sets), or bulk asynchronous copies into a shared-memory
// ring whose tiles run on across tensor boundaries, so that the copy pipeline
// never drains between tensors (BULK).
//
// The reference's counterpart is its per-tensor thread pool
// (src/stdml/collective/session.cpp:83-97 there).
#include "ar_kernel.cuh"
#include "group_walk.cuh"

namespace stdml::collective::cuda
{
namespace
{
// One tile in the ring: whole vectors [v0, v0 + nv) of an entry.
struct SlotTile {
    const PeerEntry *e;  // null: the block has no more tiles
    unsigned long long v0;
    unsigned int nv;
};

// Entries whose first vectors are searched in shared memory.
constexpr int kPeerStarts = 1024;

// The owner's reduce with bulk pulls.  The flat index space is cut into chunks of
// kChunkTiles tiles, which the blocks take by ticket (the first by index; see
// draw_ticket), and a chunk is walked tile by tile, tensor after tensor.  Ring slot
// k % stages holds the k-th tile: `world` pieces of tile_vec vectors, rank-major.
// One thread of a warp of its own (the block's last) walks the table, whose dependent loads
// would hold up a warp that also reduces, issues the copies as slots become
// free and leaves each tile's place in slots[]; the other warps wait on a slot's `full`
// mbarrier, reduce, and arrive one by one on its `empty` one, so that no warp waits for the
// slowest of its tile.  Returns false after a wait that ran out.
// bf16, 199 tensors, 219 MB, 8 ranks on one GPU: 655 us with equal contiguous spans, 730
// by ticket with the walk in a warp that also reduces, 574 so (HBM floor 536).
constexpr unsigned long long kChunkTiles = 8;
constexpr int kWalkThreads = kThreads + 32;

template <int DT, int OP>
__device__ __forceinline__ bool bulk_walk(const CommCtx &ctx, const GroupPeerArgs &a, int rank,
                                          unsigned char *ring, unsigned long long *full,
                                          unsigned long long *empty, SlotTile *slots, const unsigned int *starts,
                                          bool searchable, BlockSync *sync)
{
    constexpr unsigned long long N = lanes_of<DT>();
    const int world = ctx.world;
    const int stages = a.tma_stages;
    const unsigned int tile_vec = a.tma_tile_vec;
    const unsigned int tile_bytes = tile_vec * 16u;
    const uint32_t ring_s = smem_addr(ring);
    const uint32_t full_s = smem_addr(full), empty_s = smem_addr(empty);
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full_s + 8u * s, 1u);
            mbar_init(empty_s + 8u * s, kThreads / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_proxy();
    }
    __syncthreads();

    const bool walker = threadIdx.x == kThreads;
    const unsigned int blocks = gridDim.x * (ctx.one_gpu ? gridDim.y : 1u);
    SignalPad *tickets = ticket_pad(ctx, rank);
    bool ok = true;
    int issued = 0;  // walker only
    if (walker) {
        fence_async_proxy();  // the barriers it has passed against the copies it issues
        // on one GPU every block may serve every shard
        const bool any = ctx.one_gpu != 0;
        const Span shard = any ? Span{0ull, a.nvec} : span_of(a.nvec, world, rank, 1, 0);
        const unsigned long long chunk_vec = kChunkTiles * tile_vec;
        unsigned long long chunk = any ? blockIdx.y * static_cast<unsigned long long>(gridDim.x) + blockIdx.x
                                       : blockIdx.x;
        Span sp{0, 0};
        TileCursor ahead{a.ntable, 0, 0};
        for (bool first = true; ok; ++issued) {
            const int s = issued % stages;
            if (issued >= stages &&
                !mbar_wait(ctx, empty_s + 8u * s, static_cast<uint32_t>((issued / stages - 1) & 1),
                           ctx.timeout_ns)) {
                ok = false;
                break;
            }
            Tile t;
            bool have = true;
            while (ahead.i >= a.ntable || !cursor_next<N>(a, sp, &ahead, tile_vec, &t)) {
                if (!first) { chunk = static_cast<unsigned long long>(blocks) + draw_ticket(tickets); }
                first = false;
                sp.lo = shard.lo + chunk * chunk_vec;
                have = sp.lo < shard.hi;
                if (!have) { break; }
                sp.hi = sp.lo + chunk_vec < shard.hi ? sp.lo + chunk_vec : shard.hi;
                if (searchable) {
                    int lo = 0, hi = a.ntable - 1;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (starts[mid] <= static_cast<unsigned int>(sp.lo)) {
                            lo = mid;
                        } else {
                            hi = mid - 1;
                        }
                    }
                    ahead.i = lo;
                } else {
                    ahead.i = find_peer_entry(a.table, a.ntable, sp.lo);
                }
                ahead.v = ahead.end = 0;
                // (a chunk may hold no whole vector)
                if (!cursor_enter<N>(a, sp, &ahead)) { ahead.i = a.ntable; }
            }
            const uint32_t bar = full_s + 8u * s;
            if (!have) {
                slots[s].e = nullptr;
                mbar_expect_tx(bar, 0u);
                ++issued;
                break;
            }
            slots[s] = SlotTile{t.e, t.v0, t.nv};
            const uint32_t bytes = t.nv * 16u;
            mbar_expect_tx(bar, bytes * static_cast<uint32_t>(world));
            for (int i = 0; i < world; ++i) {
                // start with the next rank, so that the owners do not all pull from
                // the same GPU at the same moment
                const int r = (rank + 1 + i) % world;
                bulk_load(ring_s + (static_cast<uint32_t>(s) * world + r) * tile_bytes,
                          t.e->in[r] + t.v0 * 16ull, bytes, bar);
            }
        }
    } else if (threadIdx.x < kThreads) {
        const bool has_scale = a.has_scale != 0;
        for (int done = 0;; ++done) {
            const int s = done % stages;
            if (!mbar_wait(ctx, full_s + 8u * s, static_cast<uint32_t>((done / stages) & 1),
                           ctx.timeout_ns)) {
                ok = false;
                break;
            }
            const SlotTile t = slots[s];
            if (t.e == nullptr) { break; }
            const uint4 *slot =
                reinterpret_cast<const uint4 *>(ring + static_cast<size_t>(s) * world * tile_bytes);
            char *outs[kMaxRanks];
#pragma unroll
            for (int r = 0; r < kMaxRanks; ++r) {
                outs[r] = r < world ? t.e->out[r] + t.v0 * 16ull : nullptr;
            }
            for (unsigned int i = threadIdx.x; i < t.nv; i += kThreads) {
                Accum<DT> acc;
                for (int r0 = 0; r0 < world; r0 += 4) {
                    uint4 x[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (r0 + j < world) { x[j] = slot[static_cast<size_t>(r0 + j) * tile_vec + i]; }
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
                const uint4 res = acc.finish(a.scale, has_scale);
#pragma unroll
                for (int r = 0; r < kMaxRanks; ++r) {
                    if (r < world) { st_arena_v4(outs[r] + i * 16ull, res); }
                }
            }
            __syncwarp();
            if ((threadIdx.x & 31u) == 0u) { mbar_arrive(empty_s + 8u * s); }
        }
    }
    if (__syncthreads_and(ok ? 1 : 0) == 0) {
        if (walker) {
            report_timeout(ctx, rank, -1, 0u, 0u, 64 + sync->phase);
            // copies already issued still write into this CTA's shared memory: give
            // them one more (bounded) chance to land before the CTA goes away
            for (int k = issued > stages ? issued - stages : 0; k < issued; ++k) {
                (void)mbar_wait(ctx, full_s + 8u * (k % stages),
                                static_cast<uint32_t>((k / stages) & 1), ctx.timeout_ns / 4);
            }
        }
        __syncthreads();
        return false;
    }
    if (walker) { leave_tickets(tickets, blocks); }
    return true;
}

// Elements [e0, count) of an entry, one by one: the ragged last vector of a tensor.
template <int DT, int OP>
static __device__ __noinline__ void reduce_tail(const PeerEntry *e, unsigned long long e0, int world,
                                                double scale, bool has_scale)
{
    using S = typename Tr<DT>::storage;
    for (unsigned long long j = e0; j < e->count; ++j) {
        typename Tr<DT>::acc acc =
            Tr<DT>::widen(*reinterpret_cast<const volatile S *>(e->in[0] + j * sizeof(S)));
        for (int r = 1; r < world; ++r) {
            acc = combine<OP>(acc, Tr<DT>::widen(*reinterpret_cast<const volatile S *>(
                                       e->in[r] + j * sizeof(S))));
        }
        if constexpr (Tr<DT>::is_float) {
            if (has_scale) { acc = acc * static_cast<typename Tr<DT>::acc>(scale); }
        }
        const S res = Tr<DT>::narrow(acc);
        for (int r = 0; r < world; ++r) {
            *reinterpret_cast<volatile S *>(e->out[r] + j * sizeof(S)) = res;
        }
    }
}

template <int DT, int OP, bool BULK>
__global__ void __launch_bounds__(BULK ? kWalkThreads : kThreads)
    group_peer_kernel(const __grid_constant__ CommCtx ctx, const __grid_constant__ GroupPeerArgs a)
{
    constexpr unsigned long long N = lanes_of<DT>();
    extern __shared__ __align__(128) unsigned char ring[];
    __shared__ BlockSync sync;
    __shared__ __align__(8) unsigned long long full[BULK ? kTmaMaxStages : 1];
    __shared__ __align__(8) unsigned long long empty[BULK ? kTmaMaxStages : 1];
    __shared__ SlotTile slots[BULK ? kTmaMaxStages : 1];
    __shared__ unsigned int starts[kPeerStarts];
    const int rank = ctx.rank + static_cast<int>(blockIdx.y);
    const int world = ctx.world;
    const int nb = static_cast<int>(gridDim.x);
    const int b = static_cast<int>(blockIdx.x);
    sync_begin(ctx, rank, &sync);
    const bool searchable = a.ntable <= kPeerStarts && a.nvec >> 32 == 0;
    if (searchable) {
        for (int i = static_cast<int>(threadIdx.x); i < a.ntable; i += static_cast<int>(blockDim.x)) {
            starts[i] = static_cast<unsigned int>(a.table[i].voff);
        }
    }
    // every rank is here: its inputs are final, its outputs may be written
    if (!peer_barrier(ctx, rank, &sync)) { return; }

    const Span sp = span_of(a.nvec, world, rank, nb, b);
    if constexpr (BULK) {
        if (!bulk_walk<DT, OP>(ctx, a, rank, ring, full, empty, slots, starts, searchable, &sync)) {
            return;
        }
        // the ragged last vectors in this block's span, a tensor per thread
        if (sp.lo < sp.hi) {
            for (int i = find_peer_entry(a.table, a.ntable, sp.lo) + static_cast<int>(threadIdx.x);
                 i < a.ntable; i += kWalkThreads) {
                const PeerEntry *e = &a.table[i];
                const unsigned long long voff = e->voff;
                if (voff >= sp.hi) { break; }
                const unsigned long long whole = e->count / N;
                const unsigned long long tail = voff + whole;
                if (whole * N < e->count && tail >= sp.lo && tail < sp.hi) {
                    reduce_tail<DT, OP>(e, whole * N, world, a.scale, a.has_scale != 0);
                }
            }
        }
    } else {
        // Small sets: a vector per thread, which looks for its own tensor.  (Walking the
        // tensors of the span one after the other costs their latency each: 158 tensors,
        // 0.55 MB, 8 ranks on one GPU: 103 us, so 17 us.)
        for (unsigned long long v = sp.lo + threadIdx.x; v < sp.hi; v += kThreads) {
            int i;
            if (searchable) {
                int lo = 0, hi = a.ntable - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (starts[mid] <= static_cast<unsigned int>(v)) {
                        lo = mid;
                    } else {
                        hi = mid - 1;
                    }
                }
                i = lo;
            } else {
                i = find_peer_entry(a.table, a.ntable, v);
            }
            const PeerEntry *e = &a.table[i];
            const unsigned long long lv = v - e->voff;
            if ((lv + 1) * N > e->count) {
                reduce_tail<DT, OP>(e, lv * N, world, a.scale, a.has_scale != 0);
                continue;
            }
            Accum<DT> acc;
            for (int r0 = 0; r0 < world; r0 += 4) {
                uint4 x[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (r0 + j < world) { x[j] = ld_arena_v4(e->in[r0 + j] + lv * 16ull); }
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
            for (int k = 0; k < world; ++k) {
                const int r = rank + k < world ? rank + k : rank + k - world;
                st_arena_v4(e->out[r] + lv * 16ull, res);
            }
        }
    }
    if (!peer_barrier(ctx, rank, &sync)) { return; }
    sync_end(ctx, rank, &sync);
}

template <int DT, int OP, bool BULK>
int launch_gp_mode(const CommCtx &ctx, const GroupPeerArgs &a, dim3 grid, int vranks,
                   unsigned int smem, cudaStream_t s)
{
    if (smem > (48u << 10)) {
        // the opt-in to more than 48 KB is per function and per device
        static bool opted_in[64] = {};
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { dev = 0; }
        if (!opted_in[dev]) {
            const cudaError_t e = cudaFuncSetAttribute(
                reinterpret_cast<const void *>(&group_peer_kernel<DT, OP, BULK>),
                cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTmaSmemBudget));
            if (e != cudaSuccess) { return static_cast<int>(e); }
            opted_in[dev] = true;
        }
    }
    if (vranks > 1) {
        void *params[2] = {const_cast<CommCtx *>(&ctx), const_cast<GroupPeerArgs *>(&a)};
        return static_cast<int>(cudaLaunchCooperativeKernel(
            reinterpret_cast<const void *>(&group_peer_kernel<DT, OP, BULK>), grid,
            dim3(BULK ? kWalkThreads : kThreads), params, smem, s));
    }
    group_peer_kernel<DT, OP, BULK><<<grid, BULK ? kWalkThreads : kThreads, smem, s>>>(ctx, a);
    return static_cast<int>(cudaGetLastError());
}

template <int DT, int OP>
int launch_gp(const CommCtx &ctx, const GroupPeerArgs &a, int blocks, int vranks, cudaStream_t s)
{
    dim3 grid(blocks, vranks, 1);
    if (a.tma_stages > 0) {
        const unsigned int smem = static_cast<unsigned int>(a.tma_stages) *
                                  static_cast<unsigned int>(ctx.world) * a.tma_tile_vec * 16u;
        return launch_gp_mode<DT, OP, true>(ctx, a, grid, vranks, smem, s);
    }
    return launch_gp_mode<DT, OP, false>(ctx, a, grid, vranks, 0u, s);
}

template <int DT>
int launch_gp_ops(const CommCtx &ctx, const GroupPeerArgs &a, int op, int blocks, int vranks,
                  cudaStream_t s)
{
    switch (op) {
    case OP_SUM:
        return launch_gp<DT, OP_SUM>(ctx, a, blocks, vranks, s);
    case OP_MIN:
        return launch_gp<DT, OP_MIN>(ctx, a, blocks, vranks, s);
    case OP_MAX:
        return launch_gp<DT, OP_MAX>(ctx, a, blocks, vranks, s);
    case OP_PROD:
        return launch_gp<DT, OP_PROD>(ctx, a, blocks, vranks, s);
    case OP_XOR:
        if constexpr (!Tr<DT>::is_float) { return launch_gp<DT, OP_XOR>(ctx, a, blocks, vranks, s); }
        return -1;
    }
    return -1;
}
}  // namespace

int launch_group_peer(const CommCtx &ctx, const GroupPeerArgs &a, int dt, int op, int blocks,
                      int vranks, void *stream)
{
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (dt) {
    case DT_I8:
        return launch_gp_ops<DT_I8>(ctx, a, op, blocks, vranks, s);
    case DT_I16:
        return launch_gp_ops<DT_I16>(ctx, a, op, blocks, vranks, s);
    case DT_I32:
        return launch_gp_ops<DT_I32>(ctx, a, op, blocks, vranks, s);
    case DT_I64:
        return launch_gp_ops<DT_I64>(ctx, a, op, blocks, vranks, s);
    case DT_U8:
        return launch_gp_ops<DT_U8>(ctx, a, op, blocks, vranks, s);
    case DT_U16:
        return launch_gp_ops<DT_U16>(ctx, a, op, blocks, vranks, s);
    case DT_U32:
        return launch_gp_ops<DT_U32>(ctx, a, op, blocks, vranks, s);
    case DT_U64:
        return launch_gp_ops<DT_U64>(ctx, a, op, blocks, vranks, s);
    case DT_BF16:
        return launch_gp_ops<DT_BF16>(ctx, a, op, blocks, vranks, s);
    case DT_F16:
        return launch_gp_ops<DT_F16>(ctx, a, op, blocks, vranks, s);
    case DT_F32:
        return launch_gp_ops<DT_F32>(ctx, a, op, blocks, vranks, s);
    case DT_F64:
        return launch_gp_ops<DT_F64>(ctx, a, op, blocks, vranks, s);
    }
    return -1;
}
}  // namespace stdml::collective::cuda
