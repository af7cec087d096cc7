// How the warps of a block work together where some of them look after flags and loads and the
// others (the workers) move bytes in rounds: staged_kernel.cuh, kernels_pull.cu.
#pragma once
#include "ar_kernel.cuh"
#include "copy.cuh"

namespace stdml::collective::cuda
{
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t at)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(at)
                 : "memory");
    return v;
}

// One phase per round of something, on N barriers in turn: who waits for round k finds it although
// up to N - 1 later ones are over too.
template <int N>
struct Phases {
    unsigned long long bar[N];

    __device__ __forceinline__ void init(unsigned int count)
    {
        for (int i = 0; i < N; ++i) { mbar_init(smem_addr(&bar[i]), count); }
    }
    __device__ __forceinline__ uint32_t at(int k) const { return smem_addr(&bar[k % N]); }
    // (may sleep a while on a round that is not over)
    __device__ __forceinline__ bool try_wait(int k) const
    {
        return mbar_try_wait(at(k), static_cast<uint32_t>(k / N & 1));
    }
    __device__ __forceinline__ bool over(int k) const
    {
        uint32_t done;
        asm volatile("{\n\t"
                     ".reg .pred p;\n\t"
                     "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t"
                     "}"
                     : "=r"(done)
                     : "r"(at(k)), "r"(static_cast<uint32_t>(k / N & 1))
                     : "memory");
        return done != 0;
    }
};

// Waits for round k of something.  False: the block gives up.  `dead`, in shared memory, says why: 1, a peer's
// flag did not come, which the poll has reported; kRanOut + k, this wait ran out (the teller reports it).
constexpr int kRanOut = 2;

template <int N>
__device__ __forceinline__ bool ring_wait(const CommCtx &ctx, int &dead, const Phases<N> &phases, int k)
{
    unsigned long long t0 = 0;
    for (unsigned int spins = 0; !phases.try_wait(k); ++spins) {
        if (*static_cast<volatile int *>(&dead) != 0) { return false; }
        if ((spins & 63u) != 63u) { continue; }
        const unsigned long long now = global_ns();
        if (t0 == 0) { t0 = now; }
        // (twice the limit of a wait for a peer's flag, of whose end `dead` tells)
        if (now - t0 > 2 * ctx.timeout_ns || spins >= ctx.max_spins) {
            *static_cast<volatile int *>(&dead) = kRanOut + k;
            return false;
        }
    }
    return true;
}

// A warp that gives up with another's wait or its own poll, which has reported.
__device__ __forceinline__ void ring_give_up(int &dead)
{
    if (*static_cast<volatile int *>(&dead) == 0) { *static_cast<volatile int *>(&dead) = 1; }
}

// A warp that gives up: its copies in flight end before the block does.  `last`: the last round that it has
// asked for (-1: none), which up to N - 1 before it may still be under way with.
template <int N>
__device__ __forceinline__ void drain(const CommCtx &ctx, const Phases<N> &phases, int last)
{
    for (int k = last; k >= 0 && k > last - N; --k) {
        (void)mbar_wait(ctx, phases.at(k), static_cast<uint32_t>(k / N & 1), ctx.timeout_ns / 4);
    }
}

// What each lane has acquired (a peer's flag, a phase) is then seen by all of them: a vote orders nothing between lanes.
__device__ __forceinline__ bool warp_agrees(bool ok)
{
    const bool all = __all_sync(0xffffffffu, ok ? 1 : 0) != 0;
    __syncwarp();
    return all;
}

// One lane of a worker warp for all of it.
__device__ __forceinline__ void warp_arrive(uint32_t bar)
{
    __syncwarp();
    if ((threadIdx.x & 31u) == 0u) { mbar_arrive(bar); }
}

// Asks for the first `bytes` bytes at src, of tensor memory, past the L2 as far as it can; every lane
// of a barrier of 32 calls it.
__device__ __forceinline__ void ask_stream(uint32_t bar, uint32_t dst, const void *src,
                                           unsigned int bytes, unsigned long long policy)
{
    if (bytes == 0u) {
        mbar_arrive(bar);
        return;
    }
    mbar_expect_tx(bar, bytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
                 "[%0], [%1], %2, [%3], %4;" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar), "l"(policy)
                 : "memory");
}

// The teller: lets the peers know what the passes have stored.  A warp of its own: its fences wait for
// all of the block's stores.  Over links and within a GPU alike they and the flags' way take
// longer than a pass, hence the lag.
// `done`: a phase per pass.  `left`: over when all warps that wait for something later than these have come
// through.  The teller stays until then, to report a wait of the block that ran out.  (Calls in the workers' code, at
// the waits or at its end, cost the bf16 wire 5 to 7 %.)
template <int N>
__device__ __forceinline__ void ring_tell(const CommCtx &ctx, int &dead, uint32_t epoch, const Phases<N> &done,
                                          int rank, int passes, const Phases<1> &left)
{
    const int p = static_cast<int>(threadIdx.x & 31u);
    for (int k = 0; k < passes; ++k) {
        if (!warp_agrees(ring_wait(ctx, dead, done, k))) { break; }
        // (one fence for all that are over by now)
        while (k + 1 < passes && warp_agrees(done.over(k + 1))) { ++k; }
        // The peers read the ring by bulk copies, which proxy fences order behind the generic stores: this one, before the
        // release, so that it is part of what the flag publishes, and the fetchers' between the flag's acquire and their loads.
        fence_async_proxy_global();
        fence_ranks(ctx);
        if (p < ctx.world) {
            st_relaxed_sys_u32(&pad_of(ctx, p)->flag[blockIdx.x][rank], epoch + static_cast<uint32_t>(k) + 1u);
        }
    }
    if (p != 0) { return; }
    // (in slices of a 64th of the limit, between which it looks at `dead`; the waits of the others end before it)
    int why = 0;
    for (int i = 0; i < 2048 && !mbar_wait(ctx, left.at(0), 0u, ctx.timeout_ns / 64); ++i) {
        why = *static_cast<volatile int *>(&dead);
        if (why != 0) { break; }
    }
    if (why >= kRanOut) { report_timeout(ctx, rank, -1, static_cast<uint32_t>(why - kRanOut), 0u, kPhaseRing); }
}

}  // namespace stdml::collective::cuda
