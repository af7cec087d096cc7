// The waits between the warps of a block (cuda/ring_sync.cuh) on one GPU: a round that nobody
// finishes runs out, within its limit and with a status from the teller; after another warp's
// give-up nobody reports; a warp that asked for nothing drains nothing.
#include <cstdio>

#include "../cuda/ring_sync.cuh"

using namespace stdml::collective::cuda;

static int failures = 0;
#define EXPECT(c)                                                              \
    do {                                                                       \
        if (!(c)) {                                                            \
            std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c);                \
            ++failures;                                                        \
        }                                                                      \
    } while (0)

// Round 0 is over; whoever waits for round 1 gives up.  The second warp is a teller without passes.
__global__ void waits(const CommCtx ctx, int gave_up_before, int *got)
{
    __shared__ Phases<2> phases;
    __shared__ Phases<1> left;
    __shared__ int dead;
    if (threadIdx.x == 0) {
        phases.init(1u);
        left.init(1u);
        dead = gave_up_before;
        fence_async_proxy();
        mbar_arrive(phases.at(0));
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const bool first = ring_wait(ctx, dead, phases, 0), second = ring_wait(ctx, dead, phases, 1);
        if (threadIdx.x == 0) {
            got[0] = first ? 1 : 0;
            got[1] = second ? 1 : 0;
        }
        drain(ctx, phases, -1);
        drain(ctx, phases, 0);
        if (second) { warp_arrive(left.at(0)); }
    } else {
        ring_tell(ctx, dead, 0u, phases, ctx.rank, 0, left);
    }
    __syncthreads();
    if (threadIdx.x == 0) { got[2] = dead; }
}

int main()
{
    StatusBlock *status = nullptr;
    int *got = nullptr;
    if (cudaHostAlloc(&status, sizeof(*status), cudaHostAllocMapped) != cudaSuccess ||
        cudaHostAlloc(&got, 3 * sizeof(int), cudaHostAllocMapped) != cudaSuccess) {
        std::printf("no memory\n");
        return 1;
    }
    cudaEvent_t ends[2];
    for (auto &e : ends) { cudaEventCreate(&e); }
    cudaFuncAttributes loaded;  // (not within the time that is measured)
    EXPECT(cudaFuncGetAttributes(&loaded, waits) == cudaSuccess);
    for (const int gave_up_before : {0, 1}) {
        *status = StatusBlock{};
        got[0] = got[1] = got[2] = -1;
        CommCtx ctx{};
        ctx.status = status;
        ctx.timeout_ns = 20'000'000;
        ctx.max_spins = 1u << 30;
        ctx.world = 2;
        ctx.rank = 1;
        cudaEventRecord(ends[0]);
        waits<<<1, 64>>>(ctx, gave_up_before, got);
        cudaEventRecord(ends[1]);
        EXPECT(cudaDeviceSynchronize() == cudaSuccess);
        float ms = 0;
        cudaEventElapsedTime(&ms, ends[0], ends[1]);
        EXPECT(got[0] == 1 && got[1] == 0 && got[2] == (gave_up_before != 0 ? 1 : kRanOut + 1));
        if (gave_up_before != 0) {
            EXPECT(status->code == kStatusOk && ms < 20);
        } else {
            EXPECT(status->code == kStatusTimeout && status->rank == 1 && status->block == 0 && status->peer == -1 &&
                   status->phase == kPhaseRing && status->want == 1);
            EXPECT(ms >= 40 && ms < 60);
        }
    }
    std::printf("test-ring-sync: %s\n", failures == 0 ? "OK" : "FAILED");
    return failures == 0 ? 0 : 1;
}
