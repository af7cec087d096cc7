// Small all-reduce in ONE exchange: every rank stores its data straight into the peers'
// mailboxes, each 4 bytes of data beside 4 bytes of flag, and every rank polls its own
// mailbox until the flags of all sources are there.
//
// What bounds it: latency.  Pack, fence, flag, poll, fence, load is a chain of six trips to
// memory or to a peer; with the flag inside every 8-byte word the data is its own
// signal, and the chain is one store and one poll.  The price is twice the bytes, so
// this is for messages whose time is the chain (see ll_limit in algo_table.hpp).
// Three f32 elements, 8 ranks on one GPU: 6.8 us per call with a barrier, 4.1 us so;
// 16 KB in the heap, 2 ranks: 8.2 us per call in place, 4.4 us so.
//
// One vector per thread.  The flag is the block's epoch + 1, so a word from an earlier
// call never passes for this one's, and the two mailboxes of a block alternate with the
// epoch: a rank that writes into mailbox e & 1 has finished the call (or barrier) with epoch
// e - 1, in which it heard from every peer's block of this index, so each of them had left
// epoch e - 2, the last that read this mailbox.
//
// Reduction order is rank-ascending, as in the other peer-load algorithms.
// The reference's counterpart is its chunk walk (src/stdml/collective/session.cpp:49-62 there).
#include "ar_kernel.cuh"

namespace stdml::collective::cuda
{
namespace
{
// Both 8-byte halves are single accesses: data and flag of a half arrive together.
__device__ __forceinline__ void st_mail(char *p, uint32_t d0, uint32_t d1, uint32_t flag)
{
    asm volatile(
        "{\n\t"
        ".reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %3};\n\t"
        "mov.b64 b, {%2, %3};\n\t"
        "st.relaxed.sys.global.v2.b64 [%0], {a, b};\n\t"
        "}" ::"l"(p),
        "r"(d0), "r"(d1), "r"(flag)
        : "memory");
}

__device__ __forceinline__ void ld_mail(const char *p, uint32_t *d0, uint32_t *f0, uint32_t *d1,
                                        uint32_t *f1)
{
    asm volatile(
        "{\n\t"
        ".reg .b64 a, b;\n\t"
        "ld.relaxed.sys.global.v2.b64 {a, b}, [%4];\n\t"
        "mov.b64 {%0, %1}, a;\n\t"
        "mov.b64 {%2, %3}, b;\n\t"
        "}"
        : "=r"(*d0), "=r"(*f0), "=r"(*d1), "=r"(*f1)
        : "l"(p)
        : "memory");
}

template <int DT, int OP>
__global__ void __launch_bounds__(kThreads, 2)
    ll_kernel(const __grid_constant__ CommCtx ctx, const __grid_constant__ LlArgs a)
{
    const int vr = static_cast<int>(blockIdx.y);
    const int rank = ctx.rank + vr;
    const int world = ctx.world;
    SignalPad *pad = pad_of(ctx, rank);
    const unsigned int v = blockIdx.x * kThreads + threadIdx.x;
    const bool mine = v < a.nvec;
    const uint32_t epoch = ld_relaxed_sys_u32(&pad->epoch[blockIdx.x]);
    uint4 own = make_uint4(0, 0, 0, 0);
    if (mine) { own = load_user_vec<DT>(a.src[vr], false, v, a.count, ptr_aligned16(a.src[vr])); }
    const uint32_t flag = epoch + 1u;
    // mailbox [parity][source][vector], 32 bytes each
    const unsigned long long per_source = a.capacity * 32ull;
    const unsigned long long box = a.off + (epoch & 1u) * world * per_source + v * 32ull;
    bool ok = true;
    if (mine) {
        for (int i = 1; i < world; ++i) {
            const int r = rank + i < world ? rank + i : rank + i - world;
            char *to = ctx.base[r] + box + rank * per_source;
            st_mail(to, own.x, own.y, flag);
            st_mail(to + 16, own.z, own.w, flag);
        }
        Accum<DT> acc;
        for (int r0 = 0; ok && r0 < world; r0 += 4) {
            // the looks at all sources of a batch are under way together: one trip, not four
            uint4 x[4];
            unsigned int spins = 0;
            unsigned long long t0 = 0;
            for (bool all = false; !all;) {
                uint32_t f[4][4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (r0 + j < world && r0 + j != rank) {
                        const char *from = ctx.base[rank] + box + (r0 + j) * per_source;
                        ld_mail(from, &x[j].x, &f[j][0], &x[j].y, &f[j][1]);
                        ld_mail(from + 16, &x[j].z, &f[j][2], &x[j].w, &f[j][3]);
                    } else {
                        x[j] = own;
                        f[j][0] = f[j][1] = f[j][2] = f[j][3] = flag;
                    }
                }
                all = true;
                int missing = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bool here = f[j][0] == flag && f[j][1] == flag && f[j][2] == flag &&
                                      f[j][3] == flag;
                    if (!here) { missing = r0 + j; }
                    all = all && here;
                }
                if (!all && (++spins & 127u) == 0u) {
                    const unsigned long long now = global_ns();
                    if (t0 == 0) { t0 = now; }
                    if (now - t0 > ctx.timeout_ns || spins >= ctx.max_spins) {
                        report_timeout(ctx, rank, missing, flag, epoch, 0);
                        ok = false;
                        break;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (ok && r0 + j < world) {
                    if (r0 + j == 0) {
                        acc.init(x[j]);
                    } else {
                        acc.template add<OP>(x[j]);
                    }
                }
            }
        }
        if (ok) {
            store_user_vec<DT>(a.dst[vr], false, v, a.count, ptr_aligned16(a.dst[vr]),
                               acc.finish(a.scale, a.has_scale != 0));
        }
    }
    // everybody has read the epoch
    if (__syncthreads_and(ok ? 1 : 0) != 0 && threadIdx.x == 0) { pad->epoch[blockIdx.x] = flag; }
}

template <int DT>
int launch_ll_ops(const CommCtx &ctx, const LlArgs &a, int op, int vranks, cudaStream_t stream)
{
    auto go = [&](auto *kernel) {
        const dim3 grid(static_cast<unsigned int>((a.nvec + kThreads - 1) / kThreads), vranks, 1);
        if (vranks > 1) {
            void *params[2] = {const_cast<CommCtx *>(&ctx), const_cast<LlArgs *>(&a)};
            return static_cast<int>(cudaLaunchCooperativeKernel(
                reinterpret_cast<const void *>(kernel), grid, dim3(kThreads), params, 0, stream));
        }
        kernel<<<grid, kThreads, 0, stream>>>(ctx, a);
        return static_cast<int>(cudaGetLastError());
    };
    switch (op) {
    case OP_SUM:
        return go(&ll_kernel<DT, OP_SUM>);
    case OP_MIN:
        return go(&ll_kernel<DT, OP_MIN>);
    case OP_MAX:
        return go(&ll_kernel<DT, OP_MAX>);
    case OP_PROD:
        return go(&ll_kernel<DT, OP_PROD>);
    case OP_XOR:
        if constexpr (!Tr<DT>::is_float) { return go(&ll_kernel<DT, OP_XOR>); }
        return -1;
    }
    return -1;
}
}  // namespace

int launch_ll(const CommCtx &ctx, const LlArgs &a, int dt, int op, int vranks, void *stream)
{
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (dt) {
    case DT_I8:
        return launch_ll_ops<DT_I8>(ctx, a, op, vranks, s);
    case DT_I16:
        return launch_ll_ops<DT_I16>(ctx, a, op, vranks, s);
    case DT_I32:
        return launch_ll_ops<DT_I32>(ctx, a, op, vranks, s);
    case DT_I64:
        return launch_ll_ops<DT_I64>(ctx, a, op, vranks, s);
    case DT_U8:
        return launch_ll_ops<DT_U8>(ctx, a, op, vranks, s);
    case DT_U16:
        return launch_ll_ops<DT_U16>(ctx, a, op, vranks, s);
    case DT_U32:
        return launch_ll_ops<DT_U32>(ctx, a, op, vranks, s);
    case DT_U64:
        return launch_ll_ops<DT_U64>(ctx, a, op, vranks, s);
    case DT_BF16:
        return launch_ll_ops<DT_BF16>(ctx, a, op, vranks, s);
    case DT_F16:
        return launch_ll_ops<DT_F16>(ctx, a, op, vranks, s);
    case DT_F32:
        return launch_ll_ops<DT_F32>(ctx, a, op, vranks, s);
    case DT_F64:
        return launch_ll_ops<DT_F64>(ctx, a, op, vranks, s);
    }
    return -1;
}
}  // namespace stdml::collective::cuda
