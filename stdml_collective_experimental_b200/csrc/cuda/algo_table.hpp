// Which algorithm and how many CTAs a collective gets: pure functions of the
// message and of the world, so that every rank reaches the same answer and the
// table can be checked without a GPU.  Thresholds come from device-timed sweeps
// on 2, 4 and 8 B200s (f32 sum, 4 KB ... 1 GiB, all four algorithms against each
// other and against NCCL).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>

#include "comm.cuh"

namespace stdml::collective::cuda
{
struct AlgoTuning {
    int world = 1;
    int vranks = 1;       // > 1: ranks emulated as grid rows of one launch
    int num_sms = 148;
    int max_blocks = 128;
    size_t oneshot_max = 0;       // 0: measured default
    size_t nvls_oneshot_max = 0;  // 0: measured default
    bool has_nvls = false;
    // two-shot calls of at least this many bytes pull with bulk async copies
    // (kAlgoTwoShotTma); SIZE_MAX: never
    size_t tma_min = 64u << 20;  // measured at 2 GPUs: ahead of the register path from 64 MB
    // NVLS worlds: owner calls of at least this many bytes prefer the bulk-copy
    // two-shot over the in-switch reduction (fewer bytes per link direction:
    // (n-1)/n x S instead of (n+1)/n x S); SIZE_MAX: never
    size_t tma_over_nvls_min = SIZE_MAX;
    int nvls_blocks = 0;  // > 0: grid of large NVLS calls
    int tma_blocks = 0;   // > 0: grid of bulk-copy two-shot calls
};

inline size_t oneshot_limit(const AlgoTuning &t)
{
    if (t.oneshot_max != 0) { return t.oneshot_max; }
    const size_t w = static_cast<size_t>(t.world);
    return w <= 2 ? (8u << 20) : (16u << 20) / (w * w);
}

// The same for one message of ordinary tensors among ranks of one GPU: against the staged kernel, whose rounds of
// flags a short message does not repay.  us per call (one-shot / staged kernel), f32:
//   3 ranks: 2.3 MB 10.4 / 14.4, 8.9 MB 24.7 / 26.5; 4: 1.3 MB 10.3 / 12.9, 5 MB 18.6 / 21.7, 7.8 MB 29.3 / 28.8;
//   5: 2.6 MB 16.5 / 18.4, 4 MB 22.6 / 23.4, 5 MB 28.8 / 26.7; 6: 2.8 MB 20.6 / 22.7; 7: 2.6 MB 21.4 / 23.2;
//   8: 1 MB 14.4 / 16.6, 2 MB 20.6 / 22.0, 3 MB 28.8 / 27.5; 12: 1.1 MB 20.6 / 22.8; 16: 0.6 MB 20.6 / 22.4.
// Of two bytes, where every rank widens every element, bf16: 3: 5.7 MB 18.5 / 21.9; 4: 4 MB 18.5 / 20.5; 5: 2 MB 16.5 / 17.7,
//   3.2 MB 22.6 / 20.6; 8: 1 MB 16.4 / 16.9, 1.6 MB 20.6 / 18.8; 16: 0.4 MB 18.5 / 18.4.
// Of one byte (4: 1 MB 16.5 / 12.4) and groups keep the limit above: a one-shot walks the tensors of a block one after
// the other (8 ranks, 30 tensors of 0.57 MB in all: 18.6 / 16.6).
inline size_t staged_oneshot_limit(const AlgoTuning &t, size_t elem_size)
{
    if (t.oneshot_max != 0 || t.vranks <= 1 || t.world <= 2 || elem_size == 1) { return oneshot_limit(t); }
    const double mb = (elem_size >= 4 ? 44 : 26) << 20, w = t.world;
    return std::max(oneshot_limit(t), static_cast<size_t>(mb / (w * std::sqrt(w))));
}

inline size_t nvls_oneshot_limit(const AlgoTuning &t)
{
    if (t.nvls_oneshot_max != 0) { return t.nvls_oneshot_max; }
    // only staged / out-of-place calls can take it; it beats a staged owner
    // algorithm up to a few MB
    return 2u << 20;
}

// Vectors of one mailbox, the most that a message may have (kernels_ll.cu).  Between ranks
// of one GPU: one vector per thread, two blocks of 512 per SM, 512 KB at most.  Over links
// 64 KB; that is an estimate, no measurement (the exchange sends the bytes twice, 64 KB more
// to each of up to 7 peers, 0.6 us at 770 GB/s, and spares a fence, a flag and the round
// trip of the peer loads, 2 us between ranks of one GPU and no less over links).  The knob
// ll_max_bytes moves it, 0 gives the kernels with barriers back.
inline size_t ll_capacity(int world, int vranks, int num_sms)
{
    if (world < 2) { return 0; }
    if (vranks <= 1) { return (64u << 10) / 16; }
    return std::min<size_t>((512u << 10) / 16,
                            static_cast<size_t>(std::max(1, 2 * num_sms / vranks)) * kThreads);
}

// Vectors of the largest message that goes through the mailboxes.  Between ranks of one GPU,
// f32, us per call (barriers / mailboxes; a call's time moves in steps of 2 us).
// In place in the heap, against a two-shot and its two barriers:
//   2 ranks: 16 KB 8.2 / 4.4, 512 KB 10.0 / 6.2; 4: 16 KB 8.2 / 6.2, 400 KB 10.3 / 9.5, 512 KB 10.3 both;
//   6: 16 KB 8.4 / 8.2, 147 KB 11.6 / 8.3; 7: 147 KB 11.1 / 10.3;
//   8: 4 KB 8.2 / 6.3, 6 KB 8.2 both, 24 KB 8.5 / 10.1, 115 KB 10.3 both;
//   10: 4 KB 9.4 / 8.2, 6 KB 8.7 / 10.3; 16: 3 KB 10.3 / 8.2, 6 KB 10.3 / 12.3.
// Out of place, against a one-shot and its one barrier:
//   2 ranks: 512 KB 7.2 / 6.2; 3: 400 KB 8.2 / 6.9; 4: 262 KB 8.2 / 6.9, 307 KB 8.2 both, 400 KB 8.2 / 9.5;
//   5: 8 KB 8.2 / 7.1, 147 KB 8.2 both; 6: 6 KB 6.6 / 6.5, 8 KB and 115 KB 8.2 both;
//   7: 4 KB 7.6 / 6.2, 6 KB 7.2 / 8.2; 8: 12 B 6.8 / 4.1, 4 KB 6.2-7.6 / 6.3, 6 KB 7.3 / 8.2;
//   12: 2 KB 8.2 / 6.5, 6 KB 8.2 / 10.3; 16: 1.5 KB 8.2 / 6.2, 4 KB 8.2 / 10.3.
inline size_t ll_limit(int world, int vranks, size_t capacity, bool in_place_symmetric)
{
    if (vranks <= 1 || world <= 2) { return capacity; }
    const auto over_all_ranks = [&](size_t kb) {
        return std::min(capacity, (kb << 10) / 16 / static_cast<size_t>(world));
    };
    if (in_place_symmetric) {
        return world <= 4 ? capacity : over_all_ranks(world < 8 ? 1024 : 48);
    }
    if (world <= 6) { return std::min(capacity, size_t{world <= 4 ? 256u << 10 : 8u << 10} / 16); }
    return over_all_ranks(32);
}

// need_owner: the result must stay in the symmetric buffer (in place), which
// only the owner algorithms (two-shot, NVLS) can do.
inline int select_algo(const AlgoTuning &t, size_t bytes, bool nvls_defined_for_op,
                       bool need_owner)
{
    if (t.world == 1) { return need_owner ? kAlgoTwoShot : kAlgoOneShot; }
    // with two GPUs the switch has nothing to add: peer loads are faster
    const bool nvls = t.has_nvls && nvls_defined_for_op && t.world > 2;
    if (nvls) {
        if (!need_owner && bytes <= nvls_oneshot_limit(t)) { return kAlgoNvlsOneShot; }
        if (bytes >= t.tma_over_nvls_min) { return kAlgoTwoShotTma; }
        return kAlgoNvls;
    }
    if (!need_owner && bytes <= oneshot_limit(t)) { return kAlgoOneShot; }
    // Two ranks on one GPU: the register path has enough loads in flight for local
    // memory and no block sync per tile (256 MB in place: 191 us against 220-246).
    if (t.vranks == 2) { return kAlgoTwoShot; }
    return bytes >= t.tma_min ? kAlgoTwoShotTma : kAlgoTwoShot;
}

inline int select_blocks(const AlgoTuning &t, size_t nvec, int algo)
{
    const bool owner = is_owner_algo(algo);
    const size_t work = owner ? (nvec + t.world - 1) / t.world : nvec;
    // Vectors of a block where the message is small.  Over links four per thread: every
    // block costs a flag per peer.  Between ranks of one GPU flags are cheap and a
    // thread's vectors follow one another: one-shots take one each, as far as the grid goes
    // (8 ranks, 80-240 KB: 10.3 us with four, 8.3 so).  Two-shots, which have world times
    // fewer each and two barriers, gain nothing.
    const size_t per_block = static_cast<size_t>(kThreads) * (t.vranks > 1 && !owner ? 1 : 4);
    size_t b = (work + per_block - 1) / per_block;
    size_t cap = static_cast<size_t>(t.max_blocks);
    if (algo == kAlgoNvls || algo == kAlgoNvlsOneShot) {
        // the switch saturates with few CTAs; more only add contention (measured at
        // 8 GPUs, 64 MB - 1 GiB: 16 and 24 CTAs lead, 32 within 1 %, 64 and up behind)
        cap = std::min<size_t>(cap, nvec * 16 >= (16u << 20) ? 24 : 64);
        if (t.nvls_blocks > 0 && nvec * 16 >= (16u << 20)) { cap = static_cast<size_t>(t.nvls_blocks); }
    }
    if (algo == kAlgoTwoShotTma) {
        // one CTA per SM at most (the ring takes the SM's shared memory)
        cap = static_cast<size_t>(t.tma_blocks > 0 ? t.tma_blocks : t.num_sms);
        cap = std::min<size_t>(cap, static_cast<size_t>(t.num_sms));
    }
    // alone on the GPU the kernel is an HBM copy: one resident CTA per SM
    if (t.world == 1) { cap = static_cast<size_t>(t.num_sms); }
    if (t.vranks > 1) { cap = std::min<size_t>(cap, std::max(1, t.num_sms / t.vranks)); }
    b = std::max<size_t>(1, std::min(b, std::min<size_t>(cap, kMaxBlocks)));
    return static_cast<int>(b);
}
}  // namespace stdml::collective::cuda
