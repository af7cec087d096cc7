// Index arithmetic of the kernels, checked on the CPU (the functions are
// __host__ __device__): for many (vectors, shards, blocks) the block spans tile
// the buffer exactly once, and the descriptor-table search lands on the tensor
// that holds a vector.  compute-sanitizer is not available for the device
// code, so the arithmetic that decides every address is exercised here.
#include <bit>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "../cuda/ar_kernel.cuh"
#include "../cuda/group_walk.cuh"
#include "../cuda/device_session.hpp"
#include "../cuda/algo_table.hpp"
#include "../cuda/arena_layout.hpp"
#include "../cuda/offset_heap.hpp"
#include "../cuda/pull_walk.hpp"
#include "../cuda/staged_walk.hpp"

using namespace stdml::collective::cuda;

static int failures = 0;
#define EXPECT(c)                                                              \
    do {                                                                       \
        if (!(c)) {                                                            \
            std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c);                \
            ++failures;                                                        \
        }                                                                      \
    } while (0)

int main()
{
    std::mt19937_64 rng(7);
    // spans: contiguous, ordered, exact cover, every boundary but the buffer's end on a
    // 512-byte granule, balanced within one granule
    for (int trial = 0; trial < 20000; ++trial) {
        const unsigned long long nvec = rng() % (trial % 3 == 0 ? 50 : 5000000) ;
        const int shards = 1 + static_cast<int>(rng() % 16);
        const int nb = 1 + static_cast<int>(rng() % 200);
        unsigned long long expect = 0;
        for (int s = 0; s < shards; ++s) {
            unsigned long long lo_min = ~0ull, len_min = ~0ull, len_max = 0;
            for (int b = 0; b < nb; ++b) {
                const Span sp = span_of(nvec, shards, s, nb, b);
                EXPECT(sp.lo == expect && sp.hi >= sp.lo && sp.hi <= nvec);
                EXPECT(sp.lo % kSpanGranule == 0 || sp.lo == nvec);
                EXPECT(sp.hi % kSpanGranule == 0 || sp.hi == nvec);
                expect = sp.hi;
                lo_min = sp.lo < lo_min ? sp.lo : lo_min;
                const unsigned long long len = sp.hi - sp.lo;
                len_min = len < len_min ? len : len_min;
                len_max = len > len_max ? len : len_max;
            }
            EXPECT(len_max - len_min <= 2 * kSpanGranule);
        }
        EXPECT(expect == nvec);
    }
    // staged all-reduce: over shards, blocks and rounds the tiles cover the buffer exactly
    // once; the ring pieces of all blocks are disjoint and stay inside the slot
    for (int trial = 0; trial < 3000; ++trial) {
        const unsigned long long nvec = 1 + rng() % (trial % 3 == 0 ? 70 : 3000000);
        const int world = 2 + static_cast<int>(rng() % 15);
        const size_t slot = (size_t{4096} << (rng() % 15)) + 4096;
        const bool user_f32 = trial % 2 == 0;
        const int sms = 1 + static_cast<int>(rng() % 148), rows = trial % 5 < 3 ? world : 1;
        const int want = trial % 7 == 0 ? 1 + static_cast<int>(rng() % 300) : 0;
        const StagedGeometry g = staged_geometry(world, nvec, slot, sms, rows, want, user_f32);
        const int per_sm = staged_per_sm(world, g.tile_shift, user_f32);
        EXPECT(per_sm >= 1 && (staged_smem(world, g.tile_shift, user_f32) + kStagedOtherSmem) * per_sm <= kSmSmem);
        EXPECT((g.blocks - 1) * rows < per_sm * sms && (want == 0 || g.blocks <= want) && g.tile_shift >= kStagedMinShift);
        const unsigned long long ring =
            ((static_cast<unsigned long long>(kStagedRing) * world) << g.tile_shift) * 16;
        EXPECT(staged_smem(world, g.tile_shift, user_f32) <= kStagedSmem);
        if (g.blocks == 0) {
            EXPECT(slot < ring);
            continue;
        }
        EXPECT(ring * g.blocks <= slot);
        std::vector<unsigned long long> bound(world + 1);
        for (int s = 0; s <= world; ++s) { bound[s] = StagedWalk::shard_begin(nvec, world, s); }
        EXPECT(bound[0] == 0 && bound[world] == nvec);
        // larger tiles leave three SMs of four a block, if the smallest ones do
        unsigned long long longest = 0;
        for (int s = 0; s < world; ++s) { longest = std::max(longest, bound[s + 1] - bound[s]); }
        const int all = want > 0 ? std::min(want, per_sm * sms / rows) : per_sm * sms / rows;
        const unsigned long long some = std::max(1, std::min({all, kMaxBlocks, (g.tile_shift < 8 || world > 3 ? 1 : 2) * sms * 3 / 4 / rows}));
        const unsigned long long ring32 = (static_cast<unsigned long long>(kStagedRing) * world << kStagedMinShift) * 16;
        const unsigned long long tiles = (longest + (1ull << g.tile_shift) - 1) >> g.tile_shift;
        if (g.full) { EXPECT(static_cast<unsigned long long>(g.blocks) >= std::min(tiles, some)); }
        if (g.tile_shift < 8) { EXPECT(g.full == (ring32 * some <= slot && slot >= 2u << 20) || tiles < some); }
        for (int s = 0; s < world; ++s) {
            unsigned long long expect = bound[s];
            for (int k = 0; k < g.rounds; ++k) {
                for (int b = 0; b < g.blocks; ++b) {
                    const StagedWalk w{bound.data(), world, g.blocks, b, g.tile_shift};
                    const StagedTile t = w.tile_of(s, k);
                    EXPECT(t.lo == expect && t.hi >= t.lo && t.hi <= bound[s + 1]);
                    expect = t.hi;
                    const unsigned long long piece = (1ull << g.tile_shift) * 16;
                    EXPECT(w.piece(k, s) == ring * b + (k % kStagedRing * world + s) * piece);
                }
            }
            EXPECT(expect == bound[s + 1]);
        }
    }
    // 102 MB go round in slots far smaller than that in one launch, with a block on most SMs; in 64 MB in all that are resident
    for (const int world : {2, 3, 4, 8}) {
        for (const size_t mb : {2, 4, 8, 16, 32, 64}) {
            const StagedGeometry g = staged_geometry(world, 102'000'000 / 16, mb << 20, 148, world, 0, false);
            EXPECT(g.full && g.blocks * world >= 144 && g.tile_shift >= 7);
            if (mb == 64) { EXPECT(g.blocks == kStagedMinPerSm * 148 / world); }
        }
    }
    // pull: over blocks and rounds the tiles cover the vectors of every rank's block exactly
    // once, whatever its shift; ring pieces are disjoint and stay inside the slot
    for (int trial = 0; trial < 2000; ++trial) {
        const size_t bytes = 1 + rng() % (trial % 3 == 0 ? 100 : 40000000);
        const size_t stride = bytes + rng() % 40;
        const int world = 2 + static_cast<int>(rng() % 15);
        const size_t slot = (size_t{4096} << (rng() % 15)) + 4096;
        const int sms = 1 + static_cast<int>(rng() % 148), rows = trial % 5 < 3 ? world : 1;
        const int want = trial % 7 == 0 ? 1 + static_cast<int>(rng() % 300) : 0;
        const int sources = pull_sources(world, trial % 2 == 0 ? 0 : -1);
        const PullGeometry g = pull_geometry(sources, bytes, slot, sms, rows, want);
        EXPECT((g.blocks - 1) * rows < (g.lng ? kPullLongPerSm : kPullPerSm) * sms && (want == 0 || g.blocks <= want));
        EXPECT(g.tile % 32 == 0 && g.tile > 0);
        if (g.blocks == 0) {
            EXPECT(slot < (static_cast<size_t>(kPullRing) << kPullStepShift) * 16);
            continue;
        }
        if (g.lng) {
            EXPECT(g.ring == kPullLongRing && pull_long_smem(sources, g.tile) <= kPullLongSmem);
        } else {
            EXPECT(g.ring == kPullRing && (g.tile & (g.tile - 1)) == 0 && g.tile >= 1u << kPullStepShift);
        }
        // a smaller slot gives the long kernel smaller tiles, before it takes it away
        const size_t resident = std::max(1, std::min(want > 0 ? want : kMaxBlocks, kPullLongPerSm * sms / rows));
        if (pull_geometry(sources, bytes, size_t{1} << 40, sms, rows, want).lng) {
            EXPECT(g.lng == (slot >= resident * kPullLongRing * kPullLongMinTile * 16) ||
                   ((bytes + 30) / 16 < 2 * kPullLongMin * resident && slot < resident * kPullLongRing * 512 * 16));
        }
        const unsigned long long piece = g.tile * 16ull, ring = piece * g.ring;
        EXPECT(ring * g.blocks == g.ring_bytes() && g.ring_bytes() <= slot);
        unsigned long long expect = 0;
        for (int k = 0; k < g.rounds; ++k) {
            for (int b = 0; b < g.blocks; ++b) {
                const PullWalk w{{bytes, stride}, g.blocks, b, std::bit_width(g.tile) - 1};
                const PullLongWalk l{{bytes, stride}, g.blocks, b, g.tile};
                EXPECT((g.lng ? l.first_vector(k) : w.first_vector(k)) == expect);
                expect += g.tile;
                EXPECT((g.lng ? l.piece(k) : w.piece(k)) == ring * b + (k % g.ring) * piece);
            }
        }
        for (int p = 0; p < world; ++p) {
            const PullLayout w{bytes, stride};
            EXPECT(w.phase(p) == p * stride % 16);
            EXPECT(expect >= w.vectors(w.phase(p)));
            EXPECT((w.vectors(w.phase(p)) - 1) * 16 < bytes + w.phase(p));
        }
    }
    // registered groups: over all ranks and blocks, the tiles of the walk cover every whole
    // vector of every tensor exactly once, in order, never across a tensor boundary and
    // never longer than a tile; the ragged last vectors are left to the element-wise tail
    for (int trial = 0; trial < 600; ++trial) {
        constexpr unsigned long long N = 4;  // f32 lanes
        const int n = 1 + static_cast<int>(rng() % 120);
        std::vector<PeerEntry> tab;
        unsigned long long voff = 0;
        for (int i = 0; i < n; ++i) {
            PeerEntry e;
            std::memset(&e, 0, sizeof(e));
            e.voff = voff;
            e.count = 1 + rng() % (i % 7 == 0 ? 300000 : 900);  // (empty tensors never enter a table)
            voff += (e.count + N - 1) / N;
            tab.push_back(e);
        }
        GroupPeerArgs a;
        std::memset(&a, 0, sizeof(a));
        a.table = tab.data();
        a.ntable = n;
        a.nvec = voff;
        const int world = 1 + static_cast<int>(rng() % 8);
        const int nb = 1 + static_cast<int>(rng() % 40);
        const unsigned int tile_vec = 32u << (rng() % 6);
        std::vector<unsigned long long> next(n, 0);  // first vector of each tensor not covered yet
        for (int r = 0; r < world; ++r) {
            for (int b = 0; b < nb; ++b) {
                const Span sp = span_of(a.nvec, world, r, nb, b);
                if (sp.lo >= sp.hi) { continue; }
                TileCursor c;
                c.i = find_peer_entry(a.table, a.ntable, sp.lo);
                c.v = c.end = 0;
                EXPECT(tab[c.i].voff <= sp.lo);
                if (!cursor_enter<N>(a, sp, &c)) { continue; }
                Tile t;
                while (cursor_next<N>(a, sp, &c, tile_vec, &t)) {
                    const int i = static_cast<int>(t.e - tab.data());
                    EXPECT(i >= 0 && i < n);
                    EXPECT(t.nv >= 1 && t.nv <= tile_vec);
                    EXPECT(t.v0 == next[i]);                         // in order, no gap, no overlap
                    EXPECT(t.v0 + t.nv <= tab[i].count / N);         // whole vectors of this tensor only
                    EXPECT(tab[i].voff + t.v0 >= sp.lo && tab[i].voff + t.v0 + t.nv <= sp.hi);
                    next[i] = t.v0 + t.nv;
                }
            }
        }
        for (int i = 0; i < n; ++i) { EXPECT(next[i] == tab[i].count / N); }
    }
    // descriptor tables: the entry found for v really contains v (or is the
    // last one starting at or before v when v falls into padding-free gaps)
    for (int trial = 0; trial < 2000; ++trial) {
        const int n = 1 + static_cast<int>(rng() % 300);
        std::vector<GroupEntry> tab(n);
        unsigned long long voff = 0;
        for (int i = 0; i < n; ++i) {
            tab[i].src = nullptr;
            tab[i].dst = nullptr;
            tab[i].voff = voff;
            tab[i].count = rng() % 5 == 0 ? 0 : 1 + rng() % 10000;  // some empty tensors
            voff += entry_nvec<DT_F32>(tab[i].count);
        }
        for (int q = 0; q < 50 && voff > 0; ++q) {
            const unsigned long long v = rng() % voff;
            const int i = find_entry(tab.data(), n, v);
            EXPECT(i >= 0 && i < n && tab[i].voff <= v);
            EXPECT(i == n - 1 || tab[i + 1].voff > v);
            // walking forward from i (as the kernel does) reaches the owner of v
            bool found = false;
            for (int j = i; j < n && tab[j].voff <= v; ++j) {
                found = found || v < tab[j].voff + entry_nvec<DT_F32>(tab[j].count);
            }
            EXPECT(found);
        }
    }
    // group planning: every element lands in exactly one piece, chunks respect
    // the slot size, pieces start on vector boundaries and keep tensor order
    for (int trial = 0; trial < 2000; ++trial) {
        const size_t n = 1 + rng() % 60;
        const size_t lanes = size_t(1) << (rng() % 5);  // 1, 2, 4, 8, 16 elements per vector
        const size_t cap = 1 + rng() % 3000;
        std::vector<size_t> counts(n);
        for (auto &c : counts) { c = rng() % 7 == 0 ? 0 : 1 + rng() % (cap * lanes * 3); }
        const auto chunks = plan_group_pieces(n, counts.data(), lanes, cap);
        std::vector<size_t> covered(n, 0);
        size_t last_tensor = 0;
        for (const auto &chunk : chunks) {
            size_t fill = 0;
            for (const auto &p : chunk) {
                EXPECT(p.tensor >= last_tensor && p.count > 0);
                last_tensor = p.tensor;
                EXPECT(p.voff == fill && p.first_elem == covered[p.tensor]);
                covered[p.tensor] += p.count;
                fill += (p.count + lanes - 1) / lanes;
                EXPECT(p.first_elem % lanes == 0);  // splits happen at vector boundaries
            }
            EXPECT(fill <= cap);
        }
        for (size_t i = 0; i < n; ++i) { EXPECT(covered[i] == counts[i]); }
    }
    // arena: a buffer ends with the slot or the heap in which it starts, and none starts in the
    // pad or among the mailboxes
    for (const size_t staging : {size_t{4096}, size_t{1} << 20}) {
        ArenaLayout a;
        a.staging = staging;
        a.mail = 8192;
        a.end = a.heap_off() + 65536;
        for (int i = 0; i < 2; ++i) {
            EXPECT(a.holds(a.slot(i), staging) && !a.holds(a.slot(i), staging + 1));
            EXPECT(a.holds(a.slot(i) + staging - 16, 16) && !a.holds(a.slot(i) + staging - 16, 17));
            EXPECT(!a.holds(a.slot(i) + 8, 8) && !a.holds(a.slot(i), ~size_t{0}));
        }
        EXPECT(!a.holds(0, 1) && !a.holds(kDataOffset - 16, 16));
        EXPECT(!a.holds(a.mail_off(), 16) && !a.holds(a.heap_off() - 16, 16));
        EXPECT(a.holds(a.heap_off(), 65536) && !a.holds(a.heap_off() + 16, 65536) && !a.holds(a.end, 0));
    }
    // symmetric heap: deterministic first fit, 256-byte granules, coalescing
    {
        OffsetHeap h;
        h.reset(4096, 1 << 20);
        const size_t a = h.alloc(100), b = h.alloc(300), c = h.alloc(1);
        EXPECT(a == 4096 && b == 4096 + 256 && c == 4096 + 256 + 512);
        h.release(b);
        EXPECT(h.alloc(512) == b);   // exact hole reused
        h.release(a);
        h.release(b);
        EXPECT(h.alloc(700) == a);   // the two holes merged (256 + 512 >= 768)
        bool threw = false;
        try {
            h.alloc(2 << 20);
        } catch (const std::bad_alloc &) {
            threw = true;
        }
        EXPECT(threw);
        threw = false;
        try {
            h.release(12345);
        } catch (const std::invalid_argument &) {
            threw = true;
        }
        EXPECT(threw);
        // two heaps fed the same calls hand out the same offsets (ranks stay symmetric)
        OffsetHeap x, y;
        x.reset(0, 1 << 24);
        y.reset(0, 1 << 24);
        std::vector<size_t> live;
        for (int i = 0; i < 2000; ++i) {
            if (!live.empty() && rng() % 3 == 0) {
                const size_t k = rng() % live.size();
                x.release(live[k]);
                y.release(live[k]);
                live.erase(live.begin() + k);
            } else {
                const size_t bytes = 1 + rng() % 5000;
                const size_t ox = x.alloc(bytes), oy = y.alloc(bytes);
                EXPECT(ox == oy && ox % 256 == 0);
                live.push_back(ox);
            }
        }
    }
    // the measured algorithm table
    {
        AlgoTuning t8;
        t8.world = 8;
        t8.has_nvls = true;
        EXPECT(select_algo(t8, 64 << 10, true, false) == kAlgoNvlsOneShot);
        EXPECT(select_algo(t8, 2 << 20, true, false) == kAlgoNvlsOneShot);
        EXPECT(select_algo(t8, (2 << 20) + 16, true, false) == kAlgoNvls);
        EXPECT(select_algo(t8, 4096, true, true) == kAlgoNvls);            // in place
        EXPECT(select_algo(t8, 256 << 10, false, false) == kAlgoOneShot);  // e.g. prod: no NVLS
        EXPECT(select_algo(t8, (256 << 10) + 16, false, false) == kAlgoTwoShot);
        AlgoTuning t2 = t8;
        t2.world = 2;
        EXPECT(select_algo(t2, 8 << 20, true, false) == kAlgoOneShot);  // the switch adds nothing at 2
        EXPECT(select_algo(t2, 1 << 30, true, false) == kAlgoTwoShotTma);  // large: bulk-copy pulls
        EXPECT(select_algo(t2, 32 << 20, true, true) == kAlgoTwoShot);
        t2.tma_min = SIZE_MAX;
        EXPECT(select_algo(t2, 1 << 30, true, false) == kAlgoTwoShot);
        AlgoTuning t4 = t8;
        t4.world = 4;
        t4.has_nvls = false;
        EXPECT(select_algo(t4, 1 << 20, true, false) == kAlgoOneShot);
        EXPECT(select_algo(t4, (1 << 20) + 16, true, false) == kAlgoTwoShot);
        t4.tma_min = 1u << 20;
        EXPECT(select_algo(t4, (1 << 20) + 16, true, false) == kAlgoTwoShotTma);
        t4.tma_min = 64u << 20;
        EXPECT(select_algo(t4, 64u << 20, true, true) == kAlgoTwoShotTma);
        t8.tma_over_nvls_min = 32u << 20;  // NVLS worlds may prefer it from some size up
        EXPECT(select_algo(t8, 16u << 20, true, true) == kAlgoNvls);
        EXPECT(select_algo(t8, 32u << 20, true, true) == kAlgoTwoShotTma);
        t8.tma_over_nvls_min = SIZE_MAX;
        AlgoTuning t1;
        EXPECT(select_algo(t1, 1 << 20, true, false) == kAlgoOneShot);
        EXPECT(select_algo(t1, 1 << 20, true, true) == kAlgoTwoShot);
        t8.oneshot_max = 1024;  // overrides
        EXPECT(select_algo(t8, 2048, false, false) == kAlgoTwoShot);
        t8.oneshot_max = 0;
        // grids: one vector ... 1 GiB
        EXPECT(select_blocks(t8, 1, kAlgoNvls) == 1);
        EXPECT(select_blocks(t8, (1ull << 30) / 16, kAlgoNvls) == 24);
        EXPECT(select_blocks(t8, (8ull << 20) / 16, kAlgoNvls) == 32);  // 1 MB per rank / 32 KB per CTA
        EXPECT(select_blocks(t8, (1ull << 30) / 16, kAlgoTwoShot) == 128);
        EXPECT(select_blocks(t8, (1ull << 30) / 16, kAlgoOneShot) == 128);
        EXPECT(select_blocks(t1, (1ull << 30) / 16, kAlgoTwoShot) == 148);
        EXPECT(select_blocks(t8, (1ull << 30) / 16, kAlgoTwoShotTma) == 148);  // one CTA per SM
        t8.tma_blocks = 64;
        EXPECT(select_blocks(t8, (1ull << 30) / 16, kAlgoTwoShotTma) == 64);
        t8.tma_blocks = 0;
        {   // ring geometry: at least two slots, inside the budget, whole granules
            for (int w = 1; w <= kMaxRanks; ++w) {
                for (unsigned int want : {0u, 64u, 256u, 512u, 1000u, 4096u}) {
                    int st = 0;
                    unsigned int tv = 0, bytes = 0;
                    tma_geometry(w, want, &st, &tv, &bytes);
                    EXPECT(st >= 2 && st <= kTmaMaxStages && tv >= 32 && tv % 32 == 0);
                    EXPECT(bytes == st * w * tv * 16u && bytes <= kTmaSmemBudget);
                    EXPECT(w * tv * 16u < (1u << 20));  // one slot's bytes fit an mbarrier's count
                }
            }
        }
        AlgoTuning loop = t8;
        loop.vranks = 8;
        loop.has_nvls = false;
        EXPECT(select_blocks(loop, (1ull << 30) / 16, kAlgoTwoShot) == 18);  // 148 SMs / 8 rows
        {   // one-shots of ordinary tensors: further among ranks of one GPU, never where the knob says how far
            AlgoTuning t;
            for (t.world = 2; t.world <= kMaxRanks; ++t.world) {
                t.vranks = 1;
                EXPECT(staged_oneshot_limit(t, 4) == oneshot_limit(t));
                t.vranks = t.world;
                const size_t wide = staged_oneshot_limit(t, 4), narrow = staged_oneshot_limit(t, 2);
                EXPECT(narrow >= oneshot_limit(t) && (t.world == 2 ? wide == oneshot_limit(t) : wide > narrow));
                t.oneshot_max = 1024;
                EXPECT(staged_oneshot_limit(t, 4) == 1024);
                t.oneshot_max = 0;
            }
            t.world = t.vranks = 4;
            EXPECT(staged_oneshot_limit(t, 8) == 44u << 17 && staged_oneshot_limit(t, 2) == 26u << 17 &&
                   staged_oneshot_limit(t, 1) == oneshot_limit(t));
        }
        for (int w = 1; w <= 16; ++w) {  // never zero, never above the pad size
            AlgoTuning t;
            t.world = w;
            for (unsigned long long nv : {1ull, 7ull, 4096ull, 1ull << 26}) {
                for (int algo = 0; algo < kAlgoCount; ++algo) {
                    const int b = select_blocks(t, nv, algo);
                    EXPECT(b >= 1 && b <= kMaxBlocks);
                }
            }
        }
    }
    {   // mailboxes: a message never outgrows one, and with more ranks none has a higher limit
        for (int w = 2; w <= kMaxRanks; ++w) {
            for (const bool sym : {false, true}) {
                const size_t cap = ll_capacity(w, w, 148), most = ll_limit(w, w, cap, sym);
                EXPECT(most >= 1 && most <= cap && cap <= 2u * 148u / w * kThreads);
                EXPECT(w == 2 || most <= ll_limit(w - 1, w - 1, ll_capacity(w - 1, w - 1, 148), sym));
                EXPECT(ll_limit(w, 1, ll_capacity(w, 1, 148), sym) == (64u << 10) / 16);
            }
        }
        EXPECT(ll_capacity(1, 1, 148) == 0);
        EXPECT(ll_limit(8, 8, ll_capacity(8, 8, 148), false) == (4u << 10) / 16);
        EXPECT(ll_limit(8, 8, ll_capacity(8, 8, 148), true) == (6u << 10) / 16);
    }
    {   // the rules of the in-kernel argument checks
        EXPECT(buffer_offset_ok(kDataOffset) && buffer_offset_ok(kDataOffset + 4096) && buffer_offset_ok(0));
        EXPECT(!buffer_offset_ok(kDataOffset + 8) && !buffer_offset_ok(64) && !buffer_offset_ok(kDataOffset - 16));
        GroupEntry tab[3];
        for (auto &e : tab) { e.src = nullptr; e.dst = nullptr; }
        tab[0].voff = 0;  tab[0].count = 10;   // 3 vectors of f32
        tab[1].voff = 3;  tab[1].count = 4;    // 1 vector
        tab[2].voff = 4;  tab[2].count = 1;
        for (int i = 0; i < 3; ++i) { EXPECT(table_entry_in_range<DT_F32>(tab, i, 3, 5)); }
        EXPECT(!table_entry_in_range<DT_F32>(tab, 2, 3, 4));   // runs past the buffer
        tab[1].voff = 2;                                       // overlaps its predecessor
        EXPECT(!table_entry_in_range<DT_F32>(tab, 0, 3, 5));
    }
    EXPECT(entry_nvec<DT_BF16>(9) == 2 && entry_nvec<DT_U8>(16) == 1 && entry_nvec<DT_F64>(3) == 2);
    std::printf("test-partition: %s\n", failures == 0 ? "OK" : "FAILED");
    return failures == 0 ? 0 : 1;
}
