// Where the parts of a rank's arena lie: signal pad, two staging slots, the mailboxes of
// the small all-reduce, the symmetric heap.  Pure host logic, CPU-tested
// (tests/test_partition_cuda.cpp).
#pragma once
#include <cstddef>

#include "comm.cuh"

namespace stdml::collective::cuda
{
struct ArenaLayout {
    size_t staging = 0;  // bytes of one slot
    size_t mail = 0;     // bytes of all mailboxes
    size_t end = 0;      // of the arena

    size_t slot(int i) const { return kDataOffset + static_cast<size_t>(i) * staging; }
    size_t mail_off() const { return slot(2); }
    size_t heap_off() const { return mail_off() + mail; }

    // End of the slot or of the heap that holds `off`; 0: no collective's buffer starts there.
    size_t region_end(size_t off) const
    {
        if (off < slot(0) || off >= end) { return 0; }
        if (off < slot(2)) { return off < slot(1) ? slot(1) : slot(2); }
        return off < heap_off() ? 0 : end;
    }

    // Whether `bytes` bytes from `off` on are one buffer: aligned, and all of them inside the
    // slot or the heap in which they start.  (What comes behind a slot is the
    // other slot, the mailboxes and the users' tensors.)
    bool holds(size_t off, size_t bytes) const
    {
        const size_t to = region_end(off);
        return off % 16 == 0 && to != 0 && bytes <= to - off;
    }
};
}  // namespace stdml::collective::cuda
