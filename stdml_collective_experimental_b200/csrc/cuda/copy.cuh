// Moving bytes between tensors of any address and arena memory in 16-byte vectors:
// streaming accesses, sources that start at an odd byte, stores that touch a
// tensor's own bytes only.
#pragma once
#include "prims.cuh"

namespace stdml::collective::cuda
{
// Tensor memory goes past the L2 as far as it can (evict first): the L2 is for the rings.
__device__ __forceinline__ unsigned long long evict_first_policy()
{
    unsigned long long p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

__device__ __forceinline__ uint4 ld_stream_v4(const void *p, unsigned long long policy)
{
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p), "l"(policy)
                 : "memory");
    return v;
}

__device__ __forceinline__ void st_stream_v4(void *p, const uint4 &v, unsigned long long policy)
{
    asm volatile("st.global.L2::cache_hint.v4.u32 [%0], {%1,%2,%3,%4}, %5;" ::"l"(p), "r"(v.x),
                 "r"(v.y), "r"(v.z), "r"(v.w), "l"(policy)
                 : "memory");
}

// Bytes [a, a + 16) of the 32 bytes lo, hi (0 <= a < 16).
__device__ __forceinline__ uint4 shift_bytes(const uint4 &lo, const uint4 &hi, unsigned int a)
{
    uint4 v;
    uint32_t w0, w1, w2, w3, w4;
    switch (a >> 2) {
    case 0:
        w0 = lo.x, w1 = lo.y, w2 = lo.z, w3 = lo.w, w4 = hi.x;
        break;
    case 1:
        w0 = lo.y, w1 = lo.z, w2 = lo.w, w3 = hi.x, w4 = hi.y;
        break;
    case 2:
        w0 = lo.z, w1 = lo.w, w2 = hi.x, w3 = hi.y, w4 = hi.z;
        break;
    default:
        w0 = lo.w, w1 = hi.x, w2 = hi.y, w3 = hi.z, w4 = hi.w;
        break;
    }
    const uint32_t bits = (a & 3u) * 8u;
    v.x = __funnelshift_r(w0, w1, bits);
    v.y = __funnelshift_r(w1, w2, bits);
    v.z = __funnelshift_r(w2, w3, bits);
    v.w = __funnelshift_r(w3, w4, bits);
    return v;
}

// `bytes` bytes of tensor memory at any address, read as vectors in which they start
// `phase` bytes after the beginning of vector 0.  Bytes of a vector outside the
// tensor are undefined.  Reads whole aligned vectors that hold a byte of the tensor.
struct ShiftedSource {
    const char *begin, *end;
    unsigned int phase, odd;

    __device__ ShiftedSource(const void *p, unsigned long long bytes, unsigned int ph)
        : begin(static_cast<const char *>(p)), end(begin + bytes), phase(ph),
          odd(static_cast<unsigned int>((reinterpret_cast<unsigned long long>(p) - ph) & 15ull))
    {
    }

    // A vector all of whose bytes are the tensor's: no look at the ends.
    __device__ __forceinline__ uint4 load_inside(unsigned long long v, unsigned long long policy) const
    {
        const char *at = begin + 16ull * v - phase;
        if (odd == 0) { return ld_stream_v4(at, policy); }
        at -= odd;
        return shift_bytes(*reinterpret_cast<const uint4 *>(at),
                           *reinterpret_cast<const uint4 *>(at + 16), odd);
    }

    __device__ __forceinline__ uint4 load(unsigned long long v, unsigned long long policy) const
    {
        const char *at = begin + 16ull * v - phase;
        if (odd == 0) { return ld_stream_v4(at, policy); }
        at -= odd;
        uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
        if (at + 16 > begin) { lo = *reinterpret_cast<const uint4 *>(at); }
        if (at + 16 < end) { hi = *reinterpret_cast<const uint4 *>(at + 16); }
        return shift_bytes(lo, hi, odd);
    }
};

// Bytes of x that fall on [from, to) of the 16 at p, whatever their alignment.
static __device__ __noinline__ void store_some_bytes(char *p, uint4 x, int from, int to)
{
    union {
        uint4 v;
        uint32_t w[4];
        uint8_t b[16];
    } u;
    u.v = x;
    if (from == 0 && to == 16 && (reinterpret_cast<unsigned long long>(p) & 3ull) == 0ull) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { reinterpret_cast<uint32_t *>(p)[i] = u.w[i]; }
        return;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if (i >= from && i < to) { p[i] = static_cast<char>(u.b[i]); }
    }
}

// Vector v, in the numbering of ShiftedSource, to a tensor of `bytes` bytes.
__device__ __forceinline__ void store_virtual(char *tensor, unsigned long long bytes,
                                              unsigned int phase, unsigned long long v,
                                              const uint4 &x, unsigned long long policy)
{
    const long long first = static_cast<long long>(16ull * v) - static_cast<long long>(phase);
    const long long left = static_cast<long long>(bytes) - first;
    char *p = tensor + first;
    if (first >= 0 && left >= 16 && (reinterpret_cast<unsigned long long>(p) & 15ull) == 0ull) {
        st_stream_v4(p, x, policy);
        return;
    }
    store_some_bytes(p, x, first < 0 ? static_cast<int>(-first) : 0,
                     left < 16 ? static_cast<int>(left) : 16);
}
}  // namespace stdml::collective::cuda
