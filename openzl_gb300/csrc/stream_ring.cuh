// Device helpers: unaligned 16-byte reads (decoders and encoders) and kFse4's
// stream ring.
#pragma once
#include <cstdint>

namespace ozl {

// 16 bytes starting `off` bytes (1..15) into the 32 bytes (u0, u1); q and r
// are off / 4 and (off % 4) * 8, uniform across the block
__device__ __forceinline__ uint4 shiftCombine(uint4 u0, uint4 u1, uint32_t q, uint32_t r)
{
    uint32_t y0, y1, y2, y3, y4;
    switch (q) {
        case 0: y0 = u0.x; y1 = u0.y; y2 = u0.z; y3 = u0.w; y4 = u1.x; break;
        case 1: y0 = u0.y; y1 = u0.z; y2 = u0.w; y3 = u1.x; y4 = u1.y; break;
        case 2: y0 = u0.z; y1 = u0.w; y2 = u1.x; y3 = u1.y; y4 = u1.z; break;
        default: y0 = u0.w; y1 = u1.x; y2 = u1.y; y3 = u1.z; y4 = u1.w; break;
    }
    return make_uint4(__funnelshift_r(y0, y1, r), __funnelshift_r(y1, y2, r), __funnelshift_r(y2, y3, r),
                      __funnelshift_r(y3, y4, r));
}

// Chunks are the 16-byte-aligned blocks of global memory that hold at least
// one byte of the stream (such a block never crosses a page), counted from
// the block holding the stream's first byte. Positions are bit indices above
// bit 0 of that block.
template <int RING, int AHEAD>
struct StreamRing {
    static_assert((RING & (RING - 1)) == 0 && AHEAD + 1 <= RING, "ring shape");
    const uint8_t* g16;  // 16-byte aligned block holding the stream's first byte
    uint32_t* ring;      // RING * 4 words of shared memory, 16-byte aligned
    int32_t low;         // lowest chunk whose words have been read

    __device__ __forceinline__ void issue(int32_t m)
    {
        if (m >= 0) {
            uint32_t const dst = uint32_t(__cvta_generic_to_shared(ring + 4 * (m & (RING - 1))));
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(g16 + 16 * size_t(m)) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
};

} // namespace ozl
