// Launch shapes of the FSE decoders (kFse, kFse4): shared memory, streams per
// CTA, and what the autotuner tries. Host code too, for a CPU test.
#pragma once
#include <algorithm>
#include <cstdint>

#include "fse_norm.h"

namespace ozl {

// Forms of a stream's decoding table (kFse).
enum FseCells : int { kCells32, kCells24, kCells24Wide };
constexpr uint32_t kFseCtaSmem = 224 * 1024; // up to 32 tableLog-11 lanes per CTA (one decoding warp)

constexpr uint32_t kFseQuarterSmem = 56 * 1024; // four CTAs of this much fit an SM
constexpr int kFseRing = 16, kFseAhead = 12;   // stream ring: 256 bytes per lane, 192 bytes ahead
constexpr uint32_t kFseRingBytes = 16 + 16 * kFseRing; // a lane's ring and its mirror
constexpr uint32_t kFseScratch = 260 * 2 + 256 * 2 + 8; // a warp's table-build scratch: cum[260], next[256]

// warps that build a CTA's tables (the first one then decodes): a table takes
// about 5 us, and the scratch of the builders is the rings' memory where it fits.
// An odd number, so that the decoding warps of an SM's CTAs fall on different
// schedulers (with two, on every other one: 5.2 against 5.0 ms as in FseShape).
OZL_HD inline uint32_t fseWarps(uint32_t lanes) { return lanes >= 2 ? 3 : 1; }
OZL_HD inline uint32_t fseRingOff(uint32_t lanes, uint32_t tlMax, int cells)
{
    return lanes * ((cells == kCells32 ? 4u : 3u) << tlMax);
}
// shared memory of a CTA: tables of all lanes, then the rings (kFse) or the
// build scratch, whichever is larger
OZL_HD inline uint32_t fseSmemBytes(uint32_t lanes, uint32_t tlMax, int cells)
{
    uint32_t const rings = lanes * kFseRingBytes, scratch = fseWarps(lanes) * kFseScratch;
    return fseRingOff(lanes, tlMax, cells) + (rings > scratch ? rings : scratch);
}
// per lane of kFse4: 16-bit entries, symbols, stream ring (16-byte aligned
// for tableLog >= 4)
OZL_HD inline uint32_t fse4SlotBytes(uint32_t tlMax) { return (3u << tlMax) + 16u * kFseRing; }

// Launch::tune of an FSE launch: streams per CTA in the low byte; this flag
// selects the kernel with one lane per decoder state (kFse4) instead of one
// lane per stream (kFse).
constexpr uint32_t kTuneFseLanePerState = 0x100;

inline uint32_t fseLanes(uint32_t tlMax, int cells, uint32_t smem = kFseCtaSmem)
{
    uint32_t lanes = 32;
    while (lanes > 1 && fseSmemBytes(lanes, tlMax, cells) > smem) lanes--;
    return lanes;
}

// Table form and streams per CTA of a kFse launch of `streams` streams of at
// most tlMax bits on `sms` SMs; tune: Launch::tune.
// 32-bit cells step faster (96 against 115 cycles) but take a third more
// shared memory: they are used while every stream of the launch fits the SMs
// at once (24 per SM at tableLog 11), and for small tables; 24-bit cells where
// the streams come in waves (32 per SM).
// Untuned, small tables run as many lanes a CTA as fit. Large ones spread over
// the SMs, one CTA on each, up to what four CTAs of an SM hold: one decoding
// warp for each of its schedulers. (Spread over the four schedulers of an SM
// as well, a stream steps a little faster alone, but each warp then issues for
// fewer streams, which the launches beside it pay for: host-buffer decoding of
// 1024 mixed frames, eight rounds at once, 5.6 ms against 5.0 ms.)
struct FseShape {
    int cells;
    uint32_t lanes;
    FseShape(uint32_t streams, uint32_t tlMax, uint32_t tune, uint32_t sms)
    {
        uint32_t const perSm = (streams + sms - 1) / sms;
        cells = tlMax >= 12                                                                      ? kCells24Wide
                : tlMax <= 8 || perSm <= 4 * fseLanes(tlMax, kCells32, kFseQuarterSmem) ? kCells32
                                                                                                 : kCells24;
        uint32_t const maxLanes = fseLanes(tlMax, cells);
        lanes = tune & 0xFFu;
        if (!lanes) lanes = tlMax <= 8 ? maxLanes : std::min(perSm, fseLanes(tlMax, cells, kFseQuarterSmem));
        lanes = std::max(1u, std::min(lanes, maxLanes));
    }
};

// Values of Launch::tune that the autotuner times, none twice: the untuned
// shape first, which the others have to beat.
inline uint32_t fseCandidates(uint32_t streams, uint32_t tlMax, uint32_t sms, uint32_t* out, uint32_t cap)
{
    uint32_t n = 0;
    FseShape const untuned(streams, tlMax, 0, sms);
    uint32_t const most = fseLanes(tlMax, untuned.cells), most4 = fseLanes(tlMax, kCells24);
    if (n < cap) out[n++] = untuned.lanes;
    for (uint32_t c : { 32u, 17u, 16u, 11u, 8u, 6u, 5u, 4u, 3u, 2u })
        if (c <= most && c != untuned.lanes && n < cap) out[n++] = c;
    for (uint32_t c : { 8u, 6u, 4u }) // kFse4: streams per warp
        if (c <= most4 && n < cap) out[n++] = kTuneFseLanePerState | c;
    return n;
}

} // namespace ozl
