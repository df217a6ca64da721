// How kFseEncLong cuts a chunk's chains into segments: what the run-up is made
// of. Host code too, so that a CPU test sees which cells a thread reads.
#pragma once
#include <cstdint>

#include "fse_norm.h"

namespace ozl {

// The share of one of `threads` threads in a coding table's 256 symbols: how
// many of its own (tid, tid + threads, ...) are present, and the sum over them
// of 1 / cells. deltaNbBits(y) is the symbol's (fseSymbolDeltas); it is asked
// for the thread's own symbols alone, which the thread has put in place itself,
// so the shares need no barrier before them.
template <class DeltaNbBits>
OZL_HD inline uint32_t fseSymbolShare(uint32_t tid, uint32_t threads, uint32_t tableLog, DeltaNbBits deltaNbBits,
                                      float& inverse)
{
    uint32_t const absent = ((tableLog + 1) << 16) - (1u << tableLog); // (asks for tableLog + 1 bits)
    uint32_t present = 0;
    for (uint32_t y = tid; y < 256; y += threads) {
        uint32_t const d = deltaNbBits(y), mb = (d + 0xffffu) >> 16;
        if (d == absent) continue;
        present++;
        inverse += 1.f / float(((mb << 16) - d) >> mb);
    }
    return present;
}

// The run-up of a segment in batches of four steps, also the least segment:
// four times the mean number of steps in which two unlike states meet, for a
// table of `size` cells, `symbols` present and the sum of 1 / cells over them.
OZL_HD inline uint32_t fseRunUp(uint32_t least, uint32_t size, uint32_t symbols, float inverse)
{
    float const steps = 300.f / inverse + float(size) / float(symbols);
    uint32_t const batches = uint32_t(steps < 1e6f ? steps : 1e6f);
    return batches > least ? batches : least;
}

} // namespace ozl
