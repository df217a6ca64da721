// Where the Huffman decoders cut a stream into runs (splitStream of
// decode_kernels.cu). Host code too, for a CPU test.
#pragma once
#include <cstdint>

#include "fse_norm.h"

namespace ozl {

// Runs of a stream of `bits` bits on up to `lanes` lanes: at least 1,024 bits each.
OZL_HD inline uint32_t splitRuns(int32_t bits, uint32_t lanes)
{
    uint32_t const most = bits > 0 ? uint32_t(bits) >> 10 : 0u;
    return most < 1 ? 1u : most < lanes ? most : lanes;
}

// The greatest common divisor of the code lengths in use (bit l of `lengths`:
// length l, 1 to 31).
OZL_HD inline uint32_t lengthStep(uint32_t lengths)
{
    if (lengths & (lengths >> 1)) return 1; // two lengths that follow one another: nearly every code
    uint32_t step = 0;
    for (uint32_t l = 1; l < 32; l++) {
        if (!(lengths >> l & 1)) continue;
        uint32_t a = step, b = l;
        while (a) {
            uint32_t const r = b % a;
            b = a;
            a = r;
        }
        step = b;
    }
    return step ? step : 1;
}

// Bits from the stream's top to the first of run j of S (j = S: its end). All
// code boundaries are multiples of `step` from the top, so runs start at one
// too: a lane that started between two would never meet them (code lengths 2
// and 4 from an odd bit), and the runs would follow one after another.
OZL_HD inline int32_t splitStart(int32_t bits, uint32_t j, uint32_t S, uint32_t step)
{
    int32_t const at = int32_t(int64_t(bits) * j / S);
    return j == S || step < 2 ? at : at - int32_t(uint32_t(at) % step);
}

} // namespace ozl
