// Where the Huffman decoders cut a stream into runs (huf_split.h): runs start
// at multiples of the code lengths' common divisor, in order, and end at the
// stream's end; a decoder that starts at a run's first bit of a stream whose
// codes have one length meets the true boundaries at once. Prints "bad=0" when
// all held.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <random>

#include "huf_split.h"

using namespace ozl;

int main(int argc, char** argv)
{
    std::mt19937_64 rng(argc > 1 ? unsigned(std::atoi(argv[1])) : 1u);
    long bad = 0, cases = 0;
    for (int c = 0; c < 200000; c++) {
        // lengths 1 to 20, some sets of multiples of one number
        uint32_t const base = 1 + rng() % 10;
        uint32_t lengths = 0;
        for (int k = 1 + int(rng() % 4); k > 0; k--) lengths |= 1u << (c % 2 ? base * (1 + rng() % (20 / base)) : 1 + rng() % 20);
        uint32_t want = 0;
        for (uint32_t l = 1; l <= 20; l++)
            if (lengths >> l & 1) want = std::gcd(want, l);
        uint32_t const step = lengthStep(lengths);
        bad += step != want;
        // a stream of codes of these lengths
        int32_t const bits = int32_t(step * (rng() % (c % 5 ? 3000 : 700000)));
        uint32_t const lanes = c % 3 ? 8 : 128, S = splitRuns(bits, lanes);
        bad += S < 1 || S > lanes || (S > 1 && bits / int32_t(S) < 1024);
        int32_t before = 0;
        for (uint32_t j = 0; j <= S; j++) {
            int32_t const at = splitStart(bits, j, S, step);
            bad += at % int32_t(step) != 0 || at < before || (j == 0 && at != 0) || (j == S && at != bits);
            bad += at > int32_t(int64_t(bits) * j / S) || at + int32_t(step) <= int32_t(int64_t(bits) * j / S);
            before = at;
        }
        cases++;
    }
    // a corrupt stream's bits are no multiple: it still ends at its end
    for (int32_t bits : { -1, 0, 1, 1023, 1024, 2047, 9999, 10001 })
        for (uint32_t step : { 1u, 2u, 7u, 20u }) bad += splitStart(bits, splitRuns(bits, 8), splitRuns(bits, 8), step) != bits;
    std::printf("cases=%ld bad=%ld\n", cases, bad);
    return bad != 0;
}
