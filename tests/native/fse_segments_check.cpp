// What kFseEncLong's threads count of a coding table before its first barrier
// (fse_segments.h): each reads the symbols that it wrote itself and no other,
// and all together find every symbol that is present, once, and the sum of
// 1 / cells. Prints "bad=0" when every table agreed.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "fse_segments.h"

using namespace ozl;

int main(int argc, char** argv)
{
    std::mt19937_64 rng(argc > 1 ? unsigned(std::atoi(argv[1])) : 1u);
    long bad = 0, tables = 0;
    uint32_t const threads = 128;
    for (int c = 0; c < 4000; c++) {
        // normalized counts of 2 to 256 symbols anywhere in the alphabet
        uint32_t const tl = 5 + rng() % 7, size = 1u << tl;
        uint32_t const symbols = 2 + rng() % (std::min(size, 256u) - 1);
        int norm[256] = {};
        for (uint32_t k = 0; k < symbols;) {
            uint32_t const y = c % 3 ? rng() % 256 : (c % 2 ? k : 255 - k); // spread, low half or high half first
            if (norm[y]) continue;
            norm[y] = rng() % 2 ? 1 : -1;
            k++;
        }
        for (uint32_t left = size - symbols; left;) {
            uint32_t const y = rng() % 256, by = 1 + rng() % left;
            if (!norm[y]) continue;
            norm[y] = (norm[y] < 0 ? 1 : norm[y]) + int(by);
            left -= by;
        }
        uint32_t dnb[256], present = 0, cumul = 0;
        double sum = 0;
        for (uint32_t y = 0; y < 256; y++) {
            int32_t find;
            ent::fseSymbolDeltas(norm[y], tl, cumul, dnb[y], find);
            uint32_t const cells = norm[y] < 0 ? 1 : uint32_t(norm[y]);
            cumul += cells;
            if (cells) {
                present++;
                sum += 1.0 / cells;
            }
        }
        uint32_t atLeastOne = 0, two = 0;
        float inverse = 0;
        for (uint32_t tid = 0; tid < threads; tid++) {
            uint32_t const own = fseSymbolShare(tid, threads, tl, [&](uint32_t y) {
                bad += y % threads != tid; // another thread's: not there before the barrier
                return dnb[y];
            }, inverse);
            atLeastOne += own > 0;
            two += own > 1;
        }
        bad += atLeastOne + two != present;
        bad += std::fabs(double(inverse) - sum) > 257 * std::ldexp(sum, -24); // at most 256 additions and one rounding each
        bad += fseRunUp(16, size, present, inverse) < 16;
        tables++;
    }
    std::printf("tables=%ld bad=%ld\n", tables, bad);
    return bad != 0;
}
