// Which frames of a batch decode ahead of the others because of their content
// checksums (DecodeBatch::makePlan). Host logic alone, for a CPU test.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace ozl {

// A content checksum is a serial chain (12.4 ns a KiB: 0.6 ms for 48 MiB, 3.3 ms
// for 256 MiB) that starts when its frame is decoded and then leaves the SMs to
// the rest, so a long one is worth starting early. Where the frame holds long
// FSE streams (chains of 0.4 ms and more each, which leave the SMs idle by
// themselves) that is worth less.
// ms without the rule, with the frames ahead alone, and ahead beside the others:
//   no long FSE stream: 48 MiB of timestamps beside 64 MiB 1.09, 0.75, 0.89,
//     beside 256 MiB 1.34, 0.86, 0.86; 96 MiB 1.90, 1.40, 1.44; 48 MiB column
//     beside 0.43 GB of matrices 2.42, 2.38, 2.46; 256 MiB column 4.22, 3.74,
//     4.06, beside 0.82 GB 5.33, 3.97, 4.45, beside 1.63 GB 6.60, 6.21, 5.96;
//     33 MiB of bytes beside 64 MiB 0.58, 0.63, 0.67;
//   long FSE streams: 32 MiB beside 2 GiB 5.00, 5.68, 4.93, beside 256 MiB 1.16,
//     1.65, 1.14; 64 MiB beside 64 MiB 1.29, 1.50, 1.38; four of 48 MiB, two of
//     them FSE, beside 32 MiB 1.23, 2.18, 1.21; 96 MiB beside 64 MiB 1.67,
//     1.69, 1.66, beside 256 MiB 1.90, 1.73, 1.77; 128 MiB beside 256 MiB 2.31,
//     2.25, 2.18, beside 1 GiB 3.87, 3.07, 2.82.
struct LongChecksums {
    std::vector<char> of; // per frame: decodes ahead of the others; empty if none does
    bool alone = false;   // the others wait until only checksums are left of these

    // The lines follow from the figures above. Nothing goes ahead of a frame of at
    // least half the longest that stays behind (its own path is as long: sixteen
    // of 64 MiB, half of them FSE, 2.08 and 2.21 ms; four of 48 MiB beside 32 MiB
    // 1.23 and 1.39), and FSE frames not of less work than the longest one (four
    // of 96 MiB beside 32 MiB 1.93 and 2.15).
    static constexpr uint64_t kLong = 48ull << 20, kLongFse = 96ull << 20;
    // Alone where the others' decoding (370 GB/s) is shorter than the chain that
    // it would run beside (82 GB/s): up to 4.5 times its bytes (ms alone and
    // beside: 80 MiB beside 3.2 times 1.16 and 1.24, 64 MiB beside 4 times 0.89
    // and 1.05, 48 MiB beside 5.3 times 0.89 and 0.86).
    static bool shorterThanChain(uint64_t others, uint64_t longest) { return others / 9 <= longest / 2; }

    // decoded bytes per frame, whether its content checksum is verified, and
    // whether it holds a long FSE stream
    LongChecksums(const std::vector<size_t>& bytes, const std::vector<char>& checked, const std::vector<char>& fse)
    {
        uint64_t longest = 0, others = 0;
        for (size_t i = 0; i < bytes.size(); i++)
            if (checked[i]) longest = std::max<uint64_t>(longest, bytes[i]);
        if (longest < kLong) return;
        std::vector<char> f(bytes.size(), 0);
        size_t n = 0;
        bool anyFse = false;
        for (size_t i = 0; i < bytes.size(); i++) {
            f[i] = checked[i] && bytes[i] >= longest / 2;
            if (f[i] && bytes[i] < (fse[i] ? kLongFse : kLong)) {
                if (fse[i]) return; // stays behind
                f[i] = 0;
            }
            n += f[i];
            anyFse |= f[i] && fse[i];
            if (!f[i]) others += bytes[i];
        }
        if (n == bytes.size() || (anyFse && others < longest)) return; // nothing, or little, to run beside the chains
        of = std::move(f);
        alone = !anyFse && shorterThanChain(others, longest);
    }
};

} // namespace ozl
