// Which frames decode ahead of the others for their checksums (dec_parts.h), on
// sizes at the lines of the rule. Prints "bad=0" when all held.
#include <cstdio>
#include <string>

#include "dec_parts.h"

using namespace ozl;

static int bad = 0;
#define CHECK(x) do { if (!(x)) { bad++; std::printf("line %d: %s\n", __LINE__, #x); } } while (0)

int main()
{
    size_t const M = size_t(1) << 20, K = LongChecksums::kLong, F = LongChecksums::kLongFse;
    auto rule = [](std::vector<size_t> b, char fse) {
        return LongChecksums(b, std::vector<char>(b.size(), 1), std::vector<char>(b.size(), fse));
    };
    auto marks = [&](std::vector<size_t> b, char fse) {
        std::string s;
        for (char c : rule(b, fse).of) s += c ? '1' : '0';
        return s;
    };
    // one frame just long enough beside a small one, and just not
    CHECK(marks({ K, 4 * M }, 0) == "10" && rule({ K, 4 * M }, 0).alone);
    CHECK(marks({ K - 1, 4 * M }, 0) == "" && !rule({ K - 1, 4 * M }, 0).alone);
    // with long FSE streams, beside as much work in small frames, and a little less
    std::vector<size_t> f(5, F / 4);
    f[0] = F;
    CHECK(marks(f, 1) == "10000" && !rule(f, 1).alone);
    f[4]--;
    CHECK(marks(f, 1) == "");
    f[4]++;
    f[0]--;
    CHECK(marks(f, 1) == "");
    for (char fse : { char(0), char(1) }) {
        size_t const L = fse ? F : K;
        // every frame long: kinds and runs stay
        CHECK(marks({ L }, fse) == "" && marks({ L, L }, fse) == "");
        CHECK(marks(std::vector<size_t>(16, 2 * L), fse) == "");
        // at least half the longest
        CHECK(marks({ 4 * L, 2 * L, 2 * L - 1, 3 * L / 2, 3 * L / 2 }, fse) == "11000");
    }
    CHECK(marks({ 32 * M, 4 * M, 4 * M }, 0) == "" && marks({ 64 * M, 64 * M, M }, 1) == "");
    // alone while the others are short beside the chain: 4.5 times the longest frame
    std::vector<size_t> b(1, K);
    while (b.size() <= 9) b.push_back(K / 2 - 16);
    b.push_back(9 * 16);
    CHECK(rule(b, 0).of[0] && rule(b, 0).alone);
    b.push_back(16);
    CHECK(rule(b, 0).of[0] && !rule(b, 0).of[1] && !rule(b, 0).alone);
    // a frame whose checksum is not verified is one of the others
    LongChecksums const c({ 2 * K, K, M }, { 0, 1, 0 }, { 0, 0, 0 });
    CHECK(c.of.size() == 3 && !c.of[0] && c.of[1] && !c.of[2] && c.alone);
    CHECK(LongChecksums({ K, M }, { 0, 0 }, { 0, 0 }).of.empty());
    CHECK(LongChecksums({}, {}, {}).of.empty() && LongChecksums({ 0, 0 }, { 1, 1 }, { 0, 0 }).of.empty());
    // nothing goes ahead of a frame of half the longest that stays behind
    CHECK(LongChecksums({ F, F - 1, M }, { 1, 1, 1 }, { 0, 1, 0 }).of.empty());
    CHECK(LongChecksums({ F, F / 2, M }, { 1, 1, 1 }, { 0, 1, 0 }).of.empty());
    LongChecksums const d({ F, F / 2 - 1, M }, { 1, 1, 1 }, { 0, 1, 0 });
    CHECK(d.of[0] && !d.of[1] && !d.of[2] && d.alone);
    // one kind of each
    LongChecksums const e({ F, F, F / 3, F / 3, F / 3 }, { 1, 1, 1, 1, 1 }, { 0, 1, 0, 1, 0 });
    CHECK(e.of[0] && e.of[1] && !e.of[2] && !e.alone);
    std::printf("bad=%d\n", bad);
    return bad != 0;
}
