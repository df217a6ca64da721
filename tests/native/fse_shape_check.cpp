// Launch shapes of the FSE decoder (fse_shape.h): the autotuner times the
// untuned shape, first, and no shape twice; every shape fits a CTA's shared
// memory. Prints "bad=0" when all held.
#include <cstdio>
#include <set>

#include "fse_shape.h"

using namespace ozl;

int main()
{
    long bad = 0, launches = 0;
    for (uint32_t sms : { 1u, 148u, 152u })
        for (uint32_t tl = 5; tl <= 12; tl++)
            for (uint32_t streams = 1; streams <= 12000; streams += streams < 200 ? 1 : 37) {
                FseShape const untuned(streams, tl, 0, sms);
                uint32_t cand[16];
                uint32_t const n = fseCandidates(streams, tl, sms, cand, 16);
                std::set<uint32_t> lanes, all;
                bad += n < 2 || n >= 16;
                bad += cand[0] != untuned.lanes;
                for (uint32_t k = 0; k < n; k++) {
                    bad += !all.insert(cand[k]).second;
                    if (cand[k] & kTuneFseLanePerState) {
                        bad += (cand[k] & 255u) * fse4SlotBytes(tl) > kFseCtaSmem || (cand[k] & 255u) > 8;
                        continue;
                    }
                    FseShape const s(streams, tl, cand[k], sms);
                    bad += s.cells != untuned.cells || s.lanes != cand[k] || !lanes.insert(s.lanes).second;
                    bad += s.lanes > 32 || fseSmemBytes(s.lanes, tl, s.cells) > kFseCtaSmem;
                }
                uint32_t few[2];
                bad += fseCandidates(streams, tl, sms, few, 2) > 2;
                launches++;
            }
    std::printf("launches=%ld bad=%ld\n", launches, bad);
    return bad != 0;
}
