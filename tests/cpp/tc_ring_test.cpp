// CPU model of the shared-memory ring of the tcgen05 kernels: parity barriers, producers that take the k-blocks in turn,
// one consumer that releases the stages in order, and a drain by the first producer, under random schedules.
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "../../vai_b200/csrc/tc_ring.h"

namespace {

struct Barrier {
    uint32_t done = 0;                                      // completed phases
    bool passed(uint32_t parity) const { return (done & 1u) != (parity & 1u); }      // the phase of that parity is over
};

// false: a stage was overwritten before its k-block was used, read before it was filled, or nothing could move any more.
// first: k-blocks of the first tile, whose start fills the empty ring without waiting.
bool ring_holds(uint32_t stages, uint32_t producers, uint32_t kblocks, uint32_t first, uint32_t seed)
{
    std::mt19937 rng(seed);
    std::vector<Barrier> full(stages), empty(stages);
    std::vector<int64_t> holds(stages, -1);                 // k-block in the stage, -1 when released
    struct Producer { uint32_t kb, stage, phase, turn, drained; };
    const uint32_t npre = first < stages ? first : stages;
    std::vector<Producer> prod(producers, Producer{npre, npre == stages ? 0u : npre, npre == stages ? 1u : 0u, npre % producers, 0u});
    for (uint32_t i = 0; i < npre; ++i) { holds[i] = i; ++full[i].done; }
    uint32_t used = 0;
    auto finished = [&]() {
        if (used < kblocks || prod[0].drained < stages) return false;
        for (const Producer& p : prod)
            if (p.kb < kblocks) return false;
        return true;
    };
    for (uint32_t idle = 0; !finished();) {
        const uint32_t who = rng() % (producers + 1u);
        bool moved = false;
        if (who == producers) {                             // the consumer: k-blocks in order
            const uint32_t s = used % stages;
            if (used < kblocks && full[s].passed((used / stages) & 1u)) {
                if (holds[s] != (int64_t)used) return false;
                holds[s] = -1;
                ++empty[s].done;
                ++used;
                moved = true;
            }
        } else {
            Producer& p = prod[who];
            auto step = [&]() { if (++p.stage == stages) { p.stage = 0; p.phase ^= 1u; } };
            if (p.kb < kblocks) {
                if (p.turn != who) moved = true;
                else if (empty[p.stage].passed(p.phase ^ 1u)) {
                    if (holds[p.stage] != -1) return false;
                    holds[p.stage] = p.kb;
                    ++full[p.stage].done;
                    moved = true;
                }
                if (moved) { ++p.kb; p.turn = p.turn + 1u == producers ? 0u : p.turn + 1u; step(); }
            } else if (who == 0u && p.drained < stages && empty[p.stage].passed(p.phase ^ 1u)) {
                ++p.drained;
                step();
                moved = true;
                if (p.drained == stages && used < kblocks) return false;        // it may leave only when all is released
            }
        }
        idle = moved ? 0u : idle + 1u;
        if (idle > 10000u) return false;
    }
    return true;
}

bool holds_always(uint32_t stages, uint32_t producers)
{
    for (uint32_t seed = 0; seed < 200u; ++seed)
        for (uint32_t kblocks : {1u, 2u, 3u, 5u, 12u, 48u, 129u})
            if (!ring_holds(stages, producers, kblocks, seed % 2u ? kblocks : 1u + seed / 2u % kblocks, seed * 7919u + kblocks)) return false;
    return true;
}

}  // namespace

int main()
{
    int bad = 0;
    for (uint32_t stages = 2; stages <= 8u; ++stages) {
        const uint32_t p = vaicu::tc_producers(stages);
        if (p < 1u || !holds_always(stages, p)) { printf("%u stages with %u producers: broken ring\n", stages, p); ++bad; }
    }
    if (holds_always(2, 3)) { printf("the model misses three producers on two stages\n"); ++bad; }
    return bad;
}
