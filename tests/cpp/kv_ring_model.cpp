// The K/V ring of the prefill kernel on the CPU: loads land in any order, every role runs at any speed. Uses the order,
// the barrier choice and the phase bookkeeping of kv_ring.cuh; prints, per plan, how many of the runs read a tile that
// was not there ("early") and how many came to a stop ("stuck").
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "kv_ring.cuh"

using namespace sca_b200;

// kOwn: the kernel's plan. The other two are mistakes: K and V of a slot on one barrier, the warps that rewrite V waiting
// for V only, or for every tile.
enum Plan { kOwn = 0, kSharedSkipK = 1, kSharedSeeAll = 2 };

struct Barrier {  // mbarrier as a waiter sees it: the phase of the given parity is over, or it is not
    int arrivals = 0, need = 1, phases = 0;
    void Arrive() {
        if (++arrivals == need) arrivals = 0, ++phases;
    }
    bool Over(uint32_t parity) const { return (phases & 1u) != parity; }
};
struct Load {
    bool is_v;
    int slot;
};

// 0 = sound, 1 = early, 2 = stuck
int Run(Plan plan, int slots, bool double_scores, int converters, unsigned seed) {
    std::mt19937 rng(seed);
    std::vector<Load> loads;
    for (int item = 0; item < 3; ++item) {
        const int n = 1 + static_cast<int>(rng() % 9);
        for (int it = 0; it < 2 * n; ++it) {
            const int slot = static_cast<int>(loads.size()) % slots;
            loads.push_back({RingOrder(it, n, double_scores).is_v, slot});
        }
    }
    const int total = static_cast<int>(loads.size());
    auto phase_of = [&](int i) { return static_cast<uint32_t>(i / slots) & 1u; };
    std::vector<Barrier> full(2 * slots), empty(slots), ready(slots);
    for (Barrier& b : ready) b.need = converters;
    auto full_of = [&](int i) { return plan == kOwn ? RingFullBarrier(loads[i].is_v, loads[i].slot, slots) : loads[i].slot; };
    std::vector<int> content(slots, -1), rewritten(slots, 0);
    std::vector<char> landed(total, 0);
    std::vector<int> flying;
    int issued = 0, consumed = 0;
    std::vector<int> walked(converters, 0);
    RingPhases k_phases, mma_v_phases;
    std::vector<RingPhases> v_phases(converters);
    const int actors = 3 + converters;  // producer, memory, products, converters
    std::vector<int> weight(actors);
    for (int& w : weight) w = 1 << (rng() % 8);

    while (consumed < total) {
        std::vector<int> able;
        auto may = [&](int actor) {
            for (int i = 0; i < weight[actor]; ++i) able.push_back(actor);
        };
        if (issued < total && empty[loads[issued].slot].Over(phase_of(issued) ^ 1u)) may(0);
        if (!flying.empty()) may(1);
        {
            const Load& l = loads[consumed];
            RingPhases look = l.is_v ? mma_v_phases : k_phases;
            const bool wait_ready = l.is_v && converters > 0;
            const uint32_t parity = plan == kOwn || wait_ready ? look.Take(l.slot) : phase_of(consumed);
            if ((wait_ready ? ready[l.slot] : full[full_of(consumed)]).Over(parity)) may(2);
        }
        for (int c = 0; c < converters; ++c) {
            while (walked[c] < total && plan != kSharedSeeAll && !loads[walked[c]].is_v) ++walked[c];
            if (walked[c] == total) continue;
            RingPhases look = v_phases[c];
            const uint32_t parity = plan == kOwn ? look.Take(loads[walked[c]].slot) : phase_of(walked[c]);
            if (full[full_of(walked[c])].Over(parity)) may(3 + c);
        }
        if (able.empty()) return 2;
        const int actor = able[rng() % able.size()];
        if (actor == 0) {
            content[loads[issued].slot] = issued;
            rewritten[loads[issued].slot] = 0;
            flying.push_back(issued++);
        } else if (actor == 1) {
            const size_t pick = rng() % flying.size();
            landed[flying[pick]] = 1;
            full[full_of(flying[pick])].Arrive();
            flying.erase(flying.begin() + static_cast<long>(pick));
        } else if (actor == 2) {
            const Load& l = loads[consumed];
            if (content[l.slot] != consumed || !landed[consumed] || (l.is_v && rewritten[l.slot] != converters)) return 1;
            if (l.is_v) mma_v_phases.Take(l.slot);
            else k_phases.Take(l.slot);
            empty[l.slot].Arrive();
            ++consumed;
        } else {
            const int c = actor - 3, i = walked[c]++, slot = loads[i].slot;
            if (!loads[i].is_v) continue;
            v_phases[c].Take(slot);
            if (content[slot] != i || !landed[i]) return 1;
            ++rewritten[slot];
            ready[slot].Arrive();
        }
    }
    return 0;
}

int main() {
    for (int plan = 0; plan < 3; ++plan) {
        for (int slots : {5, 8}) {
            for (int converters : {0, 1, 2}) {
                if (plan != kOwn && converters == 0) continue;
                int early = 0, stuck = 0;
                const int runs = 4000;
                for (int seed = 0; seed < runs; ++seed) {
                    const int r = Run(static_cast<Plan>(plan), slots, slots == 5 && seed % 2, converters, static_cast<unsigned>(seed));
                    early += r == 1;
                    stuck += r == 2;
                }
                std::printf("%d %d %d %d %d\n", plan, slots, converters, early, stuck);
            }
        }
    }
    return 0;
}
