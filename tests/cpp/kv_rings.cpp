// The K/V rings of the prefill kernel, each as RingOf describes it, on the CPU: loads land in any order, every role runs at any
// speed. The thread that issues the products waits for the slots of a step one by one and frees them when the step is over.
// Prints, per ring, number of warps that rewrite V and plan, how many runs read a slot that did not hold what was waited for
// ("early") and how many came to a stop ("stuck").
#include <cstdio>
#include <random>
#include <vector>

#include "kv_ring.cuh"

using namespace sca_b200;

// kOwn: the kernel's plan. kCommon, a mistake: K and V of a slot complete one barrier, of which the warps that rewrite V see V only.
enum Plan { kOwn = 0, kCommon = 1 };

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
    bool frees;  // the last slot of a step: the step's slots are freed behind it
};

// The loads of an item of n tiles, and where the products free what they have waited for.
void AddItem(const RingShape& ring, int n, std::vector<Load>* loads) {
    const int first = static_cast<int>(loads->size()), count = 2 * n * ring.parts;
    for (int it = 0; it < count; ++it) {
        loads->push_back({RingOrder(it / ring.parts, n, ring.scores_ahead).is_v, (first + it) % ring.slots, true});
    }
    // One query tile (two slots per tile): a slot at a time. Two query tiles: K_0 alone, then {K_j+1, V_j} with the scores ahead,
    // {V_j, K_j+1} without, and at last V_n-1 alone.
    if (ring.parts == 1) {
        for (int it = 1; it + 1 < count; it += 2) (*loads)[static_cast<size_t>(first + it)].frees = false;
    }
}

// 0 = sound, 1 = early, 2 = stuck
int Run(Plan plan, const RingShape& ring, int converters, unsigned seed) {
    std::mt19937 rng(seed);
    std::vector<Load> loads;
    for (int item = 0; item < 3; ++item) AddItem(ring, 1 + static_cast<int>(rng() % 9), &loads);
    const int total = static_cast<int>(loads.size()), slots = ring.slots;
    auto phase_of = [&](int i) { return static_cast<uint32_t>(i / slots) & 1u; };
    std::vector<Barrier> full(2 * slots), empty(slots), ready(slots);
    for (Barrier& b : ready) b.need = converters;
    auto full_of = [&](int i) { return plan == kOwn ? RingFullBarrier(loads[i].is_v, loads[i].slot, slots) : loads[i].slot; };
    std::vector<int> content(slots, -1), rewritten(slots, 0), flying, walked(converters, 0);
    std::vector<char> landed(total, 0);
    int issued = 0, waited = 0, freed = 0;
    RingPhases k_phases, mma_v_phases;
    std::vector<RingPhases> v_phases(converters);
    std::vector<int> weight(3 + converters);  // producer, memory, products, converters
    for (int& w : weight) w = 1 << (rng() % 8);
    auto there = [&](int i) { return content[loads[i].slot] == i && landed[i] && (!loads[i].is_v || rewritten[loads[i].slot] == converters); };

    while (freed < total) {
        std::vector<int> able;
        auto may = [&](int actor) { able.insert(able.end(), static_cast<size_t>(weight[actor]), actor); };
        if (issued < total && empty[loads[issued].slot].Over(phase_of(issued) ^ 1u)) may(0);
        if (!flying.empty()) may(1);
        {
            const Load& l = loads[waited];
            const bool wait_ready = l.is_v && converters > 0;
            RingPhases look = l.is_v ? mma_v_phases : k_phases;
            const uint32_t parity = plan == kOwn || wait_ready ? look.Take(l.slot) : phase_of(waited);
            if ((wait_ready ? ready[l.slot] : full[full_of(waited)]).Over(parity)) may(2);
        }
        for (int c = 0; c < converters; ++c) {
            while (walked[c] < total && !loads[walked[c]].is_v) ++walked[c];
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
            const Load& l = loads[waited];
            (l.is_v ? mma_v_phases : k_phases).Take(l.slot);
            if (!there(waited)) return 1;
            ++waited;
            if (!l.frees) continue;
            for (; freed < waited; ++freed) {
                if (!there(freed)) return 1;
                empty[loads[freed].slot].Arrive();
            }
        } else {
            const int c = actor - 3, i = walked[c]++, slot = loads[i].slot;
            v_phases[c].Take(slot);
            if (content[slot] != i || !landed[i]) return 1;
            ++rewritten[slot];
            ready[slot].Arrive();
        }
    }
    return 0;
}

int main() {
    for (int dim : {64, 128, 256}) {
        const RingShape ring = RingOf(dim);
        for (int converters : {0, ring.converters}) {
            for (Plan plan : {kOwn, kCommon}) {
                int early = 0, stuck = 0;
                for (unsigned seed = 0; seed < 3000; ++seed) {
                    const int r = Run(plan, ring, converters, seed);
                    early += r == 1;
                    stuck += r == 2;
                }
                std::printf("%d %d %d %d %d\n", dim, converters, plan, early, stuck);
            }
        }
    }
    return 0;
}
