// Plays a pair of CTAs through their ring of operand slots with arrivals in random order and asks, at the moment when the rules of
// pair_exit.cuh let both CTAs end, whether an arrival is still on its way into either's shared memory.
//   argv: seeds.  argv[2] = "unwaited": the CTAs end as soon as their threads have met, for the test of the model itself.
// Prints "<runs> <runs that gave up> <runs that ended with an arrival under way> <runs that never could end>".
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "pair_exit.cuh"

using namespace tpw;

struct Barrier {
    int arrivals = 1, pending = 1;
    long tx = 0;
    uint32_t done = 0;      // phases completed
    void settle() {
        if (pending == 0 && tx == 0) {
            ++done;
            pending = arrivals;
        }
    }
    void arrive(long expect = 0) { tx += expect; --pending; settle(); }
    void complete(long bytes) { tx -= bytes; settle(); }
    // what a wait on a parity sees: the phase of that parity is over
    bool passed(uint32_t parity) const { return (done & 1) != parity; }
};
struct Event {
    int target;             // the CTA whose shared memory it arrives in (copies: the data; their bytes count on rank 0's barrier)
    Barrier *bar;
    long bytes;             // 0: an arrival
};

int main(int argc, char **argv) {
    const int seeds = atoi(argv[1]);
    const bool unwaited = argc > 2 && !strcmp(argv[2], "unwaited");
    int gave_up = 0, early = 0, stuck = 0;
    for (int seed = 0; seed < seeds; ++seed) {
        std::mt19937 rng(seed);
        auto pick = [&](uint32_t n) { return (uint32_t)(rng() % n); };
        const uint32_t slots = pick(2) ? 5 : pick(2) ? 4 : 2, total = 1 + pick(20), per_fill = 1 + pick(4);
        const bool fault = pick(2);          // every role stops somewhere
        const uint32_t cut[3] = {fault ? pick(total + 1) : total, fault ? pick(total + 1) : total, fault ? pick(total + 1) : total};
        auto bytes = [&](uint32_t u) { return (long)(u % 2 ? 16 : 32); };
        std::vector<Barrier> full(slots), empty[2] = {std::vector<Barrier>(slots), std::vector<Barrier>(slots)}, filled[2] = {std::vector<Barrier>(2), std::vector<Barrier>(2)};
        std::vector<Event> air;
        uint32_t issued[2] = {0, 0}, used = 0, fills = 0;
        auto deliver = [&]() {
            const uint32_t at = pick((uint32_t)air.size());
            const Event e = air[at];
            air.erase(air.begin() + at);
            if (e.bytes) e.bar->complete(e.bytes); else e.bar->arrive();
        };
        auto producer = [&](int r) {
            const uint32_t u = issued[r];
            if (u >= cut[r] || u >= total) return false;
            if (u >= slots && !empty[r][u % slots].passed(parity_of_use(u - slots, slots))) return false;
            if (r == 0) full[u % slots].arrive(2 * bytes(u));
            air.push_back({r, &full[u % slots], bytes(u)});
            ++issued[r];
            return true;
        };
        auto issuer = [&]() {
            const uint32_t u = used;
            if (u >= cut[2] || u >= total || !full[u % slots].passed(parity_of_use(u, slots))) return false;
            for (int r = 0; r < 2; ++r) air.push_back({r, &empty[r][u % slots], 0});
            ++used;
            if (used % per_fill == 0 || used == total) {
                for (int r = 0; r < 2; ++r) air.push_back({r, &filled[r][fills % 2], 0});
                ++fills;
            }
            return true;
        };
        // an accumulator is filled again only when its last commit has been seen
        auto room = [&]() {
            return fills < 2 || (filled[0][fills % 2].passed(parity_of_use(fills - 2, 2)) && filled[1][fills % 2].passed(parity_of_use(fills - 2, 2)));
        };
        for (uint32_t step = pick(200); step > 0; --step) {
            const uint32_t what = pick(4);
            if (what == 0) producer(0);
            else if (what == 1) producer(1);
            else if (what == 2) { if (room()) issuer(); }
            else if (!air.empty()) deliver();
        }
        // a run with a fault: every role has stopped where it is; one without goes on to its end
        const bool error = fault && !(used == total && issued[0] == total && issued[1] == total);
        if (!error) {
            while (used < total || issued[0] < total || issued[1] < total) {
                while (producer(0) || producer(1) || (room() && issuer())) {}
                if (!air.empty()) deliver();
            }
        }
        gave_up += error;
        const uint32_t most = issued[0] > issued[1] ? issued[0] : issued[1];
        if (error && !unwaited)
            for (uint32_t u = used; u < most; ++u) {
                const PairDebt debt = debt_of_use(u, issued[0], issued[1]);
                if (debt == PairDebt::arm_other) full[u % slots].arrive(bytes(u));
                if (debt == PairDebt::forgive) full[u % slots].complete(bytes(u));
            }
        auto may_end = [&]() {
            for (int r = 0; r < 2; ++r) {
                // the epilogue of a run without errors has waited for every accumulator; after an error the same wait is made up for
                for (uint32_t u = first_of_last_uses(fills, 2); u < fills; ++u)
                    if (!filled[r][u % 2].passed(parity_of_use(u, 2)) && !(unwaited && error)) return false;
                if (unwaited) continue;
                for (uint32_t u = first_of_last_uses(used, slots); u < used; ++u)
                    if (!empty[r][u % slots].passed(parity_of_use(u, slots))) return false;
            }
            if (error && !unwaited)
                for (uint32_t u = used; u < most; ++u)
                    if (!full[u % slots].passed(parity_of_use(u, slots))) return false;
            return true;
        };
        while (!may_end() && !air.empty()) deliver();
        if (!may_end()) ++stuck;
        else if (!air.empty()) ++early;
    }
    printf("%d %d %d %d\n", seeds, gave_up, early, stuck);
    return 0;
}
