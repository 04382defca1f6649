// Model of the stage ring of matvec_tc_kernel (csrc/matvec_tc.cu) under every order in which loads can land and warps can run: a
// producer, G groups of consumers, barriers with one bit of parity, two buffers of row sums. Prints the first thing that must not happen.
// Arguments: seed, runs, and with a fourth argument the walk in which slots pass from group to group (the model has to find its fault).
#include "ring.h"

#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

struct Bar { uint32_t phase = 0; int arrivals, pending, tx = 0; explicit Bar(int n) : arrivals(n), pending(n) {}
    bool passes(uint32_t par) const { return (phase & 1u) != par; }
    void settle() { if (pending == 0 && tx == 0) { ++phase; pending = arrivals; } } };

static bool g_shared = false;   // slots handed from group to group

template <int G> void advance(uint32_t &slot, uint32_t &par, uint32_t n) {
    if (!g_shared) { flb::ring_next<G>(slot, par, n); return; }
    slot += G;
    if (slot >= n) { slot -= n; par ^= 1u; }
}

template <int G> const char *run(std::mt19937 &rng, uint32_t n, uint32_t nseg, uint32_t units) {
    std::vector<Bar> full(n, Bar(1)), empty(n, Bar(1));
    std::vector<int> holds(n, -1);                       // stage whose bytes lie in the slot
    std::vector<uint32_t> flying;                        // stages on their way
    std::vector<uint32_t> at(n, 0);
    const uint32_t total = nseg * units;
    flb::RingTurn<G> turn;
    uint32_t p_slot = 0, p_par = 1, issued = 0;
    struct Group { uint32_t it, slot, par = 0, done = 0; } grp[G];
    for (int g = 0; g < G; ++g) { grp[g].it = g; grp[g].slot = g % n; }
    std::vector<uint32_t> slot_of(total);
    uint32_t consumed = 0;
    // one slow load at a time, as a missed translation makes it
    int slow = -1;
    for (uint32_t idle = 0; consumed < total; ++idle) {
        if (idle > 100000) return "stuck";
        const uint32_t what = rng() % 4;
        if (what == 0 && issued < total) {
            const uint32_t s = g_shared ? p_slot : turn.slot[0], par = g_shared ? p_par : turn.par[0];
            if (!empty[s].passes(par)) continue;
            if (full[s].pending == 0) return "a barrier armed while its phase is pending";
            --full[s].pending; full[s].tx += 1;
            holds[s] = -1;
            slot_of[issued] = s;
            flying.push_back(issued);
            if (slow < 0 && rng() % 4 == 0) slow = (int)issued;
            ++issued;
            if (g_shared) { if (++p_slot == n) { p_slot = 0; p_par ^= 1u; } } else turn.next(n);
            idle = 0;
        } else if (what == 1 && !flying.empty()) {
            const uint32_t k = rng() % flying.size(), st = flying[k];
            if ((int)st == slow && rng() % 64) continue;
            if ((int)st == slow) slow = -1;
            flying.erase(flying.begin() + k);
            holds[slot_of[st]] = (int)st;
            --full[slot_of[st]].tx;
            full[slot_of[st]].settle();
            idle = 0;
        } else if (what >= 2) {
            Group &c = grp[rng() % G];
            if (c.it >= total) { if (c.done < units) c.done = units; continue; }
            const uint32_t u = c.it / nseg;
            // the sums of unit v go where those of v - 2 were: every group has to be done with that one
            for (; c.done < u; ++c.done) {
                bool free = true;
                for (int g = 0; g < G; ++g) free = free && (c.done < 2 || grp[g].done + 1 >= c.done);
                if (!free) break;
            }
            if (c.done < u) continue;
            if (!full[c.slot].passes(c.par)) continue;
            if (holds[c.slot] != (int)c.it) return "a wait passed before its stage had landed";
            --empty[c.slot].pending;
            empty[c.slot].settle();
            ++consumed;
            c.it += G;
            advance<G>(c.slot, c.par, n);
            idle = 0;
        }
    }
    return nullptr;
}

int main(int argc, char **argv) {
    std::mt19937 rng((unsigned)atoi(argv[1]));
    const int runs = atoi(argv[2]);
    g_shared = argc > 3;
    for (int r = 0; r < runs; ++r) {
        const uint32_t n = 2 + rng() % 12, nseg = 1 + rng() % 7, units = 1 + rng() % 12;
        const char *bad = rng() % 4 ? run<2>(rng, n, nseg, units) : run<1>(rng, n, nseg, units);
        if (bad) { printf("%s: %u slots, %u segments, %u units\n", bad, n, nseg, units); return 1; }
    }
    return 0;
}
